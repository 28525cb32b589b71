// Machinery of the fused per-page transfer kernels (Hessian-vector product,
// Newton update, P2G): a CTA works through pieces of particle groups (the
// particles whose base node lies in one SPGrid page), each of its warps in two
// phases per chunk of its own cells' particles.
//
//  phase 1 (thread per particle): the particle's B-spline weights, a gradient
//          gathered from a staged 2x2x2-page window of a grid vector, the
//          per-particle 3x3 algebra, and a record in shared memory: the
//          particle's fractional offsets and the three rows of the 3x3 matrix
//          M_p whose product with grad w_ip is scattered.
//  phase 2 (thread per (cell, row)): the particles of one cell share their 27
//          stencil nodes, so a thread sums row r of M_p grad w_ip over the
//          cell's particles in 27 registers and adds them to the shared window
//          once.  Only occupied cells get threads.
//  flush:  the window [8][3][NPB] is added to the global block-dense vector
//          with one atomic per nonzero entry.
//
// The separable stencil sums use the per-axis index offsets of the 27 nodes
// (node (i,j,k) of a particle with base cell (lx,ly,lz) sits at window offset
// X_i + Y_j + Z_k), so the index arithmetic is one add per node.
#pragma once
#include <type_traits>

#include "xfer.cuh"

namespace zmpm {

constexpr int FUSED_THREADS = 128;

// Quadratic B-spline weight and derivative of stencil offset i (0, 1, 2) for
// the fractional position d = x/dx - base (BSplines.h:55-81).
template <class T>
__device__ __forceinline__ void bspline_all(T d, T w[3], T dw[3])
{
    const T z0 = T(1.5) - d;
    const T d1 = d - T(1);
    const T z2 = d - T(0.5);
    w[0] = T(0.5) * z0 * z0;
    w[1] = T(0.75) - d1 * d1;
    w[2] = T(0.5) * z2 * z2;
    dw[0] = -z0;
    dw[1] = T(-2) * d1;
    dw[2] = z2;
}

// Packed FP32 pairs (sm_100 FFMA2 and friends: two FP32 operations per
// instruction, each rounded as the scalar one).
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// bspline_all on a pair of fractional positions.
__device__ __forceinline__ void bspline_all2(float2 d, float2 w[3], float2 dw[3])
{
    const float2 z0 = add2(d, f2(-1.5f)); // d - 1.5 = -(1.5 - d)
    const float2 d1 = add2(d, f2(-1.0f));
    const float2 z2 = add2(d, f2(-0.5f));
    w[0] = mul2(mul2(z0, z0), f2(0.5f));
    w[1] = fma2(mul2(d1, f2(-1.0f)), d1, f2(0.75f));
    w[2] = mul2(mul2(z2, z2), f2(0.5f));
    dw[0] = z0;
    dw[1] = mul2(d1, f2(-2.0f));
    dw[2] = z2;
}

// Per-axis window offsets of the three stencil nodes along each axis, for a
// window of 8 pages of NPB nodes with `comp` scalars per node-page layout
// (node-major: offset counts nodes; component-major: the caller adds r * NPB).
template <class L>
struct StencilOffsets {
    int X[3], Y[3], Z[3]; // in units of nodes of a [8][NPB] window
    __device__ __forceinline__ StencilOffsets(int lx, int ly, int lz)
    {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int wx = lx + i, wy = ly + i, wz = lz + i;
            X[i] = ((wx >= L::BX) ? 4 * L::NPB : 0) + ((wx & (L::BX - 1)) << (L::YB + L::ZB));
            Y[i] = ((wy >= L::BY) ? 2 * L::NPB : 0) + ((wy & (L::BY - 1)) << L::ZB);
            Z[i] = ((wz >= L::BZ) ? L::NPB : 0) + (wz & (L::BZ - 1));
        }
    }
};
// The window's page t and element e of a node offset o = t * NPB + e.
template <int NPB>
__device__ __forceinline__ int window_scalar(int o, int comp, int ncomp)
{
    const int t = o / NPB, e = o - t * NPB;
    return (t * ncomp + comp) * NPB + e;
}

// Input windows of a grid vector: FP32 node-major float4 slabs ([B][NPB][4],
// the copy the Krylov solver keeps for the FP32 product) or FP64
// component-major slabs ([B][3][NPB], the solver's own vectors).
template <int NPB, class TX>
struct VecWindow;
template <int NPB>
struct VecWindow<NPB, float> {
    static constexpr int ELEMS = 8 * NPB * 4;
    static constexpr uint32_t SLAB = NPB * 4 * sizeof(float);
    static constexpr int64_t PAGE = NPB * 4; // elements per page in global memory
    __device__ __forceinline__ static void node(const float* w, int o, float v[3])
    {
        const float4 q = reinterpret_cast<const float4*>(w)[o];
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
    }
};
template <int NPB>
struct VecWindow<NPB, double> {
    static constexpr int ELEMS = 8 * NPB * 3;
    static constexpr uint32_t SLAB = NPB * 3 * sizeof(double);
    static constexpr int64_t PAGE = NPB * 3;
    __device__ __forceinline__ static void node(const double* w, int o, double v[3])
    {
        const int t = o / NPB, e = o - t * NPB;
        const double* p = w + t * 3 * NPB + e;
        v[0] = p[0];
        v[1] = p[NPB];
        v[2] = p[2 * NPB];
    }
};

// Stages the 8 page slabs of `vec` for the window of a CTA's one group; all
// threads call it.
template <int NPB, class TX>
__device__ __forceinline__ void stage_vec_window(TX* win, const TX* __restrict__ vec, const int32_t* nbr, uint64_t* bar, int32_t* flags)
{
    using W = VecWindow<NPB, TX>;
    static_assert(W::SLAB % 16 == 0, "bulk copies move multiples of 16 bytes");
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, 8 * W::SLAB);
#pragma unroll
        for (int t = 0; t < 8; ++t) bulk_g2s(win + t * W::PAGE, vec + (int64_t)nbr[t] * W::PAGE, W::SLAB, bar);
    }
    __syncthreads();
    mbar_wait_bounded(bar, 0u, flags);
}

// G(r, c) = sum over the 27 stencil nodes of x_r(node) d_c w(node) * dx (the
// caller scales by 1/dx), by separable contraction along z, then y, then x.
template <class L, class T, class TX>
__device__ __forceinline__ void gather_gradient(const TX* win, const StencilOffsets<L>& so, const T w[3][3], const T dw[3][3], T G[9])
{
#pragma unroll
    for (int q = 0; q < 9; ++q) G[q] = T(0);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        T C[3] = { 0, 0, 0 }, D[3] = { 0, 0, 0 }, E[3] = { 0, 0, 0 };
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            T A[3] = { 0, 0, 0 }, B[3] = { 0, 0, 0 };
            const int oij = so.X[i] + so.Y[j];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                TX xv[3];
                VecWindow<L::NPB, TX>::node(win, oij + so.Z[k], xv);
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    A[r] += w[2][k] * (T)xv[r];
                    B[r] += dw[2][k] * (T)xv[r];
                }
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                C[r] += w[1][j] * A[r];
                D[r] += dw[1][j] * A[r];
                E[r] += w[1][j] * B[r];
            }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            G[3 * r + 0] += dw[0][i] * C[r];
            G[3 * r + 1] += w[0][i] * D[r];
            G[3 * r + 2] += w[0][i] * E[r];
        }
    }
}

// gather_gradient for an FP32 node-major window: components 0 and 1 of each
// node (adjacent in the float4 load) accumulate as one packed pair.
template <class L>
__device__ __forceinline__ void gather_gradient_f32(const float* win, const StencilOffsets<L>& so, const float w[3][3], const float dw[3][3],
    float G[9])
{
    const float4* win4 = reinterpret_cast<const float4*>(win);
    float2 G01[3] = { f2(0.f), f2(0.f), f2(0.f) };
    float G2[3] = { 0.f, 0.f, 0.f };
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float2 C01 = f2(0.f), D01 = f2(0.f), E01 = f2(0.f);
        float C2 = 0.f, D2 = 0.f, E2 = 0.f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            float2 A01 = f2(0.f), B01 = f2(0.f);
            float A2 = 0.f, B2 = 0.f;
            const int oij = so.X[i] + so.Y[j];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float4 q = win4[oij + so.Z[k]];
                const float2 x01 = f2(q.x, q.y);
                A01 = fma2(x01, f2(w[2][k]), A01);
                B01 = fma2(x01, f2(dw[2][k]), B01);
                A2 = fmaf(q.z, w[2][k], A2);
                B2 = fmaf(q.z, dw[2][k], B2);
            }
            C01 = fma2(A01, f2(w[1][j]), C01);
            D01 = fma2(A01, f2(dw[1][j]), D01);
            E01 = fma2(B01, f2(w[1][j]), E01);
            C2 = fmaf(A2, w[1][j], C2);
            D2 = fmaf(A2, dw[1][j], D2);
            E2 = fmaf(B2, w[1][j], E2);
        }
        G01[0] = fma2(C01, f2(dw[0][i]), G01[0]);
        G01[1] = fma2(D01, f2(w[0][i]), G01[1]);
        G01[2] = fma2(E01, f2(w[0][i]), G01[2]);
        G2[0] = fmaf(C2, dw[0][i], G2[0]);
        G2[1] = fmaf(D2, w[0][i], G2[1]);
        G2[2] = fmaf(E2, w[0][i], G2[2]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        G[c] = G01[c].x;
        G[3 + c] = G01[c].y;
        G[6 + c] = G2[c];
    }
}

// ------------------------------------------------------ work by particle --
// The kernels of this family walk the groups as `pieces`: a CTA's share of the
// particles, cut at group boundaries.  A group costs about K particles' worth
// of fixed work (window, flush) plus its particles, so group g spans the
// weights [W(g), W(g + 1)), W(g) = group_start[g] + K g, the total weight is
// split evenly over the grid and a group that a share boundary cuts becomes two
// pieces (pieces of one group add to the same nodes).
struct Piece {
    int g, g0, s0, s1; // group, its first slot, the piece's slots [s0, s1)
};
struct GroupArgs {
    const int32_t *group_start, *group_nbr, *cells; // cells: GroupCells records, built with the groups
    int G, K;
};
struct Share {
    const int32_t* gs;
    int64_t w0, w1;
    int G, K, first, g;

    __device__ __forceinline__ Share(const GroupArgs& a) : gs(a.group_start), w0(0), w1(0), G(a.G), K(a.K), first(0), g(0)
    {
        if (G <= 0) return;
        const int P = gs[G], n = (int)gridDim.x;
        // with clearly more CTAs than groups: K at least the share, so that no
        // share reaches particles of two groups (a second piece would double
        // the latency of the whole pass)
        if (2ll * n >= 3ll * G) K = max(K, P / (n - G) + 1);
        const int64_t total = (int64_t)P + (int64_t)K * G;
        w0 = total * blockIdx.x / n;
        w1 = total * (blockIdx.x + 1) / n;
        int lo = 0, hi = G - 1; // the last group whose weight range starts at or before w0
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if ((int64_t)gs[m] + (int64_t)K * m <= w0)
                lo = m;
            else
                hi = m - 1;
        }
        first = lo;
    }
    __device__ __forceinline__ void rewind() { g = first; }
    __device__ __forceinline__ bool next(Piece& p)
    {
        while (g < G) {
            const int c = g, g0 = gs[c], n = gs[c + 1] - g0;
            const int64_t wp = (int64_t)g0 + (int64_t)K * c + K; // weight of the group's first particle
            if (wp - K >= w1) return false;
            ++g;
            const int64_t lo = w0 - wp, hi = w1 - wp;
            p.g = c;
            p.g0 = g0;
            p.s0 = g0 + (int)(lo < 0 ? 0 : (lo > n ? n : lo));
            p.s1 = g0 + (int)(hi < 0 ? 0 : (hi > n ? n : hi));
            if (p.s0 < p.s1) return true;
        }
        return false;
    }
};

// Shared state of a CTA: input windows and accumulation windows in two buffers
// each (a piece's window arrives during the piece before; its sums are flushed
// while the next piece accumulates), three buffers of group records (the one
// being flushed, the running one, the arriving one), and per warp the records
// of its current chunk of particles, NF arrays of CH values (particle-minor:
// phase 1's threads write consecutive words).  TX: the input window's type, or
// void for kernels without one.  The accumulators are FP64 for FP32 arithmetic
// too: the warps add in whatever order they get there, and FP32 sums in a varying
// order moved a MIXED solve's residual by 10% at its FP32 floor from run to run,
// and Newton iteration counts with it (an item's own FP32 sum has a fixed order).
// FP32 kernels have one accumulator, FP64 kernels two: two FP64 ones, or an FP32
// one per warp, left FP32 chunks of 74 particles, little more than half a warp's
// usual share (1M particles: 3.69 and 3.60 ms per substep).
// CH: what is left of the shared memory that lets CTAS of these run on an SM
// (227 KB, 1 KB of it reserved per CTA).
template <class L, class TX>
struct InputWindow {
    static constexpr int ELEMS = VecWindow<L::NPB, TX>::ELEMS;
    using Elem = TX;
};
template <class L>
struct InputWindow<L, void> {
    static constexpr int ELEMS = 0;
    using Elem = int32_t;
};
template <class L>
struct MetaBuf {
    int32_t cells[GroupCells<L>::WORDS];
    int32_t nbr[8];
};
constexpr int FUSED_WARPS = FUSED_THREADS / 32;
template <class L, class T, class TX, int NF, int NC>
struct GroupSmem {
    using W = InputWindow<L, TX>;
    static constexpr int ACCS = sizeof(T) == 4 ? 1 : 2;
    static constexpr size_t FIXED = 2 * W::ELEMS * sizeof(typename W::Elem) + ACCS * 8 * NC * L::NPB * sizeof(double) + 3 * sizeof(MetaBuf<L>) + 512;
    static constexpr size_t PER4 = 232448 / 4 - 1024, PER3 = 232448 / 3 - 1024;
    // four CTAs per SM where the windows leave room for records of a warp's usual share of a page, else three
    static constexpr int CTAS = FIXED + FUSED_WARPS * NF * 49 * sizeof(T) <= PER4 ? 4 : 3;
    static constexpr int ROOM = (int)(((CTAS == 4 ? PER4 : PER3) - FIXED) / (FUSED_WARPS * NF * sizeof(T))) - 1;
    static constexpr int CH = ROOM > 160 ? 160 : ROOM & ~1;
    static constexpr int FS = CH + 1; // odd: the fields of one particle fall in different banks
    static_assert(CH >= 32, "a chunk holds at least one particle per lane");
    alignas(128) typename W::Elem win[2][W::ELEMS ? W::ELEMS : 4];
    alignas(16) double acc[ACCS][8 * NC * L::NPB];
    alignas(16) MetaBuf<L> meta[3];
    alignas(8) uint64_t bar[2];
    alignas(16) T rec[FUSED_WARPS][NF * FS];
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Once per kernel, all threads: the barriers and the accumulation windows.
template <class SM>
__device__ __forceinline__ void group_smem_init(SM& sm)
{
    if (threadIdx.x == 0) {
        mbar_init(&sm.bar[0], 1);
        mbar_init(&sm.bar[1], 1);
    }
    constexpr int N = sizeof(sm.acc) / sizeof(sm.acc[0][0]);
    for (int i = threadIdx.x; i < N; i += FUSED_THREADS) (&sm.acc[0][0])[i] = 0;
    __syncthreads();
}

// Starts the transfers of a piece's group record (all threads) and input window
// (the last warp) into the buffers of piece number ph.
template <class L, class T, class TX, int NF, int NC>
__device__ __forceinline__ void group_fetch(GroupSmem<L, T, TX, NF, NC>& sm, const GroupArgs& a, int g, int ph, const TX* x)
{
    constexpr int Q = GroupCells<L>::WORDS / 4;
    static_assert(Q + 2 <= FUSED_THREADS, "one 16-byte copy per thread");
    MetaBuf<L>& m = sm.meta[ph % 3];
    const int t = threadIdx.x;
    if (t < Q)
        cp_async16(m.cells + 4 * t, a.cells + (int64_t)g * GroupCells<L>::WORDS + 4 * t);
    else if (t < Q + 2)
        cp_async16(m.nbr + 4 * (t - Q), a.group_nbr + 8ll * g + 4 * (t - Q));
    if constexpr (!std::is_void<TX>::value) {
        using W = VecWindow<L::NPB, TX>;
        static_assert(W::SLAB % 16 == 0, "bulk copies move multiples of 16 bytes");
        const int lane = t & 31;
        if (t >= FUSED_THREADS - 32) {
            const int32_t nb = lane < 8 ? a.group_nbr[8ll * g + lane] : 0;
            uint64_t* bar = &sm.bar[ph & 1];
            if (lane == 0) mbar_expect_tx(bar, 8 * W::SLAB);
            __syncwarp();
            if (lane < 8) {
                // the vector's generic-proxy writes (other CTAs, before a grid barrier) come before the bulk reads
                asm volatile("fence.proxy.async.global;" ::: "memory");
                bulk_g2s(&sm.win[ph & 1][lane * W::PAGE], x + (int64_t)nb * W::PAGE, W::SLAB, bar);
            }
        }
    }
}

// Phase 2 forms.  sum(): a[n] over the particles p0, p0 + 1 (then every `step`
// pairs) .. of one cell for item row r, from the chunk's records.
//
// Rows: sum_p row_r(M_p) . grad w_ip * dx (the rows already carry 1/dx).
// Records: fractions at 0-2, row r of the scattered matrix at 3 + 3 r ..
// 5 + 3 r.  FP32 takes particles two at a time as packed pairs.
template <class T>
struct RowsScatter {
    static constexpr int NF = 12, NC = 3;
    template <int FS>
    __device__ __forceinline__ static void sum(const T* rec, int r, int p0, int p1, int part, int parts, T a[27])
    {
        const T* fr = rec;
        const T* rrow = rec + (3 + 3 * r) * FS;
        if constexpr (sizeof(T) == 4) {
            float2 a2[27];
#pragma unroll
            for (int n = 0; n < 27; ++n) a2[n] = f2(0.f);
            for (int p = p0 + 2 * part; p < p1; p += 2 * parts) {
                // an odd last particle pairs with itself at zero weight
                const int pq = p + 1 < p1 ? p + 1 : p;
                const float sq = p + 1 < p1 ? 1.f : 0.f;
                float2 w[3][3], dw[3][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) bspline_all2(f2(fr[d * FS + p], fr[d * FS + pq]), w[d], dw[d]);
                const float2 s0 = f2(rrow[p], sq * rrow[pq]);
                const float2 s1 = f2(rrow[FS + p], sq * rrow[FS + pq]);
                const float2 s2 = f2(rrow[2 * FS + p], sq * rrow[2 * FS + pq]);
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float2 u = mul2(s0, mul2(w[1][j], w[2][k]));
                        const float2 v = fma2(s2, mul2(w[1][j], dw[2][k]), mul2(s1, mul2(dw[1][j], w[2][k])));
#pragma unroll
                        for (int i = 0; i < 3; ++i) a2[9 * i + 3 * j + k] = fma2(w[0][i], v, fma2(dw[0][i], u, a2[9 * i + 3 * j + k]));
                    }
            }
#pragma unroll
            for (int n = 0; n < 27; ++n) a[n] = a2[n].x + a2[n].y;
        }
        else {
#pragma unroll
            for (int n = 0; n < 27; ++n) a[n] = T(0);
            for (int p = p0 + part; p < p1; p += parts) {
                T w[3][3], dw[3][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) bspline_all(fr[d * FS + p], w[d], dw[d]);
                const T s0 = rrow[p], s1 = rrow[FS + p], s2 = rrow[2 * FS + p];
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const T u = s0 * (w[1][j] * w[2][k]);
                        const T v = s1 * (dw[1][j] * w[2][k]) + s2 * (w[1][j] * dw[2][k]);
#pragma unroll
                        for (int i = 0; i < 3; ++i) a[9 * i + 3 * j + k] += dw[0][i] * u + w[0][i] * v;
                    }
            }
        }
    }
};

// Affine: item (component, cell) adds w_ip (q + a (i - 1) + b (j - 1) + c (k - 1)),
// a vector written affinely in the node offset from the stencil's centre, which
// lies within half a cell of the particle: no term is larger than the vector at
// the stencil's nodes (about node 0 the terms were up to twice as large, and the
// FP32 MLS-MPM force lost up to 5%).  MASS (APIC P2G, particlesToGridHelper,
// MpmSimulationBase.cpp:563-608): component 0 adds w_ip m_p and components 1-3 the
// momentum m (v + C (x_i - x_p)); without it the three components are a vector
// (the MLS-MPM force).  Records: fractions at 0-2, the mass at 3 if any, then (q,
// a, b, c) of each vector component.
template <class T, bool MASS>
struct AffineScatter {
    static constexpr int NF = MASS ? 16 : 15, NC = MASS ? 4 : 3;
    template <int FS>
    __device__ __forceinline__ static void sum(const T* rec, int r, int p0, int p1, int part, int parts, T a[27])
    {
        const T* fr = rec;
        const bool vec = !MASS || r != 0;
        const T* row = rec + (MASS ? (vec ? 4 * r : 3) : 3 + 4 * r) * FS;
        if constexpr (sizeof(T) == 4) {
            float2 a2[27];
#pragma unroll
            for (int n = 0; n < 27; ++n) a2[n] = f2(0.f);
            for (int p = p0 + 2 * part; p < p1; p += 2 * parts) {
                const int pq = p + 1 < p1 ? p + 1 : p;
                const float sq = p + 1 < p1 ? 1.f : 0.f;
                float2 w[3][3], dw[3][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) bspline_all2(f2(fr[d * FS + p], fr[d * FS + pq]), w[d], dw[d]);
                const float2 q0 = f2(row[p], sq * row[pq]);
                float2 ax = f2(0.f), by = f2(0.f), cz = f2(0.f);
                if (vec) {
                    ax = f2(row[FS + p], sq * row[FS + pq]);
                    by = f2(row[2 * FS + p], sq * row[2 * FS + pq]);
                    cz = f2(row[3 * FS + p], sq * row[3 * FS + pq]);
                }
                const float2 nw0 = mul2(w[0][0], f2(-1.f)); // (i - 1) w_i: -w_0, 0, w_2
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float2 t = mul2(w[1][j], w[2][k]);
                        // (q + b (j - 1) + c (k - 1)) t and a t
                        float2 l = q0;
                        if (j != 1) l = fma2(by, f2((float)(j - 1)), l);
                        if (k != 1) l = fma2(cz, f2((float)(k - 1)), l);
                        const float2 u = mul2(l, t), v = mul2(ax, t);
                        a2[3 * j + k] = fma2(w[0][0], u, fma2(nw0, v, a2[3 * j + k]));
                        a2[9 + 3 * j + k] = fma2(w[0][1], u, a2[9 + 3 * j + k]);
                        a2[18 + 3 * j + k] = fma2(w[0][2], u, fma2(w[0][2], v, a2[18 + 3 * j + k]));
                    }
            }
#pragma unroll
            for (int n = 0; n < 27; ++n) a[n] = a2[n].x + a2[n].y;
        }
        else {
#pragma unroll
            for (int n = 0; n < 27; ++n) a[n] = T(0);
            for (int p = p0 + part; p < p1; p += parts) {
                T w[3][3], dw[3][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) bspline_all(fr[d * FS + p], w[d], dw[d]);
                const T q0 = row[p];
                const T ax = vec ? row[FS + p] : T(0), by = vec ? row[2 * FS + p] : T(0), cz = vec ? row[3 * FS + p] : T(0);
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const T t = w[1][j] * w[2][k];
                        const T u = (q0 + by * T(j - 1) + cz * T(k - 1)) * t, v = ax * t;
#pragma unroll
                        for (int i = 0; i < 3; ++i) a[9 * i + 3 * j + k] += w[0][i] * (u + T(i - 1) * v);
                    }
            }
        }
    }
};

// Occupied cells of a group below which its warps share the particles instead of
// the cells: whole cells left three warps idle on a group of one.  Newton substep
// of 1500 groups of 500 particles in 1 / 2 / 4 cells, FP32: 3.36, 2.86 and 2.67 ->
// 2.15, 2.12 and 2.09 ms; FP64: 4.74, 4.36 and 4.01 -> 3.11, 3.07 and 3.01.
constexpr int CUT_CELLS = 8;

// One warp's part of a piece: the occupied cells whose first particle falls in
// its quarter of the piece's particles (CUT_CELLS: the quarter itself).  Warps do not wait for one another
// inside a piece; each alternates phase 1 (lane per particle, record into the
// warp's own shared memory) and phase 2 (lane per (row, cell) item, one shared
// atomic per node) over its own particles, so one warp's loads overlap
// another's arithmetic.  When the last round of items leaves half the lanes
// free, two lanes share an item's particles.
template <class L, class T, class TX, class Scatter, class Phase1>
__device__ __forceinline__ void group_warp(GroupSmem<L, T, TX, Scatter::NF, Scatter::NC>& sm, const Piece& pc, int ph, const Phase1& phase1)
{
    using SM = GroupSmem<L, T, TX, Scatter::NF, Scatter::NC>;
    constexpr int NPB = L::NPB, NC = Scatter::NC, FS = SM::FS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t* st = sm.meta[ph % 3].cells; // group-relative first particle of each cell, [NPB + 1]
    const int nocc = st[GroupCells<L>::NOCC];
    const uint8_t* occ = reinterpret_cast<const uint8_t*>(st + GroupCells<L>::OCC);
    const int a0 = pc.s0 - pc.g0, a1 = pc.s1 - pc.g0, n = a1 - a0;
    const int t0 = a0 + n * warp / FUSED_WARPS, t1 = a0 + n * (warp + 1) / FUSED_WARPS;
    // the warp's run [lo, hi) of the occupied cells and its particles [p_lo, p_hi)
    int lo = 0, hi = 0, p_lo, p_hi;
    if (nocc < CUT_CELLS) { // its quarter of the particles and the cells they lie in
        if (t0 >= t1) return;
        const int c = lane < nocc ? occ[lane] : 0;
        lo = __popc(__ballot_sync(0xffffffffu, lane < nocc && st[c + 1] <= t0));
        hi = __popc(__ballot_sync(0xffffffffu, lane < nocc && st[c] < t1));
        p_lo = t0;
        p_hi = t1;
    }
    else { // the cells whose first particle in the piece falls in its quarter
#pragma unroll
        for (int k = 0; k < NPB; k += 32) {
            bool below0 = false, below1 = false;
            if (k + lane < nocc) {
                const int c = occ[k + lane], b = st[c], e = st[c + 1], f = b > a0 ? b : a0;
                below0 = e <= a0 || f < t0;
                below1 = e <= a0 || f < t1;
            }
            lo += __popc(__ballot_sync(0xffffffffu, below0));
            hi += __popc(__ballot_sync(0xffffffffu, below1));
        }
        if (lo >= hi) return;
        const int b0 = st[occ[lo]], e1 = st[occ[hi - 1] + 1];
        p_lo = b0 > a0 ? b0 : a0;
        p_hi = e1 < a1 ? e1 : a1;
    }
    T* rec = sm.rec[warp];
    double* acc = sm.acc[SM::ACCS == 2 ? ph & 1 : 0];
    const int ncell = hi - lo, items = NC * ncell;
    for (int c0 = p_lo; c0 < p_hi; c0 += SM::CH) {
        const int c1 = c0 + SM::CH < p_hi ? c0 + SM::CH : p_hi;
        __syncwarp();
        for (int p = c0 + lane; p < c1; p += 32) phase1.template run<FS>(sm.win[ph & 1], (int64_t)(pc.g0 + p), rec + (p - c0));
        __syncwarp();
        for (int q0 = 0; q0 < items; q0 += 32) {
            const int left = items - q0;
            const int parts = left <= 16 ? 2 : 1, width = parts == 2 ? left : 32; // items of this round
            const int part = parts == 2 && lane >= width ? 1 : 0;
            const int q = q0 + lane - part * width;
            const bool on = q < items && (parts == 1 || lane < 2 * width);
            // items row-major: the lanes hold consecutive cells of one row, so
            // their window atomics fall in distinct banks
            const int r = on ? q / ncell : 0, ce = occ[lo + (on ? q - r * ncell : 0)];
            const int b = st[ce], e = st[ce + 1];
            const int p0 = (b > c0 ? b : c0) - c0, p1 = on ? (e < c1 ? e : c1) - c0 : p0;
            T a[27];
            Scatter::template sum<FS>(rec, r, p0, p1, part, parts, a);
            if (parts == 2) {
#pragma unroll
                for (int m = 0; m < 27; ++m) a[m] += __shfl_down_sync(0xffffffffu, a[m], width);
            }
            const bool add = p0 < p1 && !part;
            const int lx = ce >> (L::YB + L::ZB), ly = (ce >> L::ZB) & (L::BY - 1), lz = ce & (L::BZ - 1);
            const StencilOffsets<L> so(lx, ly, lz);
            if (!add) continue;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        atomicAdd(acc + window_scalar<NPB>(so.X[i] + so.Y[j] + so.Z[k], r, NC), (double)a[9 * i + 3 * j + k]);
        }
    }
}

// All pieces of the CTA's share: out += the scattered sums (component c < NC0
// to outa [B][NC0][NPB], the rest to outb).  All threads call it; ph counts the
// CTA's pieces over the kernel.  A block barrier separates a piece's sums from
// their flush, which leaves its accumulators zero; FP32 has a second one before
// their next use, FP64 uses the other buffer meanwhile.
template <class L, class T, class TX, class Scatter, int NC0, class Phase1>
__device__ __forceinline__ void group_share(GroupSmem<L, T, TX, Scatter::NF, Scatter::NC>& sm, const GroupArgs& a, Share& share, const TX* x,
    double* __restrict__ outa, double* __restrict__ outb, int32_t* flags, int& ph, const Phase1& phase1)
{
    constexpr int NPB = L::NPB, NC = Scatter::NC;
    Piece cur, nxt;
    share.rewind();
    bool have = share.next(cur);
    if (!have) return;
    group_fetch(sm, a, cur.g, ph, x);
    cp_async_wait_all();
    __syncthreads();
    while (have) {
        const bool more = share.next(nxt);
        if (more) group_fetch(sm, a, nxt.g, ph + 1, x);
        if constexpr (!std::is_void<TX>::value) mbar_wait_bounded(&sm.bar[ph & 1], (uint32_t)((ph >> 1) & 1), flags);
        group_warp<L, T, TX, Scatter>(sm, cur, ph, phase1);
        cp_async_wait_all();
        __syncthreads();
        using SM = GroupSmem<L, T, TX, Scatter::NF, Scatter::NC>;
        double* acc = sm.acc[SM::ACCS == 2 ? ph & 1 : 0];
        const int32_t* nbr = sm.meta[ph % 3].nbr;
        for (int i = threadIdx.x; i < 8 * NC * NPB; i += FUSED_THREADS) {
            const double v = acc[i];
            if (v == 0) continue;
            acc[i] = 0;
            const int t = i / (NC * NPB), r = i - t * NC * NPB, c = r / NPB, e = r - c * NPB;
            const int64_t blk = nbr[t];
            if (c < NC0)
                atomicAdd(&outa[(blk * NC0 + c) * NPB + e], v);
            else
                atomicAdd(&outb[(blk * (NC - NC0) + (c - NC0)) * NPB + e], v);
        }
        if constexpr (SM::ACCS == 1) __syncthreads(); // the accumulator is clear
        cur = nxt;
        have = more;
        ++ph;
    }
}

} // namespace zmpm
