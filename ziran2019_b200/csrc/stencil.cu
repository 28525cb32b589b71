// ADMM's global operator as an assembled 125-entry node stencil.
//
// initMultiplierAndPreconditioner (AdmmSimulationFoam.h:407-505) builds
// K_ij = sum_p grad w_ip^T B_p grad w_jp once per substep (B_p of
// k_admm_init); every product of the substep's MINRES solves (several
// hundred) is then y_i = sum_j K_ij x_j for the three velocity components
// alike.  Node j lies within two cells of node i on each axis, so a row has
// 125 entries, stored [page][125][NPB]: entry o = 25 (dx + 2) + 5 (dy + 2) +
// (dz + 2) of a page's nodes is contiguous.
//
// Why assembled: the matrix-free product (hvp.cuh, AdmmOpModel) runs every
// particle's gather and scatter per product, about 0.19 ns per particle (0.096
// ms at 498k particles); the stencil reads 125 coefficients per node slot
// from L2 and needs no atomics, no accumulator pass and one grid barrier less
// per iteration.  The product is bound by the coefficient reads.
//
// Kernels
//  k_stencil_nbr       the 27 neighbour pages of every page
//  k_stencil_assemble  K from the particles, one CTA per particle group
//  k_stencil_pre       preconditioner m_i + K_ii (:477-503)
//  k_stencil_start     dvStep's right-hand side residual and Krylov start
//  k_mr_stencil        the persistent MINRES solve on the stencil
#include "krylov.cuh"
#include "stencil.cuh"

namespace zmpm {

// ------------------------------------------------------------- neighbours --
// nbr[27 b + t], t = 9 (dx + 1) + 3 (dy + 1) + (dz + 1): the block index of the
// page at offset (dx, dy, dz) from page b, or -1 where the grid has none.  The
// dense page table keeps entries of earlier substeps, so a hit has to be a
// current block of the same coordinates.
__global__ void k_stencil_nbr(const int4* __restrict__ block_page, int B, int px, int py, int pz, const int32_t* __restrict__ page_block,
    int32_t* __restrict__ nbr)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 27ll * B) return;
    const int b = (int)(q / 27), t = (int)(q - 27ll * b);
    const int4 p = block_page[b];
    const int x = p.x + t / 9 - 1, y = p.y + (t / 3) % 3 - 1, z = p.z + t % 3 - 1;
    int r = -1;
    if (x >= 0 && x < px && y >= 0 && y < py && z >= 0 && z < pz) {
        const int c = page_block[((int64_t)x * py + y) * pz + z];
        if (c >= 0 && c < B) {
            const int4 o = block_page[c];
            if (o.x == x && o.y == y && o.z == z) r = c;
        }
    }
    nbr[q] = r;
}

// --------------------------------------------------------------- assembly --
// Item (i, occupied cell): the cell's particles' sums of a . grad w_j over the
// 27 nodes j of the cell, a = B grad w_i, in registers, then one global add
// per entry.  The cell's particles share their nodes, so the adds are one per
// (cell, i, j) instead of one per (particle, i, j).
template <class L, class T, int CH>
struct AssembleSmem {
    T rec[9 * (CH + 1)]; // fractions 0-2, B 3-8
    int32_t cells[GroupCells<L>::WORDS];
    int32_t nbr[8];
};

template <class L, class T, int CH>
__global__ void __launch_bounds__(FUSED_THREADS) k_stencil_assemble(const int32_t* __restrict__ group_start,
    const int32_t* __restrict__ group_nbr, const int32_t* __restrict__ cells, int64_t cap, double dx, const T* __restrict__ frac,
    const T* __restrict__ B, T* __restrict__ K)
{
    constexpr int NPB = L::NPB, FS = CH + 1;
    __shared__ AssembleSmem<L, T, CH> sm;
    const int g = blockIdx.x;
    if (threadIdx.x < 8) sm.nbr[threadIdx.x] = group_nbr[8 * g + threadIdx.x];
    const int s0 = group_start[g], n = group_start[g + 1] - s0;
    for (int i = threadIdx.x; i < GroupCells<L>::WORDS; i += FUSED_THREADS) sm.cells[i] = cells[(int64_t)g * GroupCells<L>::WORDS + i];
    const uint8_t* occ = reinterpret_cast<const uint8_t*>(sm.cells + GroupCells<L>::OCC);
    const T inv_dx2 = T((1.0 / dx) * (1.0 / dx));
    for (int c0 = 0; c0 < n; c0 += CH) {
        const int c1 = c0 + CH < n ? c0 + CH : n;
        __syncthreads();
        for (int p = c0 + threadIdx.x; p < c1; p += blockDim.x) {
            const int64_t s = s0 + p;
            T* rc = sm.rec + (p - c0);
#pragma unroll
            for (int d = 0; d < 3; ++d) rc[d * FS] = frac[d * cap + s];
#pragma unroll
            for (int k = 0; k < 6; ++k) rc[(3 + k) * FS] = B[(int64_t)k * cap + s] * inv_dx2;
        }
        __syncthreads();
        const int nocc = sm.cells[GroupCells<L>::NOCC];
        for (int q = threadIdx.x; q < 27 * nocc; q += blockDim.x) {
            const int i = q / nocc, ce = occ[q - i * nocc];
            const int st = sm.cells[ce], e1 = sm.cells[ce + 1];
            const int p0 = (st > c0 ? st : c0) - c0;
            const int p1 = (e1 < c1 ? e1 : c1) - c0;
            if (p0 >= p1) continue;
            const int ix = i / 9, iy = (i / 3) % 3, iz = i % 3;
            T a[27];
#pragma unroll
            for (int m = 0; m < 27; ++m) a[m] = T(0);
            for (int p = p0; p < p1; ++p) {
                T w[3][3], dw[3][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) bspline_all(sm.rec[d * FS + p], w[d], dw[d]);
                const T wx = ix == 0 ? w[0][0] : (ix == 1 ? w[0][1] : w[0][2]), gx = ix == 0 ? dw[0][0] : (ix == 1 ? dw[0][1] : dw[0][2]);
                const T wy = iy == 0 ? w[1][0] : (iy == 1 ? w[1][1] : w[1][2]), gy = iy == 0 ? dw[1][0] : (iy == 1 ? dw[1][1] : dw[1][2]);
                const T wz = iz == 0 ? w[2][0] : (iz == 1 ? w[2][1] : w[2][2]), gz = iz == 0 ? dw[2][0] : (iz == 1 ? dw[2][1] : dw[2][2]);
                const T g0 = gx * wy * wz, g1 = wx * gy * wz, g2 = wx * wy * gz;
                const T* b = sm.rec + 3 * FS + p;
                const T a0 = b[0] * g0 + b[FS] * g1 + b[2 * FS] * g2;
                const T a1 = b[FS] * g0 + b[3 * FS] * g1 + b[4 * FS] * g2;
                const T a2 = b[2 * FS] * g0 + b[4 * FS] * g1 + b[5 * FS] * g2;
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const T u = a0 * (w[1][j] * w[2][k]);
                        const T v = a1 * (dw[1][j] * w[2][k]) + a2 * (w[1][j] * dw[2][k]);
#pragma unroll
                        for (int m = 0; m < 3; ++m) a[9 * m + 3 * j + k] += dw[0][m] * u + w[0][m] * v;
                    }
            }
            const int lx = ce >> (L::YB + L::ZB), ly = (ce >> L::ZB) & (L::BY - 1), lz = ce & (L::BZ - 1);
            int e;
            const int t = win_slot<L>(lx + ix, ly + iy, lz + iz, e);
            // entry (m, j, k) of the cell sits at offset (m - ix, j - iy, k - iz) of row i
            T* row = K + ((int64_t)sm.nbr[t] * STENCIL + (2 - ix) * 25 + (2 - iy) * 5 + (2 - iz)) * NPB + e;
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) atomicAdd(row + (25 * m + 5 * j + k) * NPB, a[9 * m + 3 * j + k]);
        }
    }
}

template <int NPB, class T>
__global__ void __launch_bounds__(ND_THREADS) k_stencil_pre(int64_t nn, const double* __restrict__ gm, const T* __restrict__ K,
    double* __restrict__ pre)
{
    const int64_t n = (int64_t)blockIdx.x * ND_THREADS + threadIdx.x;
    if (n >= nn) return;
    const int64_t b = n / NPB;
    pre[n] = gm[n] + (double)K[(b * STENCIL + STENCIL / 2) * NPB + (n - b * NPB)];
}

// ---------------------------------------------------------------- product --
// One page's product: threads are (z-row of four nodes, part of the 25 (dx, dy)
// offsets).  A part's step loads the five dz coefficients of its row (16-byte
// loads; rows without mass are skipped, their coefficients are zero) and, per
// component, the row's eight window values, for 60 FMAs.  FP64 sums: first
// over the part, then the parts in a fixed order.
template <class L>
struct StencilSmem {
    static constexpr int WX = L::BX + 4, WY = L::BY + 4;
    // pitches (in doubles) that put the eight rows of a quarter-warp's 16-byte
    // loads in distinct banks
    static constexpr int ROW = 10, SLAB = WY * ROW + 8, COMP = WX * SLAB;
    static constexpr int ROWS = L::NPB / 4, SUB = 32 / ROWS, WARPS = FUSED_THREADS / 32, PARTS = SUB * WARPS;
    __align__(16) double win[3 * COMP];
    __align__(16) double part[WARPS][3][L::NPB];
    int32_t nbr[27];
};

__device__ __forceinline__ void load_quad(const float* p, float v[4])
{
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
}
__device__ __forceinline__ void load_quad(const double* p, double v[4])
{
    const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}

// y[c] = sum_j K_ij x_j[c] of node threadIdx.x of page b (threads below NPB);
// all threads call it.  x is read through L2 (other CTAs of a persistent
// kernel write it).  The window keeps x; node e's own value is own(sm, e, c).
template <class L, class TK>
__device__ __forceinline__ void stencil_page(StencilSmem<L>& sm, const TK* __restrict__ K, const int32_t* __restrict__ nbr, int b,
    const double* __restrict__ gm, const double* x, double y[3])
{
    using S = StencilSmem<L>;
    constexpr int NPB = L::NPB;
    __syncthreads(); // the previous page's sums are read
    if (threadIdx.x < 27) sm.nbr[threadIdx.x] = nbr[27 * (int64_t)b + threadIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = lane % S::ROWS, part = warp * S::SUB + lane / S::ROWS;
    const double2 ma = __ldg(reinterpret_cast<const double2*>(gm + (int64_t)b * NPB + 4 * row));
    const double2 mb = __ldg(reinterpret_cast<const double2*>(gm + (int64_t)b * NPB + 4 * row) + 1);
    const bool act = ma.x != 0 || ma.y != 0 || mb.x != 0 || mb.y != 0;
    __syncthreads();
    for (int q = threadIdx.x; q < 3 * S::WX * S::WY * 4; q += FUSED_THREADS) {
        const int h = q & 3, r = q >> 2, wy = r % S::WY, wx = (r / S::WY) % S::WX, c = r / (S::WY * S::WX);
        const int gx = wx - 2, gy = wy - 2, gz = 2 * h - 2; // first node of the pair, relative to the page
        const int tx = gx < 0 ? 0 : (gx >= L::BX ? 2 : 1), ty = gy < 0 ? 0 : (gy >= L::BY ? 2 : 1), tz = h == 0 ? 0 : (h == 3 ? 2 : 1);
        const int nb = sm.nbr[9 * tx + 3 * ty + tz];
        double2 v = make_double2(0.0, 0.0);
        if (nb >= 0)
            v = __ldcg(reinterpret_cast<const double2*>(
                x + ((int64_t)nb * 3 + c) * NPB + L::elem(gx & (L::BX - 1), gy & (L::BY - 1), gz & (L::BZ - 1))));
        *reinterpret_cast<double2*>(sm.win + c * S::COMP + wx * S::SLAB + wy * S::ROW + 2 * h) = v;
    }
    __syncthreads();
    double acc[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int z = 0; z < 4; ++z) acc[c][z] = 0;
    if (act) {
        const TK* kp = K + (int64_t)b * STENCIL * NPB + 4 * row;
        const double* wr = sm.win + (row / L::BY) * S::SLAB + (row % L::BY) * S::ROW;
#pragma unroll 1
        for (int p = part; p < 25; p += S::PARTS) {
            TK kv[5][4];
#pragma unroll
            for (int d = 0; d < 5; ++d) load_quad(kp + (5 * p + d) * NPB, kv[d]);
            const double* wp = wr + (p / 5) * S::SLAB + (p % 5) * S::ROW;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double xs[8];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const double2 v = *reinterpret_cast<const double2*>(wp + c * S::COMP + 2 * h);
                    xs[2 * h] = v.x;
                    xs[2 * h + 1] = v.y;
                }
#pragma unroll
                for (int d = 0; d < 5; ++d)
#pragma unroll
                    for (int z = 0; z < 4; ++z) acc[c][z] += (double)kv[d][z] * xs[z + d];
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int z = 0; z < 4; ++z)
#pragma unroll
            for (int o = S::ROWS; o < 32; o <<= 1) acc[c][z] += __shfl_xor_sync(0xffffffffu, acc[c][z], o);
    if (lane < S::ROWS)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<double2*>(&sm.part[warp][c][4 * row + 2 * h]) = make_double2(acc[c][2 * h], acc[c][2 * h + 1]);
    __syncthreads();
    if (threadIdx.x < NPB)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            y[c] = 0;
#pragma unroll
            for (int w = 0; w < S::WARPS; ++w) y[c] += sm.part[w][c][threadIdx.x];
        }
}
template <class L>
__device__ __forceinline__ double own(const StencilSmem<L>& sm, int e, int c)
{
    using S = StencilSmem<L>;
    const int lx = e >> (L::YB + L::ZB), ly = (e >> L::ZB) & (L::BY - 1), lz = e & (L::BZ - 1);
    return sm.win[c * S::COMP + (lx + 2) * S::SLAB + (ly + 2) * S::ROW + lz + 2];
}

// Start of dvStep's MINRES from the current dv (Minres.h:73-98), as
// k_admm_start with the product of dv in the same pass: r = project(rhs -
// (m dv + K dv)); Q0 = r, Z0 = r / pre; partial z . r.
template <class L, class TK>
__global__ void __launch_bounds__(FUSED_THREADS, 4) k_stencil_start(int B, const TK* __restrict__ K, const int32_t* __restrict__ nbr,
    const double* __restrict__ gm, const int8_t* __restrict__ col, const double* __restrict__ P6, const double* __restrict__ rhs,
    const double* __restrict__ dv, KrylovBufs kb, double* __restrict__ part, SolverScalars* __restrict__ sc)
{
    constexpr int NPB = L::NPB;
    __shared__ StencilSmem<L> sm;
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->rel_tol = 0.5; // AdmmSimulationFoam.h:779-782
    const int64_t nn = (int64_t)B * NPB;
    double acc = 0;
    for (int b = blockIdx.x; b < B; b += gridDim.x) {
        double y[3];
        stencil_page<L, TK>(sm, K, nbr, b, gm, dv, y);
        if (threadIdx.x >= NPB) continue;
        const int64_t n = (int64_t)b * NPB + threadIdx.x;
        const double m = gm[n];
        double r[3];
        for (int k = 0; k < 3; ++k) r[k] = (m != 0) ? rhs[vidx<NPB>(n, k)] - (m * own<L>(sm, threadIdx.x, k) + y[k]) : 0.0;
        if (m != 0) project3(col, P6, nn, n, r);
        for (int k = 0; k < 3; ++k) {
            const int64_t i = vidx<NPB>(n, k);
            const double z = (m != 0) ? r[k] / kb.pre[n] : 0.0;
            kb.Q[0][i] = r[k];
            kb.Z[0][i] = z;
            kb.Z[1][i] = 0; // massless nodes keep this zero
            acc += z * r[k];
        }
    }
    acc = block_sum_fused(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// The whole MINRES solve (Minres.h:69-175) on the stencil in one cooperative
// launch, as k_mr_persistent but with the product and the operator pass (the
// deferred direction of iteration k - 1, W = project(m Z_k + K Z_k)) in one
// pass over a CTA's own pages: two grid barriers per iteration.
template <class L, class TK>
__global__ void __launch_bounds__(FUSED_THREADS, 4) k_mr_stencil(NodeGeom ng, int B, const TK* __restrict__ K,
    const int32_t* __restrict__ nbr, const double* __restrict__ gm, const int8_t* __restrict__ col, const double* __restrict__ P6, KrylovBufs kb,
    double* __restrict__ part_a, double* __restrict__ part_b, SolverScalars* __restrict__ sc, int kmax, GridSync* __restrict__ gs,
    long long limit, int32_t* __restrict__ flags)
{
    if (sc->newton_done || !sc->kactive) return;
    constexpr int NPB = L::NPB;
    __shared__ StencilSmem<L> sm;
    __shared__ double mst[MST_N];
    int k = sc->kit;
    if (threadIdx.x == 0) mr_load(sc, mst, k);
    __syncthreads();
    const int nit = sc->nit;
    const double local_tol = sc->local_tol;
    unsigned epoch = 0;
    for (;;) {
        double* w = sel3(kb.Q, (k + 1) % 3);
        const double* zk = sel2(kb.Z, k & 1);
        const MrPending pd = mr_pending(kb, mst + MST_PEND, k);
        const double ibeta = mr_scale(mst[MR_BETA_KP1]);
        double acc = 0;
        for (int b = blockIdx.x; b < B; b += gridDim.x) {
            // the node pass's operands, loaded before the product
            const bool mine = threadIdx.x < NPB;
            const int64_t n = (int64_t)b * NPB + (mine ? threadIdx.x : 0);
            const double m = mine ? gm[n] : 0.0;
            double mv[3] = { 0, 0, 0 }, xv[3] = { 0, 0, 0 };
            if (m != 0 && pd.on)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int64_t i = vidx<NPB>(n, c);
                    mv[c] = mr_direction(pd, i);
                    xv[c] = pd.hasx ? kb.x[i] : 0.0;
                }
            double y[3];
            stencil_page<L, TK>(sm, K, nbr, b, gm, zk, y);
            if (m == 0) continue;
            double o[3], z[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int64_t i = vidx<NPB>(n, c);
                if (pd.on) {
                    pd.out[i] = mv[c];
                    kb.x[i] = xv[c] + pd.t * mv[c];
                }
                z[c] = own<L>(sm, threadIdx.x, c) * ibeta;
                o[c] = m * z[c] + y[c] * ibeta;
            }
            project3(col, P6, ng.nn, n, o);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                w[vidx<NPB>(n, c)] = o[c];
                acc += o[c] * z[c];
            }
        }
        acc = block_sum_fused(acc);
        if (threadIdx.x == 0) part_a[blockIdx.x] = acc;
        if (!grid_sync(gs, epoch, limit, flags)) return;
        double rnorm;
        if (!mr_lanczos<NPB>(ng, gm, kb, k, mst, part_a, part_b, gs, epoch, limit, flags, rnorm)) return;
        ++k;
        const bool go = !(rnorm < local_tol || k >= kmax);
        mr_store(sc, mst, k, nit, rnorm, go);
        if (!go) return;
    }
}

// -------------------------------------------------------------- host side --
// The stencil's product costs the reads of its coefficients, the matrix-free one
// its particles and about 192 particles' worth per group; the rule is a limit of
// bytes per such unit (a dense scene has about 150, a spray of single particles
// up to 2600).  Coefficients that stay in L2 win at any density measured; above
// that sparse scenes lose.  Substeps of four iterations with 20 products each,
// matrix-free / stencil, against MB of coefficients and bytes per unit:
//   FP64  43.5, 665: 3.13 / 2.35 ms;  104, 625: 4.15 / 4.33;  168, 629: 5.7 / 7.1;
//         215, 216: 12.0 / 11.4;  202, 321: 8.5 / 9.4;  182, 489: 6.3 / 7.8
//   FP32  99.6, 426: 5.9 / 5.3;  164, 368: 8.0 / 8.3;  319, 345: 16.1 / 15.6;
//         108, 247: 7.5 / 6.5;  287, 201: 22.0 / 17.2
// Few iterations do not change the side: the assembly costs less than the gathers
// it saves in the preconditioner (498k particles, one iteration of 3 products: 5.7
// / 2.7 ms).
bool stencil_pays(const Ctx* ctx)
{
    const double bytes = (double)ctx->B * STENCIL * ctx->npb() * (ctx->mixed ? sizeof(float) : sizeof(double));
    const double units = (double)ctx->P + 192.0 * (double)ctx->G;
    return bytes <= (bytes <= 96e6 ? 1024.0 : (ctx->mixed ? 352.0 : 256.0)) * units;
}

template <class L, class T>
static int stencil_build_impl(Ctx* ctx)
{
    cudaStream_t st = ctx->stream;
    const int64_t nn = ctx->B * L::NPB;
    const int B = (int)ctx->B;
    T* K = ctx->adm_K.as<T>();
    k_stencil_nbr<<<(unsigned)((27ll * B + 255) / 256), 256, 0, st>>>(ctx->block_page.as<int4>(), B, ctx->pages[0], ctx->pages[1], ctx->pages[2],
        ctx->page_block.as<int32_t>(), ctx->adm_nbr.as<int32_t>());
    ZMPM_CUDA(cudaMemsetAsync(K, 0, (size_t)nn * STENCIL * sizeof(T), st));
    k_stencil_assemble<L, T, sizeof(T) == 4 ? 512 : 256><<<(unsigned)ctx->G, FUSED_THREADS, 0, st>>>(ctx->group_start.as<int32_t>(),
        ctx->group_nbr.as<int32_t>(), ctx->group_cells.as<int32_t>(), ctx->Pcap, ctx->cfg.dx, ctx->frac.as<T>(), ctx->adm_B.as<T>(), K);
    k_stencil_pre<L::NPB, T><<<(unsigned)((nn + ND_THREADS - 1) / ND_THREADS), ND_THREADS, 0, st>>>(nn, ctx->gm.as<double>(), K,
        ctx->adm_pre.as<double>());
    g_kernel_launches += 3;
    return ZMPM_OK;
}

// Allocates the operator's arrays; false (the caller stays matrix-free) when
// the device has no room for them.
bool stencil_reserve(Ctx* ctx)
{
    const size_t bytes = (size_t)ctx->B * ctx->npb() * STENCIL * (ctx->mixed ? sizeof(float) : sizeof(double));
    if (ctx->adm_K.ensure(bytes) == cudaSuccess && ctx->adm_nbr.ensure((size_t)ctx->B * 27 * sizeof(int32_t)) == cudaSuccess) return true;
    cudaGetLastError(); // the failed allocation is not the substep's error
    return false;
}

int launch_stencil_build(Ctx* ctx)
{
    if (ctx->layout == 1) return ctx->mixed ? stencil_build_impl<Layout244, float>(ctx) : stencil_build_impl<Layout244, double>(ctx);
    return ctx->mixed ? stencil_build_impl<Layout444, float>(ctx) : stencil_build_impl<Layout444, double>(ctx);
}

template <class L, class T>
static int stencil_start_impl(Ctx* ctx, const KrylovBufs& kb, double* part, SolverScalars* sc, int* parts)
{
    const int grid = (int)std::min<int64_t>(ctx->B, RED_MAX_CTAS);
    *parts = grid;
    k_stencil_start<L, T><<<grid, FUSED_THREADS, 0, ctx->stream>>>((int)ctx->B, ctx->adm_K.as<T>(), ctx->adm_nbr.as<int32_t>(),
        ctx->gm.as<double>(), ctx->collided.as<int8_t>(), ctx->proj.as<double>(), ctx->adm_rhs.as<double>(), ctx->dv.as<double>(), kb, part, sc);
    ++g_kernel_launches;
    return ZMPM_OK;
}
int launch_stencil_start(Ctx* ctx, const KrylovBufs& kb, double* part, SolverScalars* sc, int* parts)
{
    if (ctx->layout == 1)
        return ctx->mixed ? stencil_start_impl<Layout244, float>(ctx, kb, part, sc, parts) : stencil_start_impl<Layout244, double>(ctx, kb, part, sc, parts);
    return ctx->mixed ? stencil_start_impl<Layout444, float>(ctx, kb, part, sc, parts) : stencil_start_impl<Layout444, double>(ctx, kb, part, sc, parts);
}

template <class L, class T>
static int stencil_minres_impl(Ctx* ctx, const NodeGeom& ng, const KrylovBufs& kb, double* pA, double* pB, SolverScalars* sc, int kmax)
{
    return launch_resident(ctx, ctx->stream, true, ctx->B, 0, k_mr_stencil<L, T>, ng, (int)ctx->B, ctx->adm_K.as<T>(), ctx->adm_nbr.as<int32_t>(),
        ctx->gm.as<double>(), ctx->collided.as<int8_t>(), ctx->proj.as<double>(), kb, pA, pB, sc, kmax, ctx->gsync.as<GridSync>(),
        ctx->spin_limit, &ctx->counters.as<DevCounters>()->flags);
}
int launch_stencil_minres(Ctx* ctx, const NodeGeom& ng, const KrylovBufs& kb, double* pA, double* pB, SolverScalars* sc, int kmax)
{
    if (ctx->layout == 1)
        return ctx->mixed ? stencil_minres_impl<Layout244, float>(ctx, ng, kb, pA, pB, sc, kmax)
                          : stencil_minres_impl<Layout244, double>(ctx, ng, kb, pA, pB, sc, kmax);
    return ctx->mixed ? stencil_minres_impl<Layout444, float>(ctx, ng, kb, pA, pB, sc, kmax)
                      : stencil_minres_impl<Layout444, double>(ctx, ng, kb, pA, pB, sc, kmax);
}

} // namespace zmpm
