// Parts shared by the persistent Krylov kernels (solver.cu, stencil.cu): the
// collision projection, the solvers' buffers and scalars, MINRES's deferred
// direction and Givens update, fixed-order reductions and the bounded grid
// barrier.
#pragma once
#include <algorithm>
#include <utility>

#include "fused.cuh"
#include "internal.cuh"
#include "node.cuh"

namespace zmpm {

__device__ __forceinline__ void project3(const int8_t* col, const double* P6, int64_t nn, int64_t n, double v[3])
{
    if (!col[n]) return;
    double p00 = P6[n], p01 = P6[nn + n], p02 = P6[2 * nn + n], p11 = P6[3 * nn + n], p12 = P6[4 * nn + n], p22 = P6[5 * nn + n];
    double a = v[0], b = v[1], c = v[2];
    v[0] = p00 * a + p01 * b + p02 * c;
    v[1] = p01 * a + p11 * b + p12 * c;
    v[2] = p02 * a + p12 * b + p22 * c;
}

// Solver buffers of one linear solve.  MINRES rotates its three Lanczos
// vectors Q, three search directions M and two preconditioned vectors Z by the
// iteration index k read from device memory, so the same kernels (and the same
// graph body) serve every iteration.
struct KrylovBufs {
    double *x, *r, *p, *q, *tmp;      // CG
    double *Q[3], *M[3], *Z[2];       // MINRES
    float* Zf[2];                     // FP32 node-major copies of Z ([B][NPB][4]) for the FP32 product (MIXED MINRES), or null
    float* pf;                        // FP32 node-major copy of p for the FP32 product (MIXED CG), or null
    double* hacc;                     // Hessian accumulator
    const double* pre;                // diagonal preconditioner per node (the mass for Newton)
};

struct NewtonParams {
    int32_t minres, kmax, nmax;
    int32_t escalate;                 // MIXED: FP64 residual once the FP32 one stalls
    double tol, abs_tol, tol_scale, dt;
};

// Role selection by iteration index without indexing the parameter arrays at
// run time (which would copy the kernel parameters to local memory).
__device__ __forceinline__ double* sel3(double* const (&a)[3], int i) { return i == 0 ? a[0] : (i == 1 ? a[1] : a[2]); }
template <class T>
__device__ __forceinline__ T* sel2(T* const (&a)[2], int i) { return i == 0 ? a[0] : a[1]; }

// MINRES keeps its Lanczos vectors Q_j and preconditioned vectors Z_j
// unnormalised (Minres.h:170-173 divides them by beta_j at the end of
// iteration j - 1); every reader scales by 1 / beta_j.  beta_j = 0 leaves them
// as they are, as there.  The node passes multiply by reciprocals formed once
// per thread: an FP64 division is a chain of about 300 cycles, and the 24 of a
// thread's two nodes were most of a small scene's operator pass (7.7 of 39 us
// per iteration at 33k particles).
__device__ __forceinline__ double mr_scale(double beta) { return beta > 0 ? 1.0 / beta : 1.0; }

// The search direction of iteration j = k - 1 (Minres.h:167-170):
// M_j = (Z_j - delta M_{j-1} - epsilon M_{j-2}) / gamma, then x += t M_j.
// The Lanczos step computes its scalars; the vector update runs in the next
// iteration's operator pass or, after the last iteration, where the solve's x
// is used (newton_step, k_admm_dv_update).  M_{-1}, M_{-2} and the first x are
// zero and not stored: has1, has2 and hasx say which vectors exist.
struct MrPending {
    const double *z, *m1, *m2;
    double* out;
    double delta, eps, t, ibeta, igamma;
    bool on, has1, has2, hasx;
};
__device__ __forceinline__ MrPending mr_pending(const KrylovBufs& kb, const double* pend, int k)
{
    MrPending p;
    p.on = k > 0;
    p.has1 = k > 1;
    p.has2 = k > 2;
    p.hasx = k > 1;
    p.z = sel2(kb.Z, (k + 1) & 1);   // Z_{k-1}, unnormalised
    p.m1 = sel3(kb.M, (k + 1) % 3);  // M_{k-2}
    p.m2 = sel3(kb.M, k % 3);        // M_{k-3}
    p.out = sel3(kb.M, (k + 2) % 3); // M_{k-1}
    p.delta = pend[0];
    p.eps = pend[1];
    p.igamma = p.on ? 1.0 / pend[2] : 0.0;
    p.t = pend[3];
    p.ibeta = p.on ? mr_scale(pend[4]) : 0.0; // beta_{k-1}
    return p;
}
__device__ __forceinline__ double mr_direction(const MrPending& p, int64_t i)
{
    const double m1 = p.has1 ? p.m1[i] : 0.0, m2 = p.has2 ? p.m2[i] : 0.0;
    return (p.z[i] * p.ibeta - p.delta * m1 - p.eps * m2) * p.igamma;
}

// The Givens update of MINRES iteration k (Minres.h:151-175): from the state
// cur of iteration k (Minres.h:16-24), alpha = Z_k . W, beta_k and dz =
// Z~_{k+1} . Q~_{k+1}, the state of iteration k + 1 into nx and the deferred
// search direction's delta, epsilon, gamma, t and beta into pend; returns the
// preconditioned residual norm.
__device__ __forceinline__ double mr_givens(const double* cur, double alpha, double beta_k, double dz, double* nx, double* pend)
{
    const double beta_kp1 = sqrt(dz > 0 ? dz : 0.0);
    // Gkm2 = Gkm1, Gkm1 = Gk
    double c2 = cur[MR_GC1], s2 = cur[MR_GS1], c1 = cur[MR_GC0], s1 = cur[MR_GS0];
    double e0 = c2 * 0 - s2 * beta_k, e1 = s2 * 0 + c2 * beta_k;
    const double epsilon = e0;
    double d0 = c1 * e1 - s1 * alpha, d1 = s1 * e1 + c1 * alpha;
    const double delta = d0;
    double t0 = d1, t1 = beta_kp1;
    double c0 = 1, s0 = 0;
    {
        double dd = t0 * t0 + t1 * t1;
        double sd = sqrt(dd);
        if (sd != 0) {
            double tt = 1 / sd;
            c0 = t0 * tt;
            s0 = -t1 * tt;
        }
    }
    const double gamma = c0 * t0 - s0 * t1;
    const double r0 = cur[MR_RHS0], r1 = cur[MR_RHS1];
    const double tk = c0 * r0 - s0 * r1;
    const double residual = s0 * r0 + c0 * r1;
    nx[MR_GC0] = c0;
    nx[MR_GS0] = s0;
    nx[MR_GC1] = c1;
    nx[MR_GS1] = s1;
    nx[MR_GC2] = c2;
    nx[MR_GS2] = s2;
    nx[MR_RHS0] = residual;
    nx[MR_RHS1] = 0;
    nx[MR_BETA_KP1] = beta_kp1;
    pend[0] = delta;
    pend[1] = epsilon;
    pend[2] = gamma;
    pend[3] = tk;
    pend[4] = beta_k;
    return residual < 0 ? -residual : residual;
}

// Block sum for FUSED_THREADS threads; the result in every thread.
__device__ __forceinline__ double block_sum_fused(double v)
{
    __shared__ double ws[FUSED_THREADS / 32];
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) ws[w] = v;
    __syncthreads();
    double t = 0;
#pragma unroll
    for (int i = 0; i < FUSED_THREADS / 32; ++i) t += ws[i];
    return t;
}
// Sum of n partials written by other CTAs of this kernel (read through L2), in
// a fixed order identical in every CTA.
__device__ __forceinline__ double reduce_partials_fused(const double* part, int n)
{
    double s = 0;
    for (int i = threadIdx.x; i < n; i += FUSED_THREADS) s += __ldcg(part + i);
    return block_sum_fused(s);
}

// Bounded grid-wide barrier number `epoch` (counted from 0 by every CTA alike):
// each CTA adds itself to one running count and waits until the count shows all
// of them, so a barrier is one release and one acquire apart (a separate
// generation word, written by the last arrival, cost another trip to L2; with
// its fences 2.3 us on 592 CTAs).  The count's top bit is the abort flag.  Returns false
// in every thread of the CTA when this CTA gave up after `limit` polls or
// another CTA did; the caller then returns.
__device__ __forceinline__ bool grid_sync(GridSync* gs, unsigned& epoch, long long limit, int32_t* flags)
{
    __shared__ int ok;
    ++epoch;
    __syncthreads();
    if (threadIdx.x == 0) {
        constexpr unsigned long long ABORT = 1ull << 63;
        const unsigned long long target = (unsigned long long)epoch * gridDim.x;
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&gs->count), "l"(1ull) : "memory");
        int good = 1;
        long long it = 0;
        for (;;) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&gs->count) : "memory");
            if (v & ABORT) {
                good = 0;
                break;
            }
            if (v >= target) break;
            if (++it > limit) {
                atomicOr(flags, (int32_t)FLAG_TIMEOUT);
                atomicOr(&gs->count, ABORT);
                good = 0;
                break;
            }
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// ---------------------------------------- MINRES iteration, shared parts --
// Nodes per thread and step in the node passes (their loads all issue before
// the arithmetic: the passes are latency-bound).
constexpr int MR_UNROLL = 2;

// A persistent MINRES kernel's state in shared memory: the MINRES state of
// iteration k (Minres.h:16-24), the deferred direction's scalars, beta_{k-1}
// and the residual norm.
constexpr int MST_PEND = 12, MST_BETA_KM1 = 17, MST_RNORM = 18, MST_N = 19;
__device__ __forceinline__ void mr_load(const SolverScalars* sc, double* mst, int k) // one thread
{
    for (int i = 0; i < 12; ++i) mst[i] = sc->mr[k & 1][i];
    for (int i = 0; i < 5; ++i) mst[MST_PEND + i] = sc->pend[i];
    mst[MST_BETA_KM1] = sc->mr[(k + 1) & 1][MR_BETA_KP1];
}
__device__ __forceinline__ void mr_init(double* mst, double rnorm) // one thread: the state before iteration 0
{
    for (int i = 0; i < MST_N; ++i) mst[i] = 0;
    mst[MR_GC0] = mst[MR_GC1] = mst[MR_GC2] = 1;
    mst[MR_RHS0] = mst[MR_BETA_KP1] = rnorm;
}
// CTA 0 stores the state after an iteration (k counts it already).
__device__ __forceinline__ void mr_store(SolverScalars* sc, const double* mst, int k, int nit, double rnorm, bool go)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int i = 0; i < 12; ++i) sc->mr[k & 1][i] = mst[i];
    for (int i = 0; i < 5; ++i) sc->pend[i] = mst[MST_PEND + i];
    sc->rnorm = rnorm;
    sc->krylov_iters += 1;
    sc->hvp_count += 1;
    if (nit < 64) sc->kcount[nit] += 1;
    sc->kit = k;
    if (!go) sc->kactive = 0;
}

// The Lanczos step of iteration k after the operator pass (its partials of
// Z_k . W in part_a complete): Q~_{k+1} = W - alpha Q_k - beta_k Q_{k-1},
// Z~_{k+1} = Q~_{k+1} / pre (and its FP32 copy), a partial of Z~_{k+1} .
// Q~_{k+1}, a grid barrier, and the Givens update of mst.  Returns false when
// a barrier gave up.
template <int NPB>
__device__ __forceinline__ bool mr_lanczos(NodeGeom ng, const double* __restrict__ gm, const KrylovBufs& kb, int k, double* mst,
    const double* part_a, double* part_b, GridSync* gs, unsigned& epoch, long long limit, int32_t* flags, double& rnorm)
{
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    const double alpha = reduce_partials_fused(part_a, gridDim.x);
    const double beta_k = mst[MR_BETA_KP1];
    const double ak = alpha * mr_scale(beta_k), bk = beta_k * mr_scale(mst[MST_BETA_KM1]);
    const bool first = k == 0; // Q_{-1} = 0 is not stored
    // (W may come from other CTAs: ordinary loads, not the read-only path)
    double* qkp1 = sel3(kb.Q, (k + 1) % 3);
    const double* qk = sel3(kb.Q, k % 3);
    const double* qkm1 = sel3(kb.Q, (k + 2) % 3);
    double* zout = sel2(kb.Z, (k + 1) & 1);
    float* zfout = sel2(kb.Zf, (k + 1) & 1);
    double acc = 0;
    for (int64_t n = t0; n < ng.nn; n += MR_UNROLL * nt) {
        int64_t nn2[MR_UNROLL];
        double mm[MR_UNROLL];
#pragma unroll
        for (int u = 0; u < MR_UNROLL; ++u) {
            const bool in = n + u * nt < ng.nn;
            nn2[u] = in ? n + u * nt : n;
            mm[u] = in ? gm[nn2[u]] : 0.0;
        }
        double pre[MR_UNROLL], qa[MR_UNROLL][3], qb[MR_UNROLL][3], qc[MR_UNROLL][3];
#pragma unroll
        for (int u = 0; u < MR_UNROLL; ++u) {
            pre[u] = kb.pre[nn2[u]];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int64_t i = vidx<NPB>(nn2[u], c);
                qa[u][c] = qkp1[i];
                qb[u][c] = qk[i];
                qc[u][c] = first ? 0.0 : qkm1[i];
            }
        }
#pragma unroll
        for (int u = 0; u < MR_UNROLL; ++u) {
            if (mm[u] == 0) continue;
            float zf[3];
            const double ipre = 1.0 / pre[u];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int64_t i = vidx<NPB>(nn2[u], c);
                double q = qa[u][c];
                q -= ak * qb[u][c];
                q -= bk * qc[u][c];
                qkp1[i] = q;
                const double z = q * ipre;
                zout[i] = z;
                zf[c] = (float)z;
                acc += z * q;
            }
            if (zfout) reinterpret_cast<float4*>(zfout)[nn2[u]] = make_float4(zf[0], zf[1], zf[2], 0.f);
        }
    }
    acc = block_sum_fused(acc);
    if (threadIdx.x == 0) part_b[blockIdx.x] = acc;
    if (!grid_sync(gs, epoch, limit, flags)) return false;
    const double dz = reduce_partials_fused(part_b, gridDim.x);
    if (threadIdx.x == 0) {
        double nx[12] = {};
        mst[MST_RNORM] = mr_givens(mst, alpha, beta_k, dz, nx, mst + MST_PEND);
        for (int i = 0; i < 12; ++i) mst[i] = nx[i];
        mst[MST_BETA_KM1] = beta_k;
    }
    __syncthreads();
    rnorm = mst[MST_RNORM];
    return true;
}

// A kernel of as many CTAs of FUSED_THREADS threads as fit on the device at
// once, or `useful` (the CTAs its work can occupy; fewer make barriers cheaper)
// if that is less; `smem`: its dynamic shared memory.  coop: cooperative, so
// that all CTAs are co-resident, which the grid barrier needs (the launch fails
// rather than oversubscribes; GridSync must be zero).  The CTAs that fit are
// found once per kernel.
template <class... P, class... A>
int launch_resident(Ctx* ctx, cudaStream_t st, bool coop, int64_t useful, size_t smem, void (*kern)(P...), A&&... args)
{
    int& blocks = ctx->coop_blocks[reinterpret_cast<const void*>(kern)];
    if (blocks <= 0) {
        int per_sm = 0, sms = 0;
        if (smem > 0) ZMPM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        ZMPM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, FUSED_THREADS, smem));
        ZMPM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
        blocks = std::min(per_sm * sms, RED_MAX_CTAS);
        if (blocks <= 0) {
            ctx->err = "a kernel does not fit on this device";
            return ZMPM_CUDA_ERROR;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(blocks, useful)));
    cfg.blockDim = dim3(FUSED_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = coop ? 1 : 0;
    ZMPM_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
    ++g_kernel_launches;
    return ZMPM_OK;
}

// CTAs that a pass over the particles in pieces can occupy: about PIECE_MIN
// particles' worth of work each.
constexpr int PIECE_MIN = 32;
inline int64_t useful_ctas(const Ctx* ctx, int K) { return (ctx->P + (int64_t)K * ctx->G + PIECE_MIN - 1) / PIECE_MIN; }

} // namespace zmpm
