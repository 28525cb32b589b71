// Particle <-> grid transfers of the implicit substep (helpers in xfer.cuh).
//
// Kernels
//  k_p2g_fused particlesToGridHelper<APIC> (MpmSimulationBase.cpp:563-608)
//  k_force   rasterizeForceToTVStack (MpmForceBase.cpp:102-152) of ADMM's
//            right-hand side
//  k_force_fused  the explicit substep's stress and force scatter
//  k_update_fused  updatePositionBasedState + rasterizeForceToTVStack in one
//            pass (gather of grad v, F, stress and Hessian scratch, force scatter)
//  k_product  MpmForceBase::addScaledForceDifferential (MpmForceBase.cpp:259-302):
//            G2P of grad(dv), dS = V0 dP Fn^T, P2G of dS grad w in one pass;
//            and ADMM's global operator in the same form
//  k_g2p     gridToParticlesHelper<APIC> (MpmSimulationBase.cpp:906-1016) +
//            evolveStrain + applyPlasticity (:1018-1030)
#include "admm.cuh"
#include "eig3.cuh"
#include "fused.cuh"
#include "hvp.cuh"
#include "krylov.cuh"
#include "xfer.cuh"

namespace zmpm {

// ------------------------------------------------------------------ P2G ----
// APIC P2G as a fused kernel (fused.cuh): phase 1 writes each particle's cell
// fractions (also to `frac`, for the Newton kernels), its mass and the affine
// form of its momentum; phase 2 (AffineScatter) sums them into the window by
// (component, occupied cell) items.  T: arithmetic (FP32 in MIXED contexts);
// the window is flushed into the FP64 grid sums.
template <class L, class T>
struct P2gPhase1 {
    const double* pd;
    int64_t cap;
    const short4* base;
    double inv_dx;
    T tdx;
    T* frac;

    template <int FS>
    __device__ __forceinline__ void run(const void*, int64_t s, T* rc) const
    {
        const short4 b = base[s];
        T fr[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double d0 = inv_dx * pd[(PD_X + d) * cap + s] - (double)((&b.x)[d]);
            fr[d] = (T)d0;
            frac[d * cap + s] = fr[d];
            rc[d * FS] = fr[d];
        }
        const double mass = pd[PD_M * cap + s];
        rc[3 * FS] = (T)mass;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            T mC[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) mC[q] = (T)(mass * pd[(PD_C + 3 * r + q) * cap + s]);
            const T mv = (T)(mass * pd[(PD_V + r) * cap + s]);
            rc[(4 + 4 * r) * FS] = mv + tdx * (mC[0] * (T(1) - fr[0]) + mC[1] * (T(1) - fr[1]) + mC[2] * (T(1) - fr[2]));
#pragma unroll
            for (int q = 0; q < 3; ++q) rc[(5 + 4 * r + q) * FS] = tdx * mC[q];
        }
    }
};
template <class L, class T>
using P2gSmem = GroupSmem<L, T, void, AffineScatter<T, true>::NF, AffineScatter<T, true>::NC>;
constexpr int P2G_PIECE = 96; // fixed cost of a piece in particles

template <class L, class T>
__global__ void __launch_bounds__(FUSED_THREADS, P2gSmem<L, T>::CTAS) k_p2g_fused(GroupArgs ga, const double* __restrict__ pd, int64_t cap,
    const short4* __restrict__ base, double dx, double* __restrict__ gm, double* __restrict__ gmv, T* __restrict__ frac, int32_t* __restrict__ flags)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    P2gSmem<L, T>& sm = *reinterpret_cast<P2gSmem<L, T>*>(smem_raw);
    group_smem_init(sm);
    Share share(ga);
    int ph = 0;
    group_share<L, T, void, AffineScatter<T, true>, 1>(sm, ga, share, nullptr, gm, gmv, flags, ph,
        P2gPhase1<L, T>{ pd, cap, base, 1.0 / dx, T(dx), frac });
}

// -------------------------------------------------------------- damage -----
// Largest eigenvalue of a symmetric 3x3 matrix by the trigonometric solution
// of the characteristic cubic (O. K. Smith, "Eigenvalues of a symmetric 3x3
// matrix", CACM 4(4), 1961).
__device__ __forceinline__ double sym3_max_eig(const M3<double>& A)
{
    const double p1 = A(0, 1) * A(0, 1) + A(0, 2) * A(0, 2) + A(1, 2) * A(1, 2);
    const double q = (A(0, 0) + A(1, 1) + A(2, 2)) / 3.0;
    const double a = A(0, 0) - q, b = A(1, 1) - q, c = A(2, 2) - q;
    const double p2 = a * a + b * b + c * c + 2.0 * p1;
    if (p2 == 0.0) return q;
    const double p = sqrt(p2 / 6.0);
    M3<double> B = A;
    B(0, 0) = a;
    B(1, 1) = b;
    B(2, 2) = c;
#pragma unroll
    for (int i = 0; i < 9; ++i) B.a[i] /= p;
    double r = m3_det(B) / 2.0;
    r = r < -1.0 ? -1.0 : (r > 1.0 ? 1.0 : r);
    const double phi = acos(r) / 3.0;
    return q + 2.0 * p * cos(phi);
}

// FractureSimulation::solvePhaseFieldSystemNaive (FractureSimulation.h:509-554)
// for particles with Rankine damage and NeoHookeanBorden: Cauchy stress of the
// undegraded (g = 1) Kirchhoff stress, c <- min(c, sigma_F / sigma_max) when
// sigma_max > sigma_F, g = c^2 (1 - k) + k.  sigma_max: the largest eigenvalue
// (ZMPM_DAMAGE_RANKINE) or the reference's first eigenvalue of Eigen's general
// eigensolver (ZMPM_DAMAGE_RANKINE_REFERENCE, eig3.cuh); first_not_max counts
// the particles of the latter whose first eigenvalue is not the largest.
__global__ void k_rankine(double* __restrict__ pd, const int32_t* __restrict__ pi, int64_t cap, int64_t P,
    unsigned long long* __restrict__ first_not_max)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P) return;
    const int dkind = pi[PI_DAMAGE * cap + s];
    if ((dkind != ZMPM_DAMAGE_RANKINE && dkind != ZMPM_DAMAGE_RANKINE_REFERENCE) || pi[PI_KIND * cap + s] != ZMPM_MODEL_NEOHOOKEAN_BORDEN) return;
    M3<double> F;
#pragma unroll
    for (int q = 0; q < 9; ++q) F.a[q] = pd[(PD_F + q) * cap + s];
    const double J = m3_det(F);
    const double mu = pd[PD_MU * cap + s], kappa = pd[PD_KAPPA * cap + s];
    // NeoHookeanBorden::kirchhoff with g = 1 (NeoHookeanBorden.cpp:67-83)
    M3<double> B = m3_mulT(F, F);
    const double tr = B(0, 0) + B(1, 1) + B(2, 2);
    const double sdev = mu * pow(J, -2.0 / 3.0);
    const double vol = J * (kappa / 2 * (J - 1 / J));
    M3<double> cauchy;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double dv = (i == j) ? B(i, j) - 1.0 / 3.0 * tr : B(i, j);
            cauchy(i, j) = ((i == j) ? sdev * dv + vol : sdev * dv) / J;
        }
    double sigma_max = sym3_max_eig(cauchy);
    if (dkind == ZMPM_DAMAGE_RANKINE_REFERENCE) {
        Eig3 eig;
        const double first = eig.first_eigenvalue(cauchy.a);
        if (!(fabs(first - sigma_max) <= 1e-9 * fabs(sigma_max))) atomicAdd(first_not_max, 1ull);
        sigma_max = first;
    }
    const double sigma_f = pd[PD_SIGMA_F * cap + s];
    double c = pd[PD_PF_C * cap + s];
    const double k = pd[PD_PF_K * cap + s];
    if (sigma_max > sigma_f) c = fmin(c, sigma_f / sigma_max);
    pd[PD_PF_C * cap + s] = c;
    pd[PD_G * cap + s] = c * c * (1 - k) + k;
}

int launch_damage(Ctx* ctx)
{
    if (!ctx->has_damage || ctx->P == 0) return ZMPM_OK;
    DevCounters* dc = ctx->counters.as<DevCounters>();
    k_rankine<<<(unsigned)((ctx->P + 255) / 256), 256, 0, ctx->stream>>>(ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap, ctx->P,
        reinterpret_cast<unsigned long long*>(&dc->first_not_max));
    ++g_kernel_launches;
    return ZMPM_OK;
}

// --------------------------------------------------------------- update ----
// gate (MIXED contexts, which launch the FP32 and the FP64 form of
// k_update_fused per Newton iteration): 0 always runs, 1 runs while the solve's
// residual is FP32, 2 once it is FP64.
__device__ __forceinline__ bool gated_off(const SolverScalars* sc, int gate)
{
    return sc && (sc->newton_done || (gate != 0 && (gate == 1) == (sc->fp64_res != 0)));
}

// Force scatters: facc -= sum_p S_p grad w_ip (rasterizeForceToTVStack,
// MpmForceBase.cpp:102-152), or with MLS the MLS-MPM weight of
// particlesToGridWithForceHelper (MpmSimulationBase.cpp:527-541), facc -= (S_p
// (x_i - x_p)) w_ip D^-1 with D^-1 = 4 / dx^2.  A particle's record from its S.
template <class T, bool MLS, int FS>
__device__ __forceinline__ void force_record(const M3<T>& S, const T fr[3], T inv_dx, T* rc)
{
#pragma unroll
    for (int d = 0; d < 3; ++d) rc[d * FS] = fr[d];
    if constexpr (MLS) {
        const T k = T(-4) * inv_dx; // dx D^-1
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            rc[(3 + 4 * r) * FS] = k * (S(r, 0) * (T(1) - fr[0]) + S(r, 1) * (T(1) - fr[1]) + S(r, 2) * (T(1) - fr[2]));
#pragma unroll
            for (int c = 0; c < 3; ++c) rc[(4 + 4 * r + c) * FS] = k * S(r, c);
        }
    }
    else {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) rc[(3 + 3 * r + c) * FS] = -S(r, c) * inv_dx;
    }
}

// The scatter of a stress buffer (ADMM's right-hand side), one CTA per group:
// thread -> one cell of the page and every (blockDim/NPB)-th particle of it; the
// cell's particles share one 27-node stencil, so their terms are summed in
// registers and added to the shared window once per thread (FP32 keeps all 81
// sums in registers, FP64 one force component per pass).  With nothing to gather
// or compute per particle this beats records in shared memory (498k particles
// FP32: 51 against 60 us; 31k FP64: 29 us, and 0.3 ms more per 20 with records).
template <class L, class TS>
__global__ void __launch_bounds__(XF_THREADS) k_force(const int32_t* __restrict__ group_start, const int32_t* __restrict__ group_nbr,
    int64_t cap, const short4* __restrict__ base, double dx, const TS* __restrict__ frac, const TS* __restrict__ stress,
    double* __restrict__ facc)
{
    constexpr int NPB = L::NPB;
    __shared__ __align__(16) TS acc[8 * 3 * NPB];
    __shared__ int32_t nbr[8];
    __shared__ CellLayout<L> cl;
    const int g = blockIdx.x;
    if (threadIdx.x < 8) nbr[threadIdx.x] = group_nbr[8 * g + threadIdx.x];
    zero_window<3, NPB>(acc);
    const TS inv_dx = TS(1.0 / dx);
    const int s0 = group_start[g], s1 = group_start[g + 1];
    build_cell_layout<L>(cl, base, s0, s1);
    const int ce = threadIdx.x % NPB;
    const int lx = ce >> (L::YB + L::ZB), ly = (ce >> L::ZB) & (L::BY - 1), lz = ce & (L::BZ - 1);
    const int cnt = cl.cnt[ce], first = s0 + cl.start[ce];
    constexpr int NCP = sizeof(TS) == 4 ? 3 : 1;
#pragma unroll 1
    for (int c0 = 0; c0 < 3; c0 += NCP) {
        TS a[27][NCP];
#pragma unroll
        for (int n = 0; n < 27; ++n)
#pragma unroll
            for (int c = 0; c < NCP; ++c) a[n][c] = TS(0);
        for (int r = threadIdx.x / NPB; r < cnt; r += blockDim.x / NPB) {
            const int s = first + r;
            TS w[3][3], dwr[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) bspline(frac[d * cap + s], w[d], dwr[d]);
            TS row[NCP][3];
#pragma unroll
            for (int c = 0; c < NCP; ++c)
#pragma unroll
                for (int q2 = 0; q2 < 3; ++q2) row[c][q2] = stress[(3 * (c0 + c) + q2) * cap + s];
            for_stencil<L>(lx, ly, lz, w, dwr, inv_dx, [&](int, int, int i, int j, int k, TS, const TS* dw) {
                const int n = 9 * i + 3 * j + k;
#pragma unroll
                for (int c = 0; c < NCP; ++c) a[n][c] -= row[c][0] * dw[0] + row[c][1] * dw[1] + row[c][2] * dw[2];
            });
        }
        if (threadIdx.x / NPB < cnt) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        int e;
                        const int t = win_slot<L>(lx + i, ly + j, lz + k, e);
#pragma unroll
                        for (int c = 0; c < NCP; ++c) atomicAdd(acc + t * 3 * NPB + (c0 + c) * NPB + e, a[9 * i + 3 * j + k][c]);
                    }
        }
    }
    __syncthreads();
    flush_window<3, 3, NPB>(acc, nbr, facc, nullptr);
}

// Explicit substep: FBasedMpmForceHelper::updateState (FBasedMpmForceHelper.cpp:
// 44-64), S = V0 tau(F) = V0 P(F) F^T, plus V0 tau(Fe) for viscoelastic particles
// (FElasticNonequilibratedBasedMpmForceHelper.h:39-60), in the pass that scatters
// it (a stress kernel before it wrote 154 B per particle, the unused Hessian
// scratch among them).  FP32 with the FP64 re-evaluation of near-degenerate SVDs.
template <class T, bool MLS>
struct ExplicitPhase1 {
    const double* pd;
    const int32_t* pi;
    int64_t cap;
    const T* frac;
    T inv_dx;

    template <int FS>
    __device__ __forceinline__ void run(const void*, int64_t s, T* rc) const
    {
        T fr[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) fr[d] = frac[d * cap + s];
        const int kind = pi[PI_KIND * cap + s];
        M3<T> S = m3_zero<T>();
        if (kind != ZMPM_MODEL_NONE) {
            T scr[NS]; // the Hessian scratch, not kept
            M3<T> F;
#pragma unroll
            for (int q = 0; q < 9; ++q) F.a[q] = (T)pd[(PD_F + q) * cap + s];
            const ModelParams mp{ pd[PD_MU * cap + s], pd[PD_LAM * cap + s], pd[PD_KAPPA * cap + s], pd[PD_G * cap + s] };
            const double V0 = pd[PD_VOL * cap + s];
            bool degenerate = false;
            S = model_update<T, T>(kind, mp, (T)V0, F, F, scr, 1, 0, sizeof(T) == 4 ? &degenerate : nullptr);
            if constexpr (sizeof(T) == 4) {
                if (degenerate) {
                    M3<double> Fd;
#pragma unroll
                    for (int q = 0; q < 9; ++q) Fd.a[q] = pd[(PD_F + q) * cap + s];
                    S = m3_cast<T>(model_update<double, T>(kind, mp, V0, Fd, Fd, scr, 1, 0, nullptr));
                }
            }
            if (pi[PI_VISCO * cap + s]) {
                M3<double> Fe;
#pragma unroll
                for (int q = 0; q < 9; ++q) Fe.a[q] = pd[(PD_FE + q) * cap + s];
                const ModelParams mv{ pd[PD_VMU * cap + s], pd[PD_VLAM * cap + s], 0.0, 1.0 };
                const M3<double> Se = model_update<double, T>(ZMPM_MODEL_STVK_HENCKY_ISOTROPIC, mv, V0, Fe, Fe, scr, 1, 0, nullptr);
#pragma unroll
                for (int q = 0; q < 9; ++q) S.a[q] += (T)Se.a[q];
            }
        }
        force_record<T, MLS, FS>(S, fr, inv_dx, rc);
    }
};

template <class L, class T, bool MLS>
using ForceSmem = GroupSmem<L, T, void, MLS ? 15 : 12, 3>;
constexpr int FORCE_PIECE = 96; // fixed cost of a piece in particles

template <class L, class T, bool MLS, class Phase1>
__global__ void __launch_bounds__(FUSED_THREADS, ForceSmem<L, T, MLS>::CTAS) k_force_fused(GroupArgs ga, Phase1 p1, double* __restrict__ facc,
    int32_t* __restrict__ flags)
{
    using Scatter = typename std::conditional<MLS, AffineScatter<T, false>, RowsScatter<T>>::type;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    ForceSmem<L, T, MLS>& sm = *reinterpret_cast<ForceSmem<L, T, MLS>*>(smem_raw);
    group_smem_init(sm);
    Share share(ga);
    int ph = 0;
    group_share<L, T, void, Scatter, 3>(sm, ga, share, nullptr, facc, nullptr, flags, ph, p1);
}

// ------------------------------------------------------- fused products ----
// A product (hvp.cuh) as a kernel of its own: the zmpm_multiply hook's Hessian
// product, and ADMM's global operator out += sum_p (grad(x)_p B_p) grad w_ip
// (the matrix-free product of dvStep's MINRES, AdmmSimulationFoam.h:167-170).
template <class L, class T, class TX, class Model>
__global__ void __launch_bounds__(FUSED_THREADS, HvpSmem<L, T, TX>::CTAS) k_product(HvpArgs ha, Model model, const TX* __restrict__ x,
    double* __restrict__ out, int32_t* __restrict__ flags)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    HvpSmem<L, T, TX>& sm = *reinterpret_cast<HvpSmem<L, T, TX>*>(smem_raw);
    group_smem_init(sm);
    Share share(ha.ga);
    int ph = 0;
    hvp_share<L, T, TX>(sm, ha, share, model, x, out, flags, ph);
}

// MpmForceBase::updatePositionBasedState + rasterizeForceToTVStack
// (MpmForceBase.cpp:306-344, 102-152) in one kernel: phase 1 gathers grad(v)
// of vstar = vn + dv at each particle, F = (I + dt grad v) Fn (evolveStrain on
// the restored Fn, FBasedMpmForceHelper.cpp:95-109), S = V0 P(F) Fn^T and the
// Hessian scratch (updateImplicitState, :68-92); FP32 evaluations of
// near-degenerate SVDs are redone in FP64.  Phase 2 adds -S_p grad w_ip to
// facc.  TH: the type of the stored fractions and the scratch; T = double with TH
// = float is the FP64 residual of a MIXED solve (weights from the positions).
template <class L, class T, class TX, class TH>
struct UpdatePhase1 {
    const double* pd;
    const int32_t* pi;
    int64_t cap;
    const short4* base;
    const TH* frac;
    TH* scr;
    unsigned long long* svd64;
    double inv_dx, dt;

    template <int FS>
    __device__ __forceinline__ void run(const TX* win, int64_t s, T* rc) const
    {
        const short4 b = base[s];
        T fr[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if constexpr (sizeof(T) == sizeof(TH))
                fr[d] = frac[d * cap + s];
            else
                fr[d] = inv_dx * pd[(PD_X + d) * cap + s] - (double)((&b.x)[d]);
        }
        const int kind = pi[PI_KIND * cap + s];
#pragma unroll
        for (int d = 0; d < 3; ++d) rc[d * FS] = fr[d];
        const T tinv = T(inv_dx), tdt = T(dt);
        M3<T> S = m3_zero<T>();
        if (kind != ZMPM_MODEL_NONE) {
            T w[3][3], dw[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) bspline_all(fr[d], w[d], dw[d]);
            const StencilOffsets<L> so(b.x & (L::BX - 1), b.y & (L::BY - 1), b.z & (L::BZ - 1));
            M3<T> gv;
            if constexpr (sizeof(T) == 4 && sizeof(TX) == 4)
                gather_gradient_f32<L>(win, so, w, dw, gv.a);
            else
                gather_gradient<L, T, TX>(win, so, w, dw, gv.a);
            M3<T> Fn, A = m3_identity<T>();
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                Fn.a[q] = (T)pd[(PD_F + q) * cap + s];
                A.a[q] += tdt * (gv.a[q] * tinv);
            }
            const ModelParams mp{ pd[PD_MU * cap + s], pd[PD_LAM * cap + s], pd[PD_KAPPA * cap + s], pd[PD_G * cap + s] };
            const double V0 = pd[PD_VOL * cap + s];
            bool degenerate = false;
            S = model_update<T, TH>(kind, mp, (T)V0, m3_mul(A, Fn), Fn, scr, cap, s, sizeof(T) == 4 ? &degenerate : nullptr);
            if constexpr (sizeof(T) == 4) {
                if (degenerate) { // FP64 re-evaluation of near-degenerate particles
                    atomicAdd(svd64, 1ull);
                    M3<double> Fnd, Ad = m3_identity<double>();
#pragma unroll
                    for (int q = 0; q < 9; ++q) {
                        Fnd.a[q] = pd[(PD_F + q) * cap + s];
                        Ad.a[q] += dt * ((double)gv.a[q] * inv_dx);
                    }
                    S = m3_cast<T>(model_update<double, T>(kind, mp, V0, m3_mul(Ad, Fnd), Fnd, scr, cap, s, nullptr));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) rc[(3 + 3 * r + c) * FS] = -S(r, c) * tinv;
    }
};
constexpr int UPDATE_PIECE = 64; // fixed cost of a piece in particles

template <class L, class T, class TX, class TH>
__global__ void __launch_bounds__(FUSED_THREADS, HvpSmem<L, T, TX>::CTAS) k_update_fused(GroupArgs ga, const double* __restrict__ pd,
    const int32_t* __restrict__ pi, int64_t cap, const short4* __restrict__ base, double dx, double dt, const TH* __restrict__ frac,
    const TX* __restrict__ vstar, TH* __restrict__ scr, double* __restrict__ facc, const SolverScalars* __restrict__ sc,
    int32_t* __restrict__ flags, int gate, unsigned long long* __restrict__ svd64)
{
    if (gated_off(sc, gate)) return;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    HvpSmem<L, T, TX>& sm = *reinterpret_cast<HvpSmem<L, T, TX>*>(smem_raw);
    group_smem_init(sm);
    Share share(ga);
    int ph = 0;
    group_share<L, T, TX, RowsScatter<T>, 3>(sm, ga, share, vstar, facc, nullptr, flags, ph,
        UpdatePhase1<L, T, TX, TH>{ pd, pi, cap, base, frac, scr, svd64, 1.0 / dx, dt });
}

// ------------------------------------------------------------------ G2P ----
// MpmSimulationBase::applyPlasticity (MpmSimulationBase.cpp:1018-1030) on one
// particle (slot s): the return map of its plasticity kind applied to F, with
// the kind's state (log Jp; yield stress, broken flag and crack normal) updated
// in the pools.
__device__ __forceinline__ void apply_return_map(double* __restrict__ pd, int32_t* __restrict__ pi, int64_t cap, int64_t s, M3<double>& F)
{
    const int pkind = pi[PI_PKIND * cap + s];
    if (pkind == ZMPM_PLASTIC_DRUCKER_PRAGER || pkind == ZMPM_PLASTIC_CAM_CLAY) {
        double logJp = pd[PD_LOGJP * cap + s];
        if (pkind == ZMPM_PLASTIC_DRUCKER_PRAGER)
            drucker_prager_project<double>(pd[PD_MU * cap + s], pd[PD_LAM * cap + s], pd[PD_YS * cap + s], pd[PD_XI * cap + s],
                pd[PD_FS * cap + s], pi[PI_BROKEN * cap + s], logJp, F);
        else
            cam_clay_project<double>(pd[PD_MU * cap + s], pd[PD_KAPPA * cap + s], pd[PD_YS * cap + s], pd[PD_XI * cap + s],
                pd[PD_FS * cap + s], logJp, F);
        pd[PD_LOGJP * cap + s] = logJp;
    }
    if (pkind == ZMPM_PLASTIC_VON_MISES) {
        double ys = pd[PD_YS * cap + s];
        int broken = pi[PI_BROKEN * cap + s];
        double crack[3] = { pd[(PD_CRACK + 0) * cap + s], pd[(PD_CRACK + 1) * cap + s], pd[(PD_CRACK + 2) * cap + s] };
        von_mises_project<double>(pd[PD_MU * cap + s], pd[PD_LAM * cap + s], ys, pd[PD_XI * cap + s], pd[PD_FS * cap + s], broken, crack, F);
        pd[PD_YS * cap + s] = ys;
        pi[PI_BROKEN * cap + s] = broken;
#pragma unroll
        for (int d = 0; d < 3; ++d) pd[(PD_CRACK + d) * cap + s] = crack[d];
    }
}

// applyPlasticity as its own pass (slot order), for callers that run
// gridToParticles without it.
__global__ void k_plasticity(double* __restrict__ pd, int32_t* __restrict__ pi, int64_t cap, int64_t P)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P || pi[PI_KIND * cap + s] == ZMPM_MODEL_NONE || pi[PI_PKIND * cap + s] == ZMPM_PLASTIC_NONE) return;
    M3<double> F;
#pragma unroll
    for (int q = 0; q < 9; ++q) F.a[q] = pd[(PD_F + q) * cap + s];
    apply_return_map(pd, pi, cap, s, F);
#pragma unroll
    for (int q = 0; q < 9; ++q) pd[(PD_F + q) * cap + s] = F.a[q];
}

int launch_plasticity(Ctx* ctx)
{
    if (ctx->P == 0) return ZMPM_OK;
    k_plasticity<<<(unsigned)((ctx->P + 127) / 128), 128, 0, ctx->stream>>>(ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap, ctx->P);
    ++g_kernel_launches;
    return ZMPM_OK;
}

// MIXED: applyPlasticity on an FP32 F.  Von Mises runs in FP32 on its FP32
// SVD unless the singular values are near inversion (|sigma2| <= 0.2) or
// strongly stretched (sigma0 >= 5), where it runs in FP64; the other return
// maps run in FP64.
__device__ __forceinline__ void apply_return_map_f32(double* __restrict__ pd, int32_t* __restrict__ pi, int64_t cap, int64_t s, M3<float>& F)
{
    const int pkind = pi[PI_PKIND * cap + s];
    if (pkind == ZMPM_PLASTIC_NONE) return;
    if (pkind == ZMPM_PLASTIC_VON_MISES) {
        M3<float> U, V;
        float sg[3];
        svd3(F, U, sg, V);
        if (fabsf(sg[2]) > 0.2f && sg[0] < 5.f) {
            float ys = (float)pd[PD_YS * cap + s];
            int broken = pi[PI_BROKEN * cap + s];
            float crack[3] = { (float)pd[(PD_CRACK + 0) * cap + s], (float)pd[(PD_CRACK + 1) * cap + s], (float)pd[(PD_CRACK + 2) * cap + s] };
            const float ys0 = ys;
            const int broken0 = broken;
            von_mises_from_svd<float>((float)pd[PD_MU * cap + s], (float)pd[PD_LAM * cap + s], ys, (float)pd[PD_XI * cap + s],
                (float)pd[PD_FS * cap + s], broken, crack, F, U, sg, V);
            if (ys != ys0) pd[PD_YS * cap + s] = ys;
            if (broken != broken0) {
                pi[PI_BROKEN * cap + s] = broken;
#pragma unroll
                for (int d = 0; d < 3; ++d) pd[(PD_CRACK + d) * cap + s] = crack[d];
            }
            return;
        }
    }
    M3<double> Fd = m3_cast<double>(F);
    apply_return_map(pd, pi, cap, s, Fd);
    F = m3_cast<float>(Fd);
}

// gridToParticlesHelper<APIC> (MpmSimulationBase.cpp:906-1016): v_p = sum w v_i,
// B = sum w v_i (x_i - x_p)^T, C = ((1 + r) B D^-1 + (r - 1) (B D^-1)^T) / 2 with
// D^-1 = 4 / dx^2, grad v_p = sum v_i grad w^T, x_p += dt v_p and the CFL flag;
// then evolveStrain F = (I + dt grad v) Fn (FBasedMpmForceHelper.cpp:95-109, and
// the viscoelastic Fe's relaxation) and, with `plastic`, applyPlasticity.
// T: the arithmetic (FP32 in MIXED contexts: weights from the stored cell
// fractions, positions advanced in FP64).  FP64: three CTAs per SM (at most
// 168 registers; the form is latency bound on FP64 chains).  FP32: four (128
// registers, a few spilled words).
template <class L, class T, class TX>
__global__ void __launch_bounds__(XF_THREADS, sizeof(T) == 4 ? 4 : 3) k_g2p(const int32_t* __restrict__ group_start, const int32_t* __restrict__ group_nbr,
    double* __restrict__ pd, int32_t* __restrict__ pi, int64_t cap, const short4* __restrict__ base, const T* __restrict__ frac, double dx,
    double dt, double apic_rpic_ratio, const TX* __restrict__ vnew, int32_t* __restrict__ flags, int mls, int plastic)
{
    constexpr int NPB = L::NPB;
    __shared__ __align__(128) TX win[VecWindow<NPB, TX>::ELEMS];
    __shared__ int32_t nbr[8];
    __shared__ __align__(8) uint64_t bar;
    const int g = blockIdx.x;
    if (threadIdx.x < 8) nbr[threadIdx.x] = group_nbr[8 * g + threadIdx.x];
    __syncthreads();
    stage_vec_window<NPB, TX>(win, vnew, nbr, &bar, flags);
    const T inv_dx = T(1.0 / dx), tdx = T(dx);
    const T D_inverse = T(4.0 / (dx * dx));
    const T ca = T((apic_rpic_ratio + 1) * 0.5), cb = T((apic_rpic_ratio - 1) * 0.5);
    const T tdt = T(dt);
    int too_fast = 0;
    const int s0 = group_start[g], s1 = group_start[g + 1];
    for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x) {
        const short4 b = base[s];
        T fr[3], w[3][3], dwr[3][3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            fr[d] = frac[d * cap + s];
            bspline(fr[d], w[d], dwr[d]);
        }
        const int lx = b.x & (L::BX - 1), ly = b.y & (L::BY - 1), lz = b.z & (L::BZ - 1);
        const StencilOffsets<L> so(lx, ly, lz);
        T pv[3] = { 0, 0, 0 };
        M3<T> Bp = m3_zero<T>(), gv = m3_zero<T>();
        double xp[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) xp[d] = pd[(PD_X + d) * cap + s];
        for_stencil<L>(lx, ly, lz, w, dwr, inv_dx, [&](int, int, int i, int j, int k, T wijk, const T* dw) {
            TX vv[3];
            VecWindow<NPB, TX>::node(win, so.X[i] + so.Y[j] + so.Z[k], vv);
            // x_i - x_p: FP64 from the node and particle positions, FP32 from the cell fractions
            T xi[3];
            if constexpr (sizeof(T) == 8) {
                xi[0] = (b.x + i) * dx - xp[0];
                xi[1] = (b.y + j) * dx - xp[1];
                xi[2] = (b.z + k) * dx - xp[2];
            }
            else {
                xi[0] = (T(i) - fr[0]) * tdx;
                xi[1] = (T(j) - fr[1]) * tdx;
                xi[2] = (T(k) - fr[2]) * tdx;
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const T vr = (T)vv[r];
                pv[r] += wijk * vr;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    Bp(r, c) += wijk * vr * xi[c];
                    gv(r, c) += vr * dw[c];
                }
            }
        });
        double inc2 = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            pd[(PD_V + d) * cap + s] = pv[d];
            const double inc = dt * (double)pv[d];
            pd[(PD_X + d) * cap + s] = xp[d] + inc;
            inc2 += inc * inc;
        }
        too_fast |= (inc2 > dx * dx);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T cn = ca * (Bp(r, c) * D_inverse) + cb * (Bp(c, r) * D_inverse);
                pd[(PD_C + 3 * r + c) * cap + s] = cn;
                if (mls) gv(r, c) = cn; // MLS: gradVp = C_p (MpmSimulationBase.cpp:958-961)
            }
        const int kind = pi[PI_KIND * cap + s];
        if (kind == ZMPM_MODEL_NONE) continue;
        // evolveStrain (FBasedMpmForceHelper.cpp:95-109) on the restored F = Fn
        M3<T> F0, A = m3_identity<T>();
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            F0.a[q] = (T)pd[(PD_F + q) * cap + s];
            A.a[q] += tdt * gv.a[q];
        }
        M3<T> F = m3_mul(A, F0);
        if (plastic) {
            if constexpr (sizeof(T) == 8)
                apply_return_map(pd, pi, cap, s, F);
            else
                apply_return_map_f32(pd, pi, cap, s, F);
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) pd[(PD_F + q) * cap + s] = F.a[q];
        if (pi[PI_VISCO * cap + s]) {
            // FElasticNonequilibratedBasedMpmForceHelper::evolveStrain (h:62-87), FP64
            M3<double> Fe;
#pragma unroll
            for (int q = 0; q < 9; ++q) Fe.a[q] = pd[(PD_FE + q) * cap + s];
            Fe = m3_mul(m3_cast<double>(A), Fe);
            viscous_return<double>(pd[PD_VMU * cap + s], pd[PD_VLAM * cap + s], pd[PD_VD * cap + s], pd[PD_VV * cap + s], dt, Fe);
#pragma unroll
            for (int q = 0; q < 9; ++q) pd[(PD_FE + q) * cap + s] = Fe.a[q];
        }
    }
    if (__syncthreads_or(too_fast) && threadIdx.x == 0) atomicOr(flags, (int32_t)FLAG_CFL);
}

// ------------------------------------------------------------- launchers --
template <class L, class T>
static int p2g_impl(Ctx* ctx)
{
    if (ctx->G == 0) return ZMPM_OK;
    return launch_resident(ctx, ctx->stream, false, useful_ctas(ctx, P2G_PIECE), sizeof(P2gSmem<L, T>), k_p2g_fused<L, T>,
        group_args(ctx, P2G_PIECE), ctx->pd.as<double>(), ctx->Pcap, ctx->base.as<short4>(), ctx->cfg.dx, ctx->gm.as<double>(),
        ctx->gmv.as<double>(), ctx->frac.as<T>(), &ctx->counters.as<DevCounters>()->flags);
}
int launch_p2g(Ctx* ctx)
{
    if (ctx->mixed) return ctx->layout == 1 ? p2g_impl<Layout244, float>(ctx) : p2g_impl<Layout444, float>(ctx);
    return ctx->layout == 1 ? p2g_impl<Layout244, double>(ctx) : p2g_impl<Layout444, double>(ctx);
}

template <class L>
static int update_impl(Ctx* ctx, bool gated)
{
    const int64_t G = ctx->G;
    if (G == 0) return ZMPM_OK;
    DevCounters* dc = ctx->counters.as<DevCounters>();
    const SolverScalars* sc = gated ? ctx->scal.as<SolverScalars>() : nullptr;
    if (ctx->mixed) {
        // FP32 stress and force; inside a solve also the FP64 form, which runs
        // instead once the FP32 residual stalled (FP32 Hessian scratch either
        // way).  The FP32 pass gathers from the FP32 copy of vstar, which the
        // Newton solve keeps current; the hooks and the adjoint set vstar directly.
        const int gate = sc ? 1 : 0;
        if (!sc || !ctx->vstarf_valid) {
            int rc = refresh_vstar_f32(ctx);
            if (rc) return rc;
            ctx->vstarf_valid = true;
        }
        int rc = launch_resident(ctx, ctx->stream, false, useful_ctas(ctx, UPDATE_PIECE), sizeof(HvpSmem<L, float, float>),
            k_update_fused<L, float, float, float>, group_args(ctx, UPDATE_PIECE), ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap, ctx->base.as<short4>(),
            ctx->cfg.dx, ctx->dt, ctx->frac.as<float>(), ctx->vstarf.as<float>(), ctx->scratch.as<float>(), ctx->facc.as<double>(), sc, &dc->flags,
            gate, reinterpret_cast<unsigned long long*>(&dc->svd_fp64));
        if (rc) return rc;
        if (sc)
            return launch_resident(ctx, ctx->stream, false, useful_ctas(ctx, UPDATE_PIECE), sizeof(HvpSmem<L, double, double>),
                k_update_fused<L, double, double, float>, group_args(ctx, UPDATE_PIECE), ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap,
                ctx->base.as<short4>(), ctx->cfg.dx, ctx->dt, ctx->frac.as<float>(), ctx->vstar.as<double>(), ctx->scratch.as<float>(),
                ctx->facc.as<double>(), sc, &dc->flags, 2, reinterpret_cast<unsigned long long*>(&dc->svd_fp64));
    }
    else {
        return launch_resident(ctx, ctx->stream, false, useful_ctas(ctx, UPDATE_PIECE), sizeof(HvpSmem<L, double, double>),
            k_update_fused<L, double, double, double>, group_args(ctx, UPDATE_PIECE), ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap, ctx->base.as<short4>(),
            ctx->cfg.dx, ctx->dt, ctx->frac.as<double>(), ctx->vstar.as<double>(), ctx->scratch.as<double>(), ctx->facc.as<double>(), sc,
            &dc->flags, 0, reinterpret_cast<unsigned long long*>(&dc->svd_fp64));
    }
    return ZMPM_OK;
}
int launch_update(Ctx* ctx, bool gated) { return ctx->layout == 1 ? update_impl<Layout244>(ctx, gated) : update_impl<Layout444>(ctx, gated); }

// out += dt^-2 (Hessian part of A) x: the fused product, T the context's HVP
// precision, on an FP64 input vector
template <class L, class T, class Model>
static int product_impl(Ctx* ctx, const Model& model, const double* x, double* out)
{
    return launch_resident(ctx, ctx->stream, false, useful_ctas(ctx, hvp_piece<T>()), sizeof(HvpSmem<L, T, double>), k_product<L, T, double, Model>,
        hvp_args(ctx, hvp_piece<T>()), model, x, out, &ctx->counters.as<DevCounters>()->flags);
}
template <class L>
static int hvp_impl(Ctx* ctx, const double* x, double* out)
{
    if (ctx->G == 0) return ZMPM_OK;
    const int32_t* pi = ctx->pi.as<int32_t>();
    if (ctx->mixed) return product_impl<L, float>(ctx, HvpModel<float>{ pi, ctx->scratch.as<float>(), ctx->Pcap }, x, out);
    return product_impl<L, double>(ctx, HvpModel<double>{ pi, ctx->scratch.as<double>(), ctx->Pcap }, x, out);
}

int launch_hvp(Ctx* ctx, const double* x, double* out, bool fp32)
{
    if (fp32 != ctx->mixed) return ZMPM_UNSUPPORTED;
    return ctx->layout == 1 ? hvp_impl<Layout244>(ctx, x, out) : hvp_impl<Layout444>(ctx, x, out);
}

template <class L, class T, bool MLS, class Phase1>
static int force_impl(Ctx* ctx, const Phase1& p1, double* out)
{
    return launch_resident(ctx, ctx->stream, false, useful_ctas(ctx, FORCE_PIECE), sizeof(ForceSmem<L, T, MLS>),
        k_force_fused<L, T, MLS, Phase1>, group_args(ctx, FORCE_PIECE), p1, out, &ctx->counters.as<DevCounters>()->flags);
}
// out -= sum_p stress_p grad w_ip with `stress` in the HVP precision.
template <class L, class T>
static int force_scatter_impl(Ctx* ctx, double* out)
{
    k_force<L, T><<<(unsigned)ctx->G, XF_THREADS, 0, ctx->stream>>>(ctx->group_start.as<int32_t>(), ctx->group_nbr.as<int32_t>(), ctx->Pcap,
        ctx->base.as<short4>(), ctx->cfg.dx, ctx->frac.as<T>(), ctx->stress.as<T>(), out);
    ++g_kernel_launches;
    return ZMPM_OK;
}
int launch_force_scatter(Ctx* ctx, double* out)
{
    if (!ctx->G) return ZMPM_OK;
    if (ctx->mixed) return ctx->layout == 1 ? force_scatter_impl<Layout244, float>(ctx, out) : force_scatter_impl<Layout444, float>(ctx, out);
    return ctx->layout == 1 ? force_scatter_impl<Layout244, double>(ctx, out) : force_scatter_impl<Layout444, double>(ctx, out);
}
// out -= the explicit substep's forces (after P2G, which forms the fractions).
template <class L, class T>
static int explicit_force_impl(Ctx* ctx, double* out, bool mls)
{
    const double* pd = ctx->pd.as<double>();
    const int32_t* pi = ctx->pi.as<int32_t>();
    const T inv_dx = T(1.0 / ctx->cfg.dx);
    if (mls) return force_impl<L, T, true>(ctx, ExplicitPhase1<T, true>{ pd, pi, ctx->Pcap, ctx->frac.as<T>(), inv_dx }, out);
    return force_impl<L, T, false>(ctx, ExplicitPhase1<T, false>{ pd, pi, ctx->Pcap, ctx->frac.as<T>(), inv_dx }, out);
}
int launch_explicit_force(Ctx* ctx, double* out, bool mls)
{
    if (!ctx->G) return ZMPM_OK;
    if (ctx->mixed)
        return ctx->layout == 1 ? explicit_force_impl<Layout244, float>(ctx, out, mls) : explicit_force_impl<Layout444, float>(ctx, out, mls);
    return ctx->layout == 1 ? explicit_force_impl<Layout244, double>(ctx, out, mls) : explicit_force_impl<Layout444, double>(ctx, out, mls);
}

// out += sum_p (grad(x)_p B_p) grad w_ip (ADMM's global operator).
template <class L>
static int admm_op_impl(Ctx* ctx, const double* x, double* out)
{
    if (ctx->mixed) return product_impl<L, float>(ctx, AdmmOpModel<float>{ ctx->adm_B.as<float>(), ctx->Pcap }, x, out);
    return product_impl<L, double>(ctx, AdmmOpModel<double>{ ctx->adm_B.as<double>(), ctx->Pcap }, x, out);
}
int launch_admm_op(Ctx* ctx, const double* x, double* out)
{
    if (!ctx->G) return ZMPM_OK;
    return ctx->layout == 1 ? admm_op_impl<Layout244>(ctx, x, out) : admm_op_impl<Layout444>(ctx, x, out);
}

template <class L>
static int g2p_impl(Ctx* ctx, bool plastic)
{
    const int64_t G = ctx->G;
    if (G == 0) return ZMPM_OK;
    DevCounters* dc = ctx->counters.as<DevCounters>();
    if (ctx->mixed)
        k_g2p<L, float, float><<<(unsigned)G, XF_THREADS, 0, ctx->stream>>>(ctx->group_start.as<int32_t>(), ctx->group_nbr.as<int32_t>(),
            ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap, ctx->base.as<short4>(), ctx->frac.as<float>(), ctx->cfg.dx, ctx->dt,
            ctx->cfg.apic_rpic_ratio, ctx->vstarf.as<float>(), &dc->flags, ctx->mls ? 1 : 0, plastic ? 1 : 0);
    else
        k_g2p<L, double, double><<<(unsigned)G, XF_THREADS, 0, ctx->stream>>>(ctx->group_start.as<int32_t>(), ctx->group_nbr.as<int32_t>(),
            ctx->pd.as<double>(), ctx->pi.as<int32_t>(), ctx->Pcap, ctx->base.as<short4>(), ctx->frac.as<double>(), ctx->cfg.dx, ctx->dt,
            ctx->cfg.apic_rpic_ratio, ctx->vstar.as<double>(), &dc->flags, ctx->mls ? 1 : 0, plastic ? 1 : 0);
    ++g_kernel_launches;
    return ZMPM_OK;
}
int launch_g2p(Ctx* ctx, bool plastic) { return ctx->layout == 1 ? g2p_impl<Layout244>(ctx, plastic) : g2p_impl<Layout444>(ctx, plastic); }

} // namespace zmpm
