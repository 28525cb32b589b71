// The Hessian-vector product, shared by the plain kernels (k_product) and the persistent Krylov kernels.
//
// MpmForceBase::addScaledForceDifferential (MpmForceBase.cpp:259-302) in one
// pass (fused.cuh): phase 1 gathers grad(x) at each particle from the staged
// window of the input vector and evaluates dS = V0 dP(grad(x) Fn) Fn^T from the
// Hessian scratch (computeStressDifferential, FBasedMpmForceHelper.cpp:132-
// 154); phase 2 adds dS grad w_ip to the nodes (rasterizeForceToTVStack with
// the differential, :102-152): out += sum_p dS_p grad w_ip.  T: arithmetic
// precision; TX: the input vector (FP32 node-major copy or FP64 vector).
// The per-particle map grad(x) -> dS is a model object: HvpModel (the
// constitutive model's differential from the Hessian scratch) or AdmmOpModel
// (the ADMM global operator's grad(x) B, AdmmSimulationFoam.h dvStep).
#pragma once
#include "fused.cuh"
#include "models.cuh"

namespace zmpm {

// dS = V0 dP(G Fn) Fn^T from the Hessian scratch; particles without a model
// contribute nothing.
template <class T>
struct HvpModel {
    const int32_t* pi;
    const T* scr;
    int64_t cap;
    __device__ __forceinline__ int kind(int64_t s) const { return pi[PI_KIND * cap + s]; }
    __device__ __forceinline__ bool active(int k) const { return k != ZMPM_MODEL_NONE; }
    __device__ __forceinline__ M3<T> operator()(int k, int64_t s, const M3<T>& G) const { return model_hvp<T>(k, scr, cap, s, G); }
};

// ADMM's global operator: dS = G B with the particle's symmetric B (six
// entries, k_admm_init), every particle.
template <class T>
struct AdmmOpModel {
    const T* B;
    int64_t cap;
    __device__ __forceinline__ int kind(int64_t) const { return 0; }
    __device__ __forceinline__ bool active(int) const { return true; }
    __device__ __forceinline__ M3<T> operator()(int, int64_t s, const M3<T>& G) const
    {
        const T b00 = B[0 * cap + s], b01 = B[1 * cap + s], b02 = B[2 * cap + s], b11 = B[3 * cap + s], b12 = B[4 * cap + s],
                b22 = B[5 * cap + s];
        M3<T> d;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            d(r, 0) = G(r, 0) * b00 + G(r, 1) * b01 + G(r, 2) * b02;
            d(r, 1) = G(r, 0) * b01 + G(r, 1) * b11 + G(r, 2) * b12;
            d(r, 2) = G(r, 0) * b02 + G(r, 1) * b12 + G(r, 2) * b22;
        }
        return d;
    }
};

// Phase 1 of the product (fused.cuh): grad(x) at the particle from the staged
// window, dS from the model, and the record of its scatter.
template <class L, class T, class TX, class Model>
struct HvpPhase1 {
    const short4* base;
    const T* frac;
    int64_t cap;
    T inv_dx;
    Model model;

    template <int FS>
    __device__ __forceinline__ void run(const TX* win, int64_t s, T* rc) const
    {
        T fr[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) fr[d] = frac[d * cap + s];
        const short4 b = base[s];
        const int kind = model.kind(s);
#pragma unroll
        for (int d = 0; d < 3; ++d) rc[d * FS] = fr[d];
        M3<T> dS = m3_zero<T>();
        if (model.active(kind)) {
            T w[3][3], dw[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) bspline_all(fr[d], w[d], dw[d]);
            const StencilOffsets<L> so(b.x & (L::BX - 1), b.y & (L::BY - 1), b.z & (L::BZ - 1));
            M3<T> G;
            if constexpr (sizeof(T) == 4 && sizeof(TX) == 4)
                gather_gradient_f32<L>(win, so, w, dw, G.a);
            else
                gather_gradient<L, T, TX>(win, so, w, dw, G.a);
#pragma unroll
            for (int q = 0; q < 9; ++q) G.a[q] *= inv_dx;
            dS = model(kind, s, G);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) rc[(3 + 3 * r + c) * FS] = dS(r, c) * inv_dx;
    }
};

// A product's particle arrays.
struct HvpArgs {
    GroupArgs ga;
    const int32_t* pi;
    const short4* base;
    const void *frac, *scr; // in the product's precision
    int64_t cap;
    double dx;
};
inline GroupArgs group_args(const Ctx* ctx, int K)
{
    return GroupArgs{ ctx->group_start.as<int32_t>(), ctx->group_nbr.as<int32_t>(), ctx->group_cells.as<int32_t>(), (int)ctx->G, K };
}
inline HvpArgs hvp_args(const Ctx* ctx, int K)
{
    HvpArgs ha;
    ha.ga = group_args(ctx, K);
    ha.pi = ctx->pi.as<int32_t>();
    ha.base = ctx->base.as<short4>();
    ha.frac = ctx->frac.p;
    ha.scr = ctx->scratch.p;
    ha.cap = ctx->Pcap;
    ha.dx = ctx->cfg.dx;
    return ha;
}

// Fixed cost of a piece in particles (fused.cuh), for FP32 and FP64 products.
// Slowest CTA of a product, 1M / 197k particles FP32 and 250k FP64, for K = 96 /
// 64: 118, 29.5 and 62 us; 200 / 130: 116, 27 and 54.5 us; 500 / 400: 122, 27
// and 53 us.
template <class T>
constexpr int hvp_piece() { return sizeof(T) == 4 ? 200 : 160; }

template <class L, class T, class TX>
using HvpSmem = GroupSmem<L, T, TX, RowsScatter<T>::NF, RowsScatter<T>::NC>;

// out += sum_p dS_p grad w_ip over the CTA's share of the particles.
template <class L, class T, class TX, class Model>
__device__ __forceinline__ void hvp_share(HvpSmem<L, T, TX>& sm, const HvpArgs& ha, Share& share, const Model& model,
    const TX* x, double* out, int32_t* flags, int& ph)
{
    const HvpPhase1<L, T, TX, Model> p1{ ha.base, static_cast<const T*>(ha.frac), ha.cap, T(1.0 / ha.dx), model };
    group_share<L, T, TX, RowsScatter<T>, 3>(sm, ha.ga, share, x, out, nullptr, flags, ph, p1);
}

} // namespace zmpm
