// ADMM's assembled global operator (stencil.cu).
#pragma once
#include "internal.cuh"
#include "krylov.cuh"

namespace zmpm {

constexpr int STENCIL = 125; // entries of a row: offsets -2 .. 2 on each axis

bool stencil_pays(const Ctx* ctx);
bool stencil_reserve(Ctx* ctx);
int launch_stencil_build(Ctx* ctx); // neighbours, K, preconditioner
int launch_stencil_start(Ctx* ctx, const KrylovBufs& kb, double* part, SolverScalars* sc, int* parts);
int launch_stencil_minres(Ctx* ctx, const NodeGeom& ng, const KrylovBufs& kb, double* pA, double* pB, SolverScalars* sc, int kmax);

} // namespace zmpm
