// damping.hpp -- coefficients of an absorbing layer's memory variables, for
// the tile kernels and, compiled for the host, for their test.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define JV_HD __host__ __device__ __forceinline__
#else
#define JV_HD inline
#endif

namespace jv {

// rounded one by one, never contracted into a fused multiply-add (a host
// build takes -ffp-contract=off)
JV_HD float mul_rn(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
JV_HD float add_rn(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}

// psi <- b psi + a D at a node with d = vp K: b = exp(-(d + alpha) dt), a = d
// (b - 1) / (d + alpha) (FD/fdtd3d_1_cpml_mpi_module/
// fdtd3d_cpml_mpi_1_host_meat.hpp:147-620).  K and alpha are the node's entry
// of an axis table, both zero where it does not absorb (a = 0, b = 1 then).
// The quotient is a division: formed from an estimate of 1 / (d + alpha) as
// (b - 1) - (b - 1) alpha / (d + alpha) it saved 2 % of a migration (200^3 + 20,
// 392 against 400 ms per 300 steps) but lost a to cancellation in a layer's
// inner cells, d << alpha: off by 3e-6 at 16 cells and 1e-4 at 20, against 1e-7.
JV_HD void damping_ab(float vp, float K, float alpha, float dt, float &a, float &b) {
    const float d = mul_rn(vp, K), e = add_rn(d, alpha);
    b = expf(-mul_rn(e, dt));
    a = mul_rn(d, add_rn(b, -1.f)) / (e == 0.f ? 1.f : e);
}

}  // namespace jv
