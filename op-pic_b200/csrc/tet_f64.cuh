// The FP64 barycentric cell test of the FemPIC move, shared by the move kernels and the
// direct-hop grid build (which must decide "point inside cell" exactly as the move does).
//
// The arithmetic uses explicit round-to-nearest intrinsics so nothing is contracted into
// FMAs: each lambda_i is bit-identical to the reference expression
//   coef * (((d0 - d1*x) + d2*y) - d3*z)          (apps/app_fempic/kernels.h:110-117)
// and the inside test / argmin follow kernels.h:121-146 exactly.
#pragma once

#include "oppb_common.cuh"

namespace oppb {
namespace {

constexpr double kTol = 1e-10;  // KERNEL_TOLERENCE, apps/app_fempic/kernels.h:44

__device__ __forceinline__ void swap_if(bool p, double& a, double& b) {
    const double t = p ? b : a;
    b = p ? a : b;
    a = t;
}

// lambda_0..3 of point (x,y,z) in cell c, evaluated exactly as the FP64 reference.
//
// The j-th 256-bit load of a lane reads sector j ^ (lane & 3) of its 128-B det record, so the
// four lanes that a wide load serves together read four different sectors.  Lanes in different
// cells that read the same sector index of their records hit the same L1 banks and are served
// one after the other; with the sectors spread the fused FP64 move of the 57M-particle state
// takes 3.46 ms instead of 4.39.  Each sector holds one vertex's four coefficients, so only the
// four lambdas have to be put back in vertex order.  Of the nav record a visit reads only the 8
// bytes of the coefficient, a wavefront or two instead of the eight that a 256-bit load returns to
// a warp at least; a particle that hops on reads its one neighbour (neighbour()): 3.46 -> 3.21 ms.
__device__ __forceinline__ void visit_f64(const oppb_tet_mesh& m, int32_t c, double x, double y, double z,
                                          double l[4]) {
    const double* d = m.det + (int64_t)c * 16;
    const uint32_t first = threadIdx.x & 3u;
    double r[16];
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
        ldg256(d + ((j ^ first) << 2), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    const double coef = __ldg(m.nav + (int64_t)c * 4);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        double t = __dsub_rn(r[4 * i], __dmul_rn(r[4 * i + 1], x));
        t = __dadd_rn(t, __dmul_rn(r[4 * i + 2], y));
        t = __dsub_rn(t, __dmul_rn(r[4 * i + 3], z));
        l[i] = __dmul_rn(coef, t);
    }
    const bool odd = (first & 1u) != 0, upper = (first & 2u) != 0;
    swap_if(odd, l[0], l[1]);
    swap_if(odd, l[2], l[3]);
    swap_if(upper, l[0], l[2]);
    swap_if(upper, l[1], l[3]);
}

// Inside test of kernels.h:121-124 and first-index argmin of kernels.h:139-146.
__device__ __forceinline__ bool inside_f64(const double l[4]) {
    bool in = true;
#pragma unroll
    for (int i = 0; i < 4; i++) in = in && (l[i] > -kTol) && (__dsub_rn(l[i], 1.0) < kTol);
    return in;
}
__device__ __forceinline__ int argmin4(const double l[4]) {
    int mi = 0;
    double mv = l[0];
#pragma unroll
    for (int i = 1; i < 4; i++)
        if (l[i] < mv) {
            mv = l[i];
            mi = i;
        }
    return mi;
}

// The cell behind face i of cell c (the nav record's c2c), -1 at the boundary.
__device__ __forceinline__ int32_t neighbour(const oppb_tet_mesh& m, int32_t c, int i) {
    return __ldg(reinterpret_cast<const int32_t*>(m.nav + (int64_t)c * 4 + 1) + i);
}

}  // namespace
}  // namespace oppb
