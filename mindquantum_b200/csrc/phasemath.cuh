// Phase factors of the diagonal gates, for the generated pass kernels (compiled by NVRTC with them).
//
// A diagonal pair (d0, d1) on a register bit is applied as d0 times (1, r), r = d1 / d0: only the amplitudes
// with the bit set are multiplied, and d0 joins factors that are applied once per stage or per pass.  The
// ratio and the product of the d0 are made in FP64 and scaled to modulus one before they are rounded, so that a
// complex64 state sees one rounding of the ratio instead of one of each entry.
#ifndef MQB_PHASEMATH_CUH_
#define MQB_PHASEMATH_CUH_

#include "regmath.cuh"

namespace mqb {
namespace reg {

// a scaled to modulus one (|a| is one to a few roundings of complex64: two Newton steps are exact in FP64)
__device__ __forceinline__ double2 unit(double2 a) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double t = 1.5 - 0.5 * fma(a.x, a.x, a.y * a.y);
        a.x *= t;
        a.y *= t;
    }
    return a;
}

template <typename V>
__device__ __forceinline__ double2 wide(V a) {
    return cval<double2>(a.x, a.y);
}

// The second entry of a unit-modulus diagonal pair becomes its ratio to the first.
template <typename V>
__device__ __forceinline__ void prepare_pair(V *M) {
    const double2 r = unit(cmul(wide(M[1]), cconj(wide(M[0]))));
    M[1] = cval<V>(r.x, r.y);
}

}  // namespace reg
}  // namespace mqb

#endif
