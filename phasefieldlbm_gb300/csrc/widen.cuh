// widen.cuh - float to double on the integer units.
//
// A conversion to 64 bits costs as much as an FP64 addition (2 lanes per
// clock and SM), and the FP64 sums over float fields need nearly one per
// addition. A normal float's double has the same mantissa bits and a rebased
// exponent, which a few 32-bit integer instructions assemble exactly.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pflbm {

// Whether widen_bits(v) is exact: v is normal or zero.
__device__ __forceinline__ bool widens(float v) {
    const uint32_t u = __float_as_uint(v) << 1;
    return u == 0u || (u >> 24) - 1u < 254u;
}
__device__ __forceinline__ double widen_bits(float v) {
    const uint32_t u = __float_as_uint(v);
    const uint32_t hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u);
    return __hiloint2double(int((u << 1) == 0u ? u : hi), int(u << 29));
}

// v[0..N) as doubles; denormals, infinities and NaN take the conversion
// instruction.
template <int N>
__device__ __forceinline__ void widen_all(const float (&v)[N], double (&d)[N]) {
    bool plain = true;
#pragma unroll
    for (int k = 0; k < N; ++k) plain = plain && widens(v[k]);
    if (plain) {
#pragma unroll
        for (int k = 0; k < N; ++k) d[k] = widen_bits(v[k]);
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) d[k] = double(v[k]);
    }
}

}  // namespace pflbm
