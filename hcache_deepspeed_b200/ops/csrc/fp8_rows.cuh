// E4M3 codes of a row of 16-bit values with one scale: amax / 448 (1 for a row of zeros).
#pragma once
#include <cuda_fp8.h>
#include "hds_ptx.cuh"

namespace hds {

constexpr float kE4M3Max = 448.0f;

// eight 16-bit values times inv -> their codes
template <bool kBf16>
__device__ __forceinline__ uint2 e4m3_codes8(const uint4& p, float inv) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
    uint32_t o[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t lo = __nv_cvt_float_to_fp8(unpack_lo<kBf16>(w[j]) * inv, __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float_to_fp8(unpack_hi<kBf16>(w[j]) * inv, __NV_SATFINITE, __NV_E4M3);
        o[j >> 1] |= (lo | (hi << 8)) << ((j & 1) * 16);
    }
    return make_uint2(o[0], o[1]);
}

}  // namespace hds
