// Which kernel takes a linear in a decode step of eight sequences; kept free of CUDA so that it can be checked on a host
// (tests/cpp/test_linear_plan.cpp).
#pragma once

#include <cstdint>

namespace prism {

// Whether the GEMM takes less time than the batched GEMV for 8 activation rows and one tensor of m rows of k weights (swiglu: two of
// them).  The GEMM costs about 12 us before its first weight and wants rows to fill tiles of 256 with; the GEMV takes a block of
// 64 rows per SM and looks every weight up, whatever its bits.  Measured on 226 shapes of 2^24 to 2^27 weights, GEMV / GEMM in us:
//  * 4 bit, one tensor, from 2^25 weights on: 2048 x 18944 26.0 / 33.2, 3584 x 11008 24.8 / 20.7, 5120 x 8192 26.5 / 20.9,
//    18944 x 3584 28.3 / 21.1.  Where the blocks just fill the SMs the GEMV is at its best: 8192 x 4096 15.3 / 17.3, 8192 x 5120
//    18.3 / 19.3, 8192 x 8192 26.2 / 24.9;
//  * 4 bit, gate and up: 5120 x 3584 24.1 / 36.4, 8192 x 4096 33.9 / 40.4, 8192 x 8192 52.9 / 50.5,
//    10240 x 3584 38.5 / 37.0, 18944 x 3584 52.9 / 39.2;
//  * 2 bit, the same bytes looked up twice as often: 2048 x 8192 (two) 32.5 / 55.4, 3584 x 3584 (two) 26.9 / 31.6, 3584 x 5120 (two)
//    35.3 / 29.4, 3584 x 11008 36.1 / 18.3, 2048 x 18944 36.1 / 31.6.
// Of the shapes that it gives to the GEMM two lose more than 2 %, both at 4 bits: 10240 x 5120 (two) 46.9 / 48.1 and 10240 x 14336
// 55.2 / 60.4 (40 tiles, which neither fill the pairs of CTAs nor halve well).
inline bool gemm_pays_at_8(uint64_t m, uint64_t k, uint32_t bits, bool swiglu, uint32_t sm_count) {
    if (m * k * (swiglu ? 2 : 1) < 1u << 25) return false;
    const uint32_t least = bits == 4 ? (!swiglu ? 3072 : k < 8192 ? 10240 : 8192) : (k < 18432 ? 3072 : 2048);
    if (m < least) return false;
    const uint64_t blocks = (m + 63) / 64;
    return !(bits == 4 && !swiglu && 4 * blocks > 3 * (uint64_t)sm_count && blocks <= sm_count && k < 8192);
}

}  // namespace prism
