// INT8 codes -> bf16 operands of the matrix instructions, shared by the warp-MMA and tcgen05 forwards.
//
// Widening bounds every one of these kernels below a few hundred tokens, so what counts is which pipe it loads.
// byte ^ 0x80 = q + 128 as an unsigned byte u; the bf16 with the bits 0x43:u is 128 + u for u < 128 and
// 256 + 2 (u - 128) above (the top bit of u lands in the exponent), i.e. with d = that - 256:
//   q < 0:  d = q           q >= 0:  d = 2 q
// so q = d - max(d, 0) / 2: three packed fused multiply-adds on two codes, every step exact (|2 q| <= 254 has at
// most seven significant bits).  Four codes cost 1 logic operation and 2 byte permutes on the 16-lane ALU pipe and
// 6 packed multiply-adds on the otherwise idle 32-lane FMA pipe: 9 issue slots, 6 ALU cycles.  The form before (f32
// magic number 2^23 + u, subtract, pack two f32) took 9 to 11 slots with 14 ALU cycles, as the pack runs on that pipe too.
#pragma once

#include "ptx_small.cuh"

namespace shrewq {
namespace {

// 4 INT8 codes (one word) -> two packed bf16x2 words, exactly: lo = codes 0, 1; hi = codes 2, 3
__device__ __forceinline__ void cvt_i8x4_bf16(uint32_t w, uint32_t &lo, uint32_t &hi) {
    constexpr uint32_t kOne = 0x3F803F80u, kMinus256 = 0xC380C380u, kMinusHalf = 0xBF00BF00u;
    const uint32_t u = w ^ 0x80808080u;
    const uint32_t p0 = __byte_perm(u, 0x43434343u, 0x4140), p1 = __byte_perm(u, 0x43434343u, 0x4342);
    lo = fma_bf16x2(fma_relu_bf16x2(p0, kOne, kMinus256), kMinusHalf, fma_bf16x2(p0, kOne, kMinus256));
    hi = fma_bf16x2(fma_relu_bf16x2(p1, kOne, kMinus256), kMinusHalf, fma_bf16x2(p1, kOne, kMinus256));
}

}  // namespace
}  // namespace shrewq
