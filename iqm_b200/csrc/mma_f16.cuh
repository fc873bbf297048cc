// FP16 tensor-core tiles (mma.sync m16n8k16, FP32 accumulation) and the packing of their operands.
//
// Split-precision products take operands as hi + lo FP16 pairs (hi = fp16(v), lo = fp16(v - hi)) and form
// A B ~ A_hi B_hi + A_hi B_lo + A_lo B_hi, about 21 significant bits per product instead of 11.
#pragma once

#include <cuda_fp16.h>

namespace iqm {

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned h2_bits(__half2 h) { return *reinterpret_cast<unsigned *>(&h); }

// (x, y) as an FP16 pair, x in the low half (the lower matrix index of a fragment register).
__device__ __forceinline__ unsigned pack_h2(float x, float y) { return h2_bits(__floats2half2_rn(x, y)); }

// hi = fp16(x, y), lo = fp16((x, y) - hi)
__device__ __forceinline__ void split_h2(float x, float y, unsigned &hi, unsigned &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 hf = __half22float2(h);
    hi = h2_bits(h);
    lo = h2_bits(__floats2half2_rn(x - hf.x, y - hf.y));
}

}  // namespace iqm
