// fp32 values as two fp16 parts for tensor-core products of fp32 precision (mlp_chain.cu, mlp_grad.cu), and the powers of two that bring them into range
#pragma once
#include "common.cuh"
#include <cuda_fp16.h>

namespace b200rl {

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi){
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void split_pair(float2 v, uint32_t& lead, uint32_t& rest){
    lead = pack_f16(v.x, v.y);
    const float2 back = __half22float2(*reinterpret_cast<const __half2*>(&lead));
    const float2 d = __ffma2_rn(back, make_float2(-1.0f, -1.0f), v);
    rest = pack_f16(d.x, d.y);
}
// biased exponent of the piece's largest magnitude, clamped so that the scale 2^(14 - e) and its inverse are normal numbers
__device__ __forceinline__ uint32_t scale_exponent(float largest){
    const uint32_t e = (__float_as_uint(largest) >> 23) & 0xFFu;
    return e < 15u ? 15u : e > 254u ? 254u : e;
}
__device__ __forceinline__ float scale_of(uint32_t e){ return __uint_as_float((268u - e) << 23); }
__device__ __forceinline__ float inverse_scale_of(uint32_t e){ return __uint_as_float((e - 14u) << 23); }

}  // namespace b200rl
