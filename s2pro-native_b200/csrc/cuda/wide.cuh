/* Outputs of a linear whose K range was split over several CTAs (wide_gemm, skinny.cu): f32 partials that the kernel which
 * consumes the outputs adds in piece order, so that no CTA has to wait for the others and no launch is spent on it. */
#pragma once
#include "common.cuh"
#include "ops.h"

namespace s2p {

/* outputs n .. n + 3 (n a multiple of 4) of batch row m, before the rounding to bf16; AHEAD pieces are asked for at once (a matrix of 2560 rows
 * comes in seven, one of 6144 in three) */
template <int AHEAD = 4>
__device__ __forceinline__ float4 wide_part4(const WidePart& p, int n, int m) {
    const float* at = p.partial + ((size_t)(n >> 7) * p.pieces * p.M + m) * 128 + (n & 127);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q0 = 0; q0 < p.pieces; q0 += AHEAD) {
        float4 v[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; q++)
            v[q] = q0 + q < p.pieces ? __ldcg(reinterpret_cast<const float4*>(at + (size_t)(q0 + q) * p.M * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int q = 0; q < AHEAD; q++)
            if (q0 + q < p.pieces) { s.x += v[q].x; s.y += v[q].y; s.z += v[q].z; s.w += v[q].w; }
    }
    if (p.scales) {
        const float4 f = *reinterpret_cast<const float4*>(p.scales + n);
        s.x = __fmul_rn(s.x, f.x); s.y = __fmul_rn(s.y, f.y); s.z = __fmul_rn(s.z, f.z); s.w = __fmul_rn(s.w, f.w);
    }
    return s;
}
template <int AHEAD = 4>
__device__ __forceinline__ uint2 wide_part4_bf16(const WidePart& p, int n, int m) {
    const float4 s = wide_part4<AHEAD>(p, n, m);
    return make_uint2((uint32_t)__bfloat16_as_ushort(f2bf(s.x)) | ((uint32_t)__bfloat16_as_ushort(f2bf(s.y)) << 16),
                      (uint32_t)__bfloat16_as_ushort(f2bf(s.z)) | ((uint32_t)__bfloat16_as_ushort(f2bf(s.w)) << 16));
}
/* 8 consecutive bf16 as the f16 unit of a matrix operand; `int4`: in the element order packed INT4 weights are converted to */
__device__ __forceinline__ uint4 wide_unit(const uint4& v, int int4) {
    __half2 h[4];
    if (int4) {
        h[0] = __floats2half2_rn(bf_lo(v.x), bf_lo(v.z));
        h[1] = __floats2half2_rn(bf_hi(v.x), bf_hi(v.z));
        h[2] = __floats2half2_rn(bf_lo(v.y), bf_lo(v.w));
        h[3] = __floats2half2_rn(bf_hi(v.y), bf_hi(v.w));
    } else {
        h[0] = __floats2half2_rn(bf_lo(v.x), bf_hi(v.x));
        h[1] = __floats2half2_rn(bf_lo(v.y), bf_hi(v.y));
        h[2] = __floats2half2_rn(bf_lo(v.z), bf_hi(v.z));
        h[3] = __floats2half2_rn(bf_lo(v.w), bf_hi(v.w));
    }
    return make_uint4(*reinterpret_cast<uint32_t*>(&h[0]), *reinterpret_cast<uint32_t*>(&h[1]), *reinterpret_cast<uint32_t*>(&h[2]),
                      *reinterpret_cast<uint32_t*>(&h[3]));
}
/* The units of an activation matrix lie [k / 8][rows padded to a power of two of at least 16]: log2 of that */
__host__ __device__ inline int wide_lg(int rows) {
    int lg = 4;
    while ((1 << lg) < rows) lg++;
    return lg;
}

}  // namespace s2p
