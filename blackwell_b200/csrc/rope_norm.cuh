// Per-head RMSNorm followed by RoPE for one 128-wide head held by a warp, four consecutive elements per lane
// (the reference's caller-side head_norm_kernel and apply_rope_kernel, server/inference_server_int4_batched.cu:49-70).
// RoPE rotates interleaved pairs (2i, 2i+1) by theta = pos * base^(-2i/128).
#pragma once
#include "common.cuh"

namespace bw {

// base^(-2i/128) of a lane's two pairs: does not depend on the position.
__device__ __forceinline__ float2 rope_frequencies(float rope_base, int lane) {
    return make_float2(powf(rope_base, -2.0f * (float)(2 * lane) / 128.0f), powf(rope_base, -2.0f * (float)(2 * lane + 1) / 128.0f));
}
// cos, sin of the first pair's angle, then of the second's.
__device__ __forceinline__ float4 rope_angles(int pos, const float2& freq) {
    const float t0 = (float)pos * freq.x, t1 = (float)pos * freq.y;
    return make_float4(cosf(t0), sinf(t0), cosf(t1), sinf(t1));
}
// (Sums of products as explicit FMAs: every kernel gets the same bits.)
__device__ __forceinline__ float4 head_norm_turn(float4 v, const float4& w, float eps, const float4& r) {
    float ss = fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x)));
    ss = warp_sum(ss);
    const float is = rsqrtf(ss / 128.0f + eps);
    v.x = v.x * is * w.x; v.y = v.y * is * w.y; v.z = v.z * is * w.z; v.w = v.w * is * w.w;
    return make_float4(fmaf(v.x, r.x, -(v.y * r.y)), fmaf(v.x, r.y, v.y * r.x), fmaf(v.z, r.z, -(v.w * r.w)), fmaf(v.z, r.w, v.w * r.z));
}
__device__ __forceinline__ float4 head_norm_rope(float4 v, const float* norm_w, float eps, int pos, float rope_base, int lane) {
    return head_norm_turn(v, *reinterpret_cast<const float4*>(norm_w + 4 * lane), eps, rope_angles(pos, rope_frequencies(rope_base, lane)));
}

// Four floats -> four binary16 values, one 8-byte store.
__device__ __forceinline__ void store_half4(__half* dst, float4 v) {
    const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<const uint32_t*>(&a);
    u.y = *reinterpret_cast<const uint32_t*>(&b);
    *reinterpret_cast<uint2*>(dst) = u;
}

}  // namespace bw
