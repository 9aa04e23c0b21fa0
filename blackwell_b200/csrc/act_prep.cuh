// Quantizing a row of activations on its own (not inside a GEMV): what the prep kernels share.  The element arithmetic and the
// rounding are those of make_xblock / quantize_block, so that every path gets the same integers.
#pragma once
#include "gemv_w4_stream.cuh"

namespace bw {

// The arrival counters of the product that follows start at zero whatever became of earlier calls (a product that gave up in a
// wait leaves tiles half counted).  Every thread of a prep kernel of 256 threads a block, after its dependency wait.
__device__ __forceinline__ void zero_counters(unsigned int* counters, int n) {
    const int step = gridDim.x * gridDim.y * 256;
    for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * 256 + threadIdx.x; i < n; i += step) counters[i] = 0;
}
// Sum of squares of one row by 256 threads -> 1 / rms, the same on every thread.
__device__ __forceinline__ float row_rstd(const GemvArgs& a, int m, int t, float* part) {
    float ss = 0.f;
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(a.x) + (size_t)m * a.x_stride);
    for (int i = t; i < a.K / 4; i += 256) {
        const float4 f = p[i];
        ss = fmaf(f.x, f.x, ss); ss = fmaf(f.y, f.y, ss); ss = fmaf(f.z, f.z, ss); ss = fmaf(f.w, f.w, ss);
    }
    ss = warp_sum(ss);
    if ((t & 31) == 0) part[t >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += part[w];
    return rsqrtf(tot / (float)a.K + a.eps);
}
// E consecutive elements of an activation row after the prologue; the element arithmetic is that of make_xblock.
template <int E>
__device__ __forceinline__ void load_elements(const GemvArgs& a, int m, int e0, float rstd, float (&v)[E]) {
    const size_t at = (size_t)m * a.x_stride + e0;
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
        float* o = v + 4 * i;
        if (a.xkind == kXHalf) {
            const uint2 u = reinterpret_cast<const uint2*>(static_cast<const __half*>(a.x) + at)[i];
            const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
            const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
            o[0] = f0.x; o[1] = f0.y; o[2] = f1.x; o[3] = f1.y;
            continue;
        }
        const float4 f = reinterpret_cast<const float4*>(static_cast<const float*>(a.x) + at)[i];
        o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
        if (a.xkind == kXFloatNorm) {
            const float4 gw = reinterpret_cast<const float4*>(a.norm_w + e0)[i];
            o[0] = o[0] * gw.x * rstd; o[1] = o[1] * gw.y * rstd; o[2] = o[2] * gw.z * rstd; o[3] = o[3] * gw.w * rstd;
        } else if (a.xkind == kXSwiglu) {
            const float4 u = reinterpret_cast<const float4*>(static_cast<const float*>(a.x2) + at)[i];
            o[0] = silu_mul(o[0], u.x); o[1] = silu_mul(o[1], u.y); o[2] = silu_mul(o[2], u.z); o[3] = silu_mul(o[3], u.w);
        }
    }
}
// The rounding of quantize_block for E elements of a block with scale sc: the integer is the low byte of q[i].
template <int E>
__device__ __forceinline__ void round_elements(const float (&v)[E], float am, float sc, uint32_t (&q)[E]) {
    const float rcp = 1.0f / sc;
    bool exact_needed = !(am < 3.0e38f);
#pragma unroll
    for (int i = 0; i < E; ++i) {
        const float r = v[i] * rcp;
        const float mg = r + kMagicFloat;
        const float ri = mg - kMagicFloat;
        exact_needed |= !(fabsf(fabsf(r - ri) - 0.5f) > 3e-5f);
        q[i] = __float_as_uint(mg);
    }
    if (exact_needed) {
#pragma unroll
        for (int i = 0; i < E; ++i) q[i] = (uint32_t)quant_i8(v[i], sc);
    }
}

}  // namespace bw
