// Element-wise and per-row kernels of the config.json models: embedding lookup, norms on the sublayer output with the
// residual sum, gated group norm, short causal convolution with its step sizes.  fp32 arithmetic throughout; activations
// are read and written as bf16 (serving) or fp32 (32-bit mode).
#include <cuda_runtime.h>

#include <algorithm>

#include "host_util.h"
#include "lm_device.cuh"
#include "lm_ops.h"

namespace bw {
namespace lm {
namespace {

// Row kernels: a block per row, VEC neighbouring columns per access (4, or 1 for widths that are not a multiple of 4), the
// first KEEP vectors of a thread in registers.  Weights are fetched before the kernel waits for its predecessor.
// SHARES: a thread does the work of that many threads of the instance with SHARES times as many (vector j is that of share
// j % SHARES).  Their sums are kept apart and added in that instance's order, so that a row has the same bits either way and
// does not depend on how many rows there are.
template <int VEC, int KEEP, int SHARES>
struct RowVecs {
    static constexpr int kVec = VEC, kKeep = KEEP, kShares = SHARES;
    static_assert(KEEP % SHARES == 0 && SHARES <= 4, "shares");
    float v[kKeep][VEC];
    static __device__ __forceinline__ int col(int j) { return (j * blockDim.x + threadIdx.x) * VEC; }
    static __device__ __forceinline__ void get(const float* p, float (&x)[VEC]) {
        if constexpr (VEC == 4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(p);
        else x[0] = p[0];
    }
    static __device__ __forceinline__ void put(float* p, const float (&x)[VEC]) {
        if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(x);
        else p[0] = x[0];
    }
    static __device__ __forceinline__ void put(bf16* p, const float (&x)[VEC]) {
        if constexpr (VEC == 4) *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
        else p[0] = __float2bfloat16_rn(x[0]);
    }
    // p NULL, or beyond the row: `other`
    __device__ __forceinline__ void load(const float* p, int width, float other) {
#pragma unroll
        for (int j = 0; j < kKeep; ++j) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) v[j][e] = other;
            if (p && col(j) < width) get(p + col(j), v[j]);
        }
    }
    // Sum over the row of the squares of the kept values and of f(column) for the others; every thread gets it.
    template <typename F>
    __device__ __forceinline__ float sum_squares(int width, float* buf, F f) const {
        float s[kShares];
#pragma unroll
        for (int h = 0; h < kShares; ++h) s[h] = 0.f;
#pragma unroll
        for (int j = 0; j < kKeep; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) s[j % kShares] = fmaf(v[j][e], v[j][e], s[j % kShares]);
        beyond(width, [&](int i) { const float x = f(i); s[0] = fmaf(x, x, s[0]); });
        return block_sum(s, buf);
    }
    // f(column) for the columns that are not kept (none where SHARES > 1)
    template <typename F>
    static __device__ __forceinline__ void beyond(int width, F f) {
        for (int i = kKeep * blockDim.x * VEC + threadIdx.x; i < width; i += blockDim.x) f(i);
    }
};

// xb = x / rms(x) * next (next NULL: x) for the block's row x, of which `keep` holds the first values, `gain` those of next.
template <typename A, typename R>
__device__ __forceinline__ void next_input(A* xb, const float* x, const float* next, const R& keep, const R& gain, int width, float eps,
                                           float* buf) {
    constexpr int VEC = R::kVec;
    float f = 1.f;
    if (next) f = 1.0f / sqrtf(keep.sum_squares(width, buf, [&](int i) { return x[i]; }) / (float)width + eps);
#pragma unroll
    for (int j = 0; j < R::kKeep; ++j)
        if (R::col(j) < width) {
            float v[VEC];
#pragma unroll
            for (int e = 0; e < VEC; ++e) v[e] = keep.v[j][e] * f * gain.v[j][e];
            R::put(xb + R::col(j), v);
        }
    R::beyond(width, [&](int i) { xb[i] = from_f<A>(x[i] * f * (next ? next[i] : 1.f)); });
}

template <typename A, int VEC, int KEEP, int SHARES>
__global__ void __launch_bounds__(512) embed_kernel(float* x, A* xb, long ldxb, const bf16* table, long ldt, const int* tokens,
                                                    int width, int vocab, float scale, const float* next, float eps) {
    __shared__ float buf[32];
    typedef RowVecs<VEC, KEEP, SHARES> R;
    R gain, keep;
    gain.load(next, width, 1.f);
    pdl_trigger();
    pdl_wait();
    const long r = blockIdx.x;
    int tok = tokens[r];
    tok = tok < 0 ? 0 : tok >= vocab ? vocab - 1 : tok;
    const bf16* row = table + (long)tok * ldt;
    float* xr = x + r * width;
#pragma unroll
    for (int j = 0; j < R::kKeep; ++j) {
        const int c = R::col(j);
#pragma unroll
        for (int e = 0; e < VEC; ++e) keep.v[j][e] = c < width ? to_f(row[c + e]) * scale : 0.f;
        if (c < width) R::put(xr + c, keep.v[j]);
    }
    R::beyond(width, [&](int i) { xr[i] = to_f(row[i]) * scale; });   // read again by this thread alone
    next_input<A, R>(xb + r * ldxb, xr, next, keep, gain, width, eps, buf);
}

// ADD: x += y / rms(y) * w and xb = the next sublayer's input; otherwise xb = x / rms(x) * w for a listed row.
template <typename A, int VEC, int KEEP, int SHARES, bool ADD>
__global__ void __launch_bounds__(512) norm_kernel(float* x, A* xb, long ldxb, const float* y, const float* w, const float* next,
                                                   const int* rows, int width, float eps) {
    __shared__ float buf[32];
    typedef RowVecs<VEC, KEEP, SHARES> R;
    R weight, gain, keep, sum;
    weight.load(w, width, 0.f);
    if (ADD) gain.load(next, width, 1.f);
    pdl_trigger();
    pdl_wait();
    const int out_row = blockIdx.x;
    const long r = rows ? rows[out_row] : out_row;
    float* xr = x + r * width;
    const float* src = ADD ? y + r * width : xr;
    keep.load(src, width, 0.f);
    if (ADD) sum.load(xr, width, 0.f);
    const float rms = 1.0f / sqrtf(keep.sum_squares(width, buf, [&](int i) { return src[i]; }) / (float)width + eps);
    A* xo = xb + out_row * ldxb;
#pragma unroll
    for (int j = 0; j < R::kKeep; ++j) {
        const int c = R::col(j);
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            const float v = keep.v[j][e] * rms * weight.v[j][e];
            keep.v[j][e] = ADD ? sum.v[j][e] + v : v;
        }
        if (c < width) {
            if (ADD) R::put(xr + c, keep.v[j]);
            else R::put(xo + c, keep.v[j]);
        }
    }
    R::beyond(width, [&](int i) {
        const float v = src[i] * rms * w[i];
        if (ADD) xr[i] += v;
        else xo[i] = from_f<A>(v);
    });
    if (ADD) next_input<A, R>(xo, xr, next, keep, gain, width, eps, buf);
}

template <typename A>
__global__ void __launch_bounds__(256) gated_norm_kernel(A* out, long ldout, const float* o, long ldo, const A* gate, long ldg,
                                                         const float* w, int heads, int V, int groups, int gate_first,
                                                         float eps) {
    __shared__ float buf[32];
    pdl_trigger();
    pdl_wait();
    const int grp = blockIdx.x, t = threadIdx.x;
    const long r = blockIdx.y;
    const int part = heads * V / groups, c0 = grp * part, V8 = pad8(V);
    const float* orow = o + r * ldo;
    const A* grow = gate + r * ldg;
    float ss = 0.f;
    for (int i = t; i < part; i += 256) {
        const int c = c0 + i, col = (c / V) * V8 + c % V;
        float v = orow[col];
        if (gate_first) v *= silu_f(to_f(grow[col]));
        ss = fmaf(v, v, ss);
    }
    const float rms = 1.0f / sqrtf(block_sum(ss, buf) / (float)part + eps);
    for (int i = t; i < part; i += 256) {
        const int c = c0 + i, h = c / V, v0 = c - h * V, col = h * V8 + v0;
        const float v = orow[col] * silu_f(to_f(grow[col])) * rms * (w ? w[c] : 1.f);
        out[r * ldout + col] = from_f<A>(v);
        if (v0 == V - 1)
            for (int z = V; z < V8; ++z) out[r * ldout + h * V8 + z] = from_f<A>(0.f);
    }
}

// The same for groups that are a run of columns in memory (one head each with the gate last, or heads without padding with the gate
// first): a warp per group, `V` columns of it at a pitch of V8 = pad8(V), up to KV * 128 of them in registers, gate and weight in
// vectors of four where they are aligned (VEC).  GATE_FIRST sums in the order of the 256 threads of gated_norm_kernel, so that a
// group has the same bits there and here; it takes up to KV * 128 columns.
template <typename A, int KV, bool GATE_FIRST, bool VEC>
__global__ void __launch_bounds__(256) gated_norm_runs_kernel(A* out, long ldout, const float* o, long ldo, const A* gate, long ldg,
                                                              const float* w, int T, int groups, int V, float eps) {
    pdl_trigger();
    pdl_wait();
    const int g = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, V8 = pad8(V);
    const int row = g / groups, h = g - row * groups;
    if (row >= T) return;
    const long r = row;
    const float* orow = o + r * ldo + (long)h * V8;
    const A* grow = gate + r * ldg + (long)h * V8;
    const float* wrow = w ? w + (long)h * V : nullptr;
    A* dst = out + r * ldout + (long)h * V8;
    auto gates = [&](int c, float (&g)[4]) {   // silu of four gates
        if constexpr (VEC && sizeof(A) == 2) {
            const uint2 u = *reinterpret_cast<const uint2*>(grow + c);
            const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
            const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
            g[0] = lo.x; g[1] = lo.y; g[2] = hi.x; g[3] = hi.y;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) g[e] = c + e < V ? to_f(grow[c + e]) : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) g[e] = silu_f(g[e]);
    };
    auto load = [&](int c) {   // columns V .. V8 of o are zero
        float4 v = *reinterpret_cast<const float4*>(orow + c);
        if (GATE_FIRST) {
            float g[4];
            gates(c, g);
            v.x *= g[0]; v.y *= g[1]; v.z *= g[2]; v.w *= g[3];
        }
        return v;
    };
    float4 x[KV];
#pragma unroll
    for (int j = 0; j < KV; ++j) {
        const int c = j * 128 + lane * 4;
        x[j] = c < V8 ? load(c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float ss;
    if constexpr (GATE_FIRST) {
        // column c is thread c % 256's: vector j of a lane is that of warp 4 (j % 2) + lane / 8 there, its element e of lane
        // 4 (lane % 8) + e
        float a[8] = {};
#pragma unroll
        for (int j = 0; j < KV; ++j) {
            const float v[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) a[4 * (j & 1) + e] = fmaf(v[e], v[e], a[4 * (j & 1) + e]);
        }
        // a warp's tree: its lane bits 4, 3, 2 are lane bits 2, 1, 0 here, handing over half of the values at each; then e
        auto halve = [&](int bit, int n) {
            const bool upper = (lane & bit) != 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float keep = upper ? a[i + n] : a[i], send = upper ? a[i] : a[i + n];
                a[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
            }
        };
        halve(4, 4);
        halve(2, 2);
        halve(1, 1);
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
        ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += __shfl_sync(0xffffffffu, a[0], (i & 3) * 8 + (i >> 2) * 4);   // the warps in turn
    } else {
        ss = 0.f;
        auto add = [&](const float4& v) { ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss)))); };
#pragma unroll
        for (int j = 0; j < KV; ++j) add(x[j]);
        for (int c = KV * 128 + lane * 4; c < V8; c += 128) add(load(c));
        ss = warp_sum(ss);
    }
    const float rms = 1.0f / sqrtf(ss / (float)V + eps);
    auto emit = [&](int c, const float4& v) {
        float z[4] = {v.x, v.y, v.z, v.w}, f[4] = {1.f, 1.f, 1.f, 1.f};
        if (!GATE_FIRST) {
            float g[4];
            gates(c, g);
#pragma unroll
            for (int e = 0; e < 4; ++e) z[e] *= g[e];
        }
        if (wrow) {
            if constexpr (VEC) {
                *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(wrow + c);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) f[e] = c + e < V ? wrow[c + e] : 0.f;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) z[e] = c + e < V ? z[e] * rms * f[e] : 0.f;
        if constexpr (sizeof(A) == 2) *reinterpret_cast<uint2*>(dst + c) = make_uint2(pack_bf16(z[0], z[1]), pack_bf16(z[2], z[3]));
        else *reinterpret_cast<float4*>(dst + c) = make_float4(z[0], z[1], z[2], z[3]);
    };
#pragma unroll
    for (int j = 0; j < KV; ++j)
        if (j * 128 + lane * 4 < V8) emit(j * 128 + lane * 4, x[j]);
    if constexpr (!GATE_FIRST)
        for (int c = KV * 128 + lane * 4; c < V8; c += 128) emit(c, load(c));
}

// bf16, a head per group without padding, everything aligned, the gate last, up to KV * 128 columns: a warp per group, which requests
// outputs, gates and weight before it sums.  Two round trips to memory one after the other bounded the kernel above here: 2,502 rows
// of 32 x 128 columns 40 us, now 26.5 (31 with four groups a warp; 82 MB are 13 us, the exact divisions of the gates as long again),
// 4,096 rows of 8 x 512 40.8 -> 27, 32 rows of 8 x 512 5.9 -> 4.9.
template <int KV>
__global__ void __launch_bounds__(256) gated_norm_heads_kernel(bf16* out, long ldout, const float* o, long ldo, const bf16* gate, long ldg,
                                                               const float* w, int T, int groups, int V, float eps) {
    const int g = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const long row = g / groups, first = (long)(g - (int)row * groups) * V;
    float4 f[KV], x[KV];
    uint2 u[KV];
#pragma unroll
    for (int j = 0; j < KV; ++j) {
        const int c = j * 128 + lane * 4;
        f[j] = w && c < V ? __ldg(reinterpret_cast<const float4*>(w + first + c)) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
    pdl_trigger();
    pdl_wait();
    if (row >= T) return;
#pragma unroll
    for (int j = 0; j < KV; ++j) {
        const int c = j * 128 + lane * 4;
        x[j] = c < V ? *reinterpret_cast<const float4*>(o + row * ldo + first + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        u[j] = c < V ? *reinterpret_cast<const uint2*>(gate + row * ldg + first + c) : make_uint2(0, 0);
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < KV; ++j) ss = fmaf(x[j].x, x[j].x, fmaf(x[j].y, x[j].y, fmaf(x[j].z, x[j].z, fmaf(x[j].w, x[j].w, ss))));
    const float rms = 1.0f / sqrtf(warp_sum(ss) / (float)V + eps);
    auto lo = [](uint32_t pair) { return silu_f(__uint_as_float(pair << 16)); };
    auto hi = [](uint32_t pair) { return silu_f(__uint_as_float(pair & 0xFFFF0000u)); };
#pragma unroll
    for (int j = 0; j < KV; ++j) {
        const int c = j * 128 + lane * 4;
        if (c < V)
            *reinterpret_cast<uint2*>(out + row * ldout + first + c) =
                make_uint2(pack_bf16(x[j].x * lo(u[j].x) * rms * f[j].x, x[j].y * hi(u[j].x) * rms * f[j].y),
                           pack_bf16(x[j].z * lo(u[j].y) * rms * f[j].z, x[j].w * hi(u[j].y) * rms * f[j].w));
    }
}

// Conv channel of a padded column (counted from the start of the convolved part), -1 for padding.
__device__ __forceinline__ int conv_channel(const ConvArgs& c, int col) {
    const int V8 = pad8(c.V), N8 = pad8(c.N), x_cols = c.heads * V8;
    if (col < x_cols) return col % V8 < c.V ? (col / V8) * c.V + col % V8 : -1;
    const int b = col - x_cols;   // k groups, then q groups
    return b % N8 < c.N ? c.heads * c.V + (b / N8) * c.N + b % N8 : -1;
}
__host__ __device__ __forceinline__ int conv_cols(const ConvArgs& c) { return c.heads * pad8(c.V) + 2 * c.groups * pad8(c.N); }

// Step size (or strength) and log decay of rows [t0, t1) of head h.
__device__ __forceinline__ void step_sizes(const ConvArgs& c, int h, int t0, int t1) {
    const float a = -expf(c.A_log[h]), b = c.dt_bias[h];
    for (int t = t0; t < t1; ++t) {
        const float dt = softplus_f(c.dt_raw[(long)t * c.ld_dt + h] + b);
        c.log_decay[(long)t * c.heads + h] = a * dt;
        c.weight[(long)t * c.heads + h] = c.beta_raw ? sigmoid_f(c.beta_raw[(long)t * c.ld_dt + h]) : dt;
    }
}

constexpr int kConvRows = 8;   // rows per block

template <typename A>
__global__ void __launch_bounds__(128) conv_silu_kernel(const ConvArgs c, const Rows r) {
    pdl_wait();
    const int channels = c.heads * c.V + 2 * c.groups * c.N, cols = conv_cols(c);
    const int col = blockIdx.x * 128 + threadIdx.x, t0 = blockIdx.y * kConvRows, t1 = min(r.T, t0 + kConvRows);
    if (col < cols) {
        const int ch = conv_channel(c, col);
        if (ch < 0) {
            for (int t = t0; t < t1; ++t) static_cast<A*>(c.out)[(long)t * c.ldo + col] = from_f<A>(0.f);
            return;
        }
        const A* u = static_cast<const A*>(c.u) + c.off + col;
        const float* ring = c.ring + (long)r.slot * c.taps * channels + ch;
        const float bias = c.bias ? c.bias[ch] : 0.f;
        for (int t = t0; t < t1; ++t) {
            float y = bias;
            for (int j = 0; j < c.taps; ++j) {
                const int s = t - (c.taps - 1) + j, p = r.pos0 + s;
                float v = 0.f;
                if (s >= 0) v = to_f(u[(long)s * c.ldu]);
                else if (p >= 0) v = ring[(long)(p % c.taps) * channels];
                y = fmaf(c.w[ch * c.taps + j], v, y);
            }
            static_cast<A*>(c.out)[(long)t * c.ldo + col] = from_f<A>(silu_f(y));
        }
    } else if (col < cols + c.heads) {
        step_sizes(c, col - cols, t0, t1);
    }
}

// bf16 prompts and few taps: a thread takes eight rows of eight columns (always of one head block) and requests all it reads before
// it computes; taps and bias come before the dependency wait.  The last columns of blocks take the step sizes, a thread per row and
// head; the threads of the first rows, which alone read the ring, also store the last inputs there.  Serial chains bounded this: a
// thread that walked down 16 rows, its loads held back by its stores, and one that went through 16 step sizes took 22 us at 249 rows
// and 27 at 1,002 (4,352 / 8,192 columns), 67 at 4,096, the ring another 4; now 15 at 249, 18 at
// 1,002, 41 at 4,096, ring included (four rows a thread: the same).  Four prompts that begin together 2449 -> 2338 us.
constexpr int kConvRun = 8;
template <int TAPS>
__global__ void __launch_bounds__(128) conv_run_kernel(const ConvArgs c, const __grid_constant__ Runs rs) {
    const Run r = rs.run[blockIdx.z];
    const int channels = c.heads * c.V + 2 * c.groups * c.N, vec = blockIdx.x * 128 + threadIdx.x, t0 = blockIdx.y * kConvRun;
    if (t0 >= r.T) return;
    const int steps = (conv_cols(c) / 8 + 127) / 128;
    if (blockIdx.x >= steps) {
        const int i = (blockIdx.x - steps) * 128 + threadIdx.x, t = t0 + i / c.heads;
        pdl_wait();
        if (i < kConvRun * c.heads && t < r.T) step_sizes(c, i % c.heads, r.row0 + t, r.row0 + t + 1);
        return;
    }
    if (vec >= conv_cols(c) / 8) return;
    const int first = conv_channel(c, vec * 8);
    const bool whole = first >= 0 && conv_channel(c, vec * 8 + 7) == first + 7;   // no padding column
    float w[8 * TAPS], bias[8];   // w[e * TAPS + j]
    if (whole && ((uintptr_t)(c.w + (long)first * TAPS) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < 2 * TAPS; ++i)
            *reinterpret_cast<float4*>(w + 4 * i) = __ldg(reinterpret_cast<const float4*>(c.w + (long)first * TAPS) + i);
#pragma unroll
        for (int e = 0; e < 8; ++e) bias[e] = c.bias ? __ldg(c.bias + first + e) : 0.f;
    } else {   // padding columns: zero weights, zero output
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int ch = conv_channel(c, vec * 8 + e);
            bias[e] = ch >= 0 && c.bias ? c.bias[ch] : 0.f;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) w[e * TAPS + j] = ch >= 0 ? c.w[ch * TAPS + j] : 0.f;
        }
    }
    pdl_wait();
    const bf16* u = static_cast<const bf16*>(c.u) + r.row0 * c.ldu + c.off + vec * 8;
    bf16* out = static_cast<bf16*>(c.out) + r.row0 * c.ldo + vec * 8;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 x[TAPS - 1 + kConvRun], last[TAPS - 1];   // rows t0 - (TAPS - 1) ..; what the ring gets
#pragma unroll
    for (int i = 0; i < TAPS - 1 + kConvRun; ++i) {
        const int t = t0 - (TAPS - 1) + i;
        x[i] = t >= 0 && t < r.T ? *reinterpret_cast<const uint4*>(u + (long)t * c.ldu) : zero;
    }
    auto unpack = [](const uint4& v, float (&f)[8]) {
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(q[i] << 16);
            f[2 * i + 1] = __uint_as_float(q[i] & 0xFFFF0000u);
        }
    };
    if (t0 == 0) {
        float* ring = c.ring + (long)r.slot * TAPS * channels;
#pragma unroll
        for (int i = 0; i < TAPS - 1; ++i)   // (there are more rows than taps)
            last[i] = *reinterpret_cast<const uint4*>(u + (long)(r.T - (TAPS - 1) + i) * c.ldu);
#pragma unroll
        for (int i = 0; i < TAPS - 1; ++i) {
            const int p = r.pos0 - (TAPS - 1) + i;
            if (p < 0) continue;
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int ch = whole ? first + e : conv_channel(c, vec * 8 + e);
                f[e] = ch >= 0 ? ring[(long)(p % TAPS) * channels + ch] : 0.f;   // a bf16 number
            }
            x[i] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        }
#pragma unroll
        for (int i = 0; i < TAPS - 1; ++i) {
            float f[8];
            unpack(last[i], f);
            const int at = (r.pos0 + r.T - (TAPS - 1) + i) % TAPS;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int ch = whole ? first + e : conv_channel(c, vec * 8 + e);
                if (ch >= 0) ring[(long)at * channels + ch] = f[e];
            }
        }
    }
    float win[TAPS][8];   // win[i]: the input TAPS - 1 - i rows back
#pragma unroll
    for (int j = 0; j < TAPS - 1; ++j) unpack(x[j], win[j]);
#pragma unroll
    for (int i = 0; i < kConvRun; ++i) {
        if (t0 + i >= r.T) break;
        unpack(x[TAPS - 1 + i], win[TAPS - 1]);
        float y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            y[e] = bias[e];
#pragma unroll
            for (int j = 0; j < TAPS; ++j) y[e] = fmaf(w[e * TAPS + j], win[j][e], y[e]);
            y[e] = __fdividef(y[e], 1.0f + __expf(-y[e]));
#pragma unroll
            for (int j = 0; j < TAPS - 1; ++j) win[j][e] = win[j + 1][e];
        }
        *reinterpret_cast<uint4*>(out + (long)(t0 + i) * c.ldo) =
            make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
    }
}
template <int TAPS>
cudaError_t conv_run(const ConvArgs& c, const Runs& rs, cudaStream_t st) {
    const dim3 grid((conv_cols(c) / 8 + 127) / 128 + (kConvRun * c.heads + 127) / 128, (rs.longest() + kConvRun - 1) / kConvRun, rs.n);
    count_launch(1);
    return launch_pdl(conv_run_kernel<TAPS>, grid, dim3(128), 0, st, c, rs);
}

template <typename A>
__global__ void __launch_bounds__(128) conv_ring_kernel(const ConvArgs c, const Rows r) {
    pdl_wait();
    const int channels = c.heads * c.V + 2 * c.groups * c.N, col = blockIdx.x * 128 + threadIdx.x;
    const int ch = col < conv_cols(c) ? conv_channel(c, col) : -1;
    if (ch < 0) return;
    const A* u = static_cast<const A*>(c.u) + c.off + col;
    float* ring = c.ring + (long)r.slot * c.taps * channels + ch;
    for (int t = max(0, r.T - (c.taps - 1)); t < r.T; ++t) ring[(long)((r.pos0 + t) % c.taps) * channels] = to_f(u[(long)t * c.ldu]);
}

}  // namespace

namespace {

// threads of a row kernel: one access per thread, up to 512
int row_threads(int width, int vec) { return std::min(512, std::max(64, (width / vec + 31) / 32 * 32)); }

// Calls f<VEC, KEEP, SHARES>(threads) with the instance for this width.  Few rows: one access per thread, the shortest chain.  Rows
// for more than three quarters of the threads that the SMs hold: the work of four threads in one, whose block sums cost a quarter of
// the warps.  Measured, norm with residual, us, four in one / one each: 2,048 columns 5.0 / 6.4 at 445 rows, 5.6 / 7.6 at 592, 25.4 /
// 34.2 at 4,096; 1,024 columns 4.1 / 4.0 at 592, 4.9 / 5.6 at 890; 512 columns 2.7 / 2.4 at 592, 3.5 / 3.4 at 1,000, 4.9 / 5.6 at
// 1,800.  Two in one beyond 2,048 columns gains nothing (4,096 rows of 4,096: 57.6 / 55.2).
template <typename F>
cudaError_t by_width(int width, int T, F f) {
    if (width % 4 != 0) return f.template operator()<1, 4, 1>(row_threads(width, 1));
    const int threads = row_threads(width, 4);
    if (width <= 2048 && threads % 128 == 0 && (long)T * threads > 1536l * sm_count(current_device()))
        return f.template operator()<4, 4, 4>(threads / 4);
    return width <= 2048 ? f.template operator()<4, 1, 1>(threads) : width <= 4096 ? f.template operator()<4, 2, 1>(threads)
                                                                                  : f.template operator()<4, 4, 1>(threads);
}
template <typename A>
struct Embed {
    float* x; void* xb; long ldxb; const bf16* table; long ldt; const int* tokens; int T, width, vocab; float scale; const float* next;
    float eps; cudaStream_t st;
    template <int VEC, int KEEP, int SHARES>
    cudaError_t operator()(int threads) const {
        return launch_pdl(embed_kernel<A, VEC, KEEP, SHARES>, dim3(T), dim3(threads), 0, st, x, static_cast<A*>(xb), ldxb, table, ldt,
                          tokens, width, vocab, scale, next, eps);
    }
};
template <typename A, bool ADD>
struct Norm {
    float* x; void* xb; long ldxb; const float *y, *w, *next; const int* rows; int T, width; float eps; cudaStream_t st;
    template <int VEC, int KEEP, int SHARES>
    cudaError_t operator()(int threads) const {
        return launch_pdl(norm_kernel<A, VEC, KEEP, SHARES, ADD>, dim3(T), dim3(threads), 0, st, x, static_cast<A*>(xb), ldxb, y, w, next,
                          rows, width, eps);
    }
};

}  // namespace

cudaError_t embed(float* x, void* xb, long ldxb, const bf16* table, long ldt, const int* tokens, int T, int width, int vocab,
                  float scale, const float* next, float eps, int f32, cudaStream_t st) {
    count_launch(1);
    return f32 ? by_width(width, T, Embed<float>{x, xb, ldxb, table, ldt, tokens, T, width, vocab, scale, next, eps, st})
               : by_width(width, T, Embed<bf16>{x, xb, ldxb, table, ldt, tokens, T, width, vocab, scale, next, eps, st});
}

cudaError_t norm_add(float* x, void* xb, long ldxb, const float* y, const float* w, const float* next, int T, int width, float eps,
                     int f32, cudaStream_t st) {
    count_launch(1);
    return f32 ? by_width(width, T, Norm<float, true>{x, xb, ldxb, y, w, next, nullptr, T, width, eps, st})
               : by_width(width, T, Norm<bf16, true>{x, xb, ldxb, y, w, next, nullptr, T, width, eps, st});
}

cudaError_t norm_rows(void* xb, long ldxb, const float* x, const float* w, const int* rows, int T, int width, float eps, int f32,
                      cudaStream_t st) {
    count_launch(1);
    float* xm = const_cast<float*>(x);
    return f32 ? by_width(width, T, Norm<float, false>{xm, xb, ldxb, nullptr, w, nullptr, rows, T, width, eps, st})
               : by_width(width, T, Norm<bf16, false>{xm, xb, ldxb, nullptr, w, nullptr, rows, T, width, eps, st});
}

// A warp per group where a group is a run of columns and the warps in flight make up for its serial chain, otherwise a block per
// group.  Measured with the gate first, us, a warp / a block: groups of 128 columns 2.0 / 2.2 at 32 groups in all, 50 / 249 at
// 131,072; of 512 columns 3.6 / 3.0 at 8, 3.8 / 3.8 at 256, 6.3 / 11.8 at 2,368, 33 / 130 at 32,768; of 520 to 1,024 columns
// 7.2 / 6.5 (1,024) and 4.5 / 4.4 (520) at 592, 8.8 / 10.8 (1,024) and 4.6 / 6.8 (520) at 800, 37 / 111 at 16,384.  Longer groups
// lie beyond a warp's registers.
template <typename A>
static cudaError_t gated_norm_as(A* out, long ldout, const float* o, long ldo, const A* gate, long ldg, const float* w, int T, int heads,
                                 int V, int groups, int gate_first, float eps, cudaStream_t st) {
    auto aligned = [](const void* p, long ld, size_t elem) { return ((uintptr_t)p | (size_t)ld * elem) % (4 * elem) == 0; };
    const int part = heads * V / groups;
    const long all = (long)T * groups;
    const bool rows = aligned(o, ldo, 4) && aligned(out, ldout, sizeof(A));
    const bool vec = part % 8 == 0 && aligned(gate, ldg, sizeof(A)) && (uintptr_t)w % 16 == 0;
    const int sms = sm_count(current_device());
    const bool runs = gate_first ? V % 8 == 0 && vec && (part <= 128 || (part <= 512 && all >= 2 * sms) || (part <= 1024 && all > 4 * sms))
                                 : groups == heads;
    if (!rows || !runs || all > 0x7ffffff0)
        return launch_pdl(gated_norm_kernel<A>, dim3(groups, T), dim3(256), 0, st, out, ldout, o, ldo, gate, ldg, w, heads, V, groups,
                          gate_first, eps);
    if constexpr (sizeof(A) == 2) {
        if (!gate_first && vec && part <= 512) {
            auto kern = part > 256 ? gated_norm_heads_kernel<4> : part > 128 ? gated_norm_heads_kernel<2> : gated_norm_heads_kernel<1>;
            return launch_pdl(kern, dim3((unsigned)(all + 7) / 8), dim3(256), 0, st, out, ldout, o, ldo, gate, ldg, w, T, groups, part, eps);
        }
    }
    const bool wide = part > 512;
    auto kern = gate_first ? (wide ? gated_norm_runs_kernel<A, 8, true, true> : gated_norm_runs_kernel<A, 4, true, true>)
                : vec && wide ? gated_norm_runs_kernel<A, 8, false, true> : gated_norm_runs_kernel<A, 4, false, false>;
    if constexpr (sizeof(A) == 4) {
        if (!gate_first && vec && !wide) kern = gated_norm_runs_kernel<A, 4, false, true>;
    }
    return launch_pdl(kern, dim3((unsigned)(all + 7) / 8), dim3(256), 0, st, out, ldout, o, ldo, gate, ldg, w, T, groups, part, eps);
}

cudaError_t gated_norm(void* out, long ldout, const float* o, long ldo, const void* gate, long ldg, const float* w, int T,
                       int heads, int V, int groups, int gate_first, float eps, int f32, cudaStream_t st) {
    if (groups < 1 || (heads * V) % groups != 0) return cudaErrorInvalidValue;
    count_launch(1);
    return f32 ? gated_norm_as(static_cast<float*>(out), ldout, o, ldo, static_cast<const float*>(gate), ldg, w, T, heads, V, groups,
                               gate_first, eps, st)
               : gated_norm_as(static_cast<bf16*>(out), ldout, o, ldo, static_cast<const bf16*>(gate), ldg, w, T, heads, V, groups,
                               gate_first, eps, st);
}

bool conv_runs_supported(const ConvArgs& c) { return c.taps >= 2 && c.taps <= 4; }

cudaError_t conv_runs(const ConvArgs& c, const Runs& rs, cudaStream_t st) {
    return c.taps == 2 ? conv_run<2>(c, rs, st) : c.taps == 3 ? conv_run<3>(c, rs, st) : c.taps == 4 ? conv_run<4>(c, rs, st) : cudaErrorInvalidValue;
}

cudaError_t conv_silu(const ConvArgs& c, const Rows& r, int f32, cudaStream_t st) {
    const int n = conv_cols(c) + c.heads;
    const dim3 grid((n + 127) / 128, (r.T + kConvRows - 1) / kConvRows), ring((conv_cols(c) + 127) / 128), block(128);
    if (!f32 && r.T >= 16 && conv_runs_supported(c)) return conv_runs(c, one_run(r), st);
    count_launch(1);
    const cudaError_t e = f32 ? launch_pdl(conv_silu_kernel<float>, grid, block, 0, st, c, r) : launch_pdl(conv_silu_kernel<bf16>, grid, block, 0, st, c, r);
    if (e != cudaSuccess) return e;
    count_launch(1);
    return f32 ? launch_pdl(conv_ring_kernel<float>, ring, block, 0, st, c, r) : launch_pdl(conv_ring_kernel<bf16>, ring, block, 0, st, c, r);
}

}  // namespace lm
}  // namespace bw
