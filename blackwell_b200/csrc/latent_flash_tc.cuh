// Prompt attention over expanded keys and values (see latent_attention.cuh) on the 5th-generation tensor cores: causal flash
// attention with a sink and a gate per head.  Unrotated keys and values have 64 or 128 columns per head, the rotated part 64.
//
// Block (128 query rows, head), two per SM: while one block's softmax runs, the tensor cores work for the other.  Warps 0-3
// softmax, a thread per query row; warps 4 and 6 TMA (64 keys, 64 values at a time, 128-byte swizzle), warp 5 MMA issuer.
//   S = Q K^T      Q and K in shared memory; two accumulators of 64 columns, so that the next scores are on their way while the
//                  softmax has these
//   P              over the scores' columns, as the bf16 A operand: 32 columns of high parts, 32 of remainders (16 significant bits,
//                  as in the mma.sync kernels)
//   O += P V       V from shared memory as it lies there ([key][column]: B is MN-major)
// O stays in tensor memory.  It is brought to a new maximum only when that grew by more than 2^8 (exp2 of the difference is exact
// bookkeeping: P and the sum use the same base, and the last step divides one by the other); otherwise the softmax never waits for
// the second product (the conditional rescaling published with FlashAttention-4).
// What bounds it: per 64 keys and 128 rows 896 cycles of the tensor pipe (384 for 192 columns of S, 512 for P V with its remainders)
// against some 500 issue slots of each softmax warp.
// Measured 1.6 us a tile where a block has its SM to itself, 1.9 us for the two tiles of two blocks: the softmax is the chain (a second
// buffer for the values changes nothing, 133.9 and 135.7 us at 4096 rows).  Times beside latent_expanded in the .cu file.
// All waits are bounded; a wait that gives up raises an abort flag.
#pragma once
#include <cuda.h>

#include "gemm_w4a8_tc.cuh"
#include "lm_device.cuh"
#include "lm_ops.h"

namespace bw {
namespace lm {

constexpr int kTcFlashQ = 128, kTcFlashK = 64;
constexpr int kTcFlashThreads = 224;
constexpr int kTcPanel = kTcFlashK * 128;   // bytes of 64 keys x 64 columns

// ND, NV: 64-column panels of the unrotated keys and of the values
template <int ND, int NV>
struct TcFlashShape {
    static constexpr int kQ = (ND + 1) * 2 * kTcPanel, kK = (ND + 1) * kTcPanel, kV = NV * kTcPanel;
    static constexpr int kSmem = 1024 + 1024 + kQ + kK + kV;   // alignment, barriers
    static constexpr int kOCol = 128;                          // tensor memory: S / P twice, then O
    static constexpr int kFullQ = 0, kFullK = 1, kEmptyK = 2, kFullV = 3, kDrain = 4, kFullS = 5, kFullP = 7, kDoneO = 9;   // the last three twice
};

struct TcFlashArgs {
    const float* gate;   // [T][ld32]
    const float* sink;   // [heads]
    bf16* out;           // [T][ldout]
    long ld32, ldout;
    int heads, T, pos0, q_head, k_head, v_head, v_first, k_rot;   // columns per head, first value column, the rotated keys' first column
    float sl2;           // score scale, base 2
    int* status;
};

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
        "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
        "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
          "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
          "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
          "r"(v[31]), "r"(addr)
        : "memory");
}
// 128-byte swizzle.  K-major rows of 128 bytes: 8-row groups `sbo` bytes apart.  MN-major: rows are k, 8-row groups `sbo` bytes apart,
// panels of 64 columns `lbo` bytes apart.
__device__ __forceinline__ uint64_t flash_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
template <int ND, int NV>
__global__ void __launch_bounds__(kTcFlashThreads, 2)
latent_flash_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                       const __grid_constant__ CUtensorMap map_rot, const TcFlashArgs a) {
    using Sh = TcFlashShape<ND, NV>;
    constexpr int NP = ND + 1, V = NV * 64;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sq = smem_u32(smem + 1024), sk = sq + Sh::kQ, sv = sk + Sh::kK, bar0 = smem_u32(smem), flag = bar0 + 516;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 516);
    const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
    auto bar = [&](int i) { return bar0 + 8 * i; };
    auto wait = [&](int i, uint32_t parity) { mbar_wait_or_abort(bar(i), parity, flag); };
    if (t == 0) {
        for (int i = 0; i < 11; ++i) mbar_init(bar(i), i == Sh::kFullP || i == Sh::kFullP + 1 ? 4 : 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 5) {
        tc::tmem_alloc(bar0 + 512, 256);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(smem + 512), 0);
    pdl_trigger();
    // heads fastest, longest rows first
    const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kTcFlashQ, h = blockIdx.x;
    const int nkeys = a.pos0 + min(a.T, q0 + kTcFlashQ), tiles = (nkeys + kTcFlashK - 1) / kTcFlashK;

    if (warp == 4) {
        if (lane == 0) {
            pdl_wait();
            mbar_expect_tx(bar(Sh::kFullQ), Sh::kQ);
            for (int p = 0; p < NP; ++p)
                tc::tma_load_2d(sq + p * 2 * kTcPanel, &map_q, h * a.q_head + 64 * p, q0, bar(Sh::kFullQ));
            int j = 0;
            for (; j < tiles; ++j) {
                wait(Sh::kEmptyK, (j & 1) ^ 1);   // (at once the first time)
                if (*abort_flag) break;
                mbar_expect_tx(bar(Sh::kFullK), Sh::kK);
                for (int p = 0; p < ND; ++p)
                    tc::tma_load_2d(sk + p * kTcPanel, &map_kv, h * a.k_head + 64 * p, j * kTcFlashK, bar(Sh::kFullK));
                tc::tma_load_2d(sk + ND * kTcPanel, &map_rot, a.k_rot, j * kTcFlashK, bar(Sh::kFullK));
            }
            if (*abort_flag) {   // gave up: the copies in flight end before the block does
                mbar_wait(bar(Sh::kFullQ), 0);
                if (j > 0) mbar_wait(bar(Sh::kFullK), (j - 1) & 1);
            }
        }
    } else if (warp == 6) {
        if (lane == 0) {
            pdl_wait();
            int j = 0;
            for (; j < tiles; ++j) {
                if (j > 0) wait(Sh::kDoneO + ((j - 1) & 1), ((j - 1) >> 1) & 1);   // the values before have been multiplied
                if (*abort_flag) break;
                mbar_expect_tx(bar(Sh::kFullV), Sh::kV);
                for (int p = 0; p < NV; ++p)
                    tc::tma_load_2d(sv + p * kTcPanel, &map_kv, a.v_first + h * a.v_head + 64 * p, j * kTcFlashK, bar(Sh::kFullV));
            }
            if (*abort_flag && j > 0) mbar_wait(bar(Sh::kFullV), (j - 1) & 1);
        }
    } else if (warp == 5) {
        // The whole warp walks the loop, one elected lane issues.  S of the next tile goes out before this tile's second product, once
        // the P that lay where it goes has been multiplied.
        constexpr uint32_t id_s = tc::idesc_bf16(kTcFlashK), id_o = tc::idesc_bf16(V, true);
        const bool elected = tc::elect_one();
        auto scores = [&](int j) {
            wait(Sh::kFullK, j & 1);
            tc::tc_fence_after();
            if (elected) {
#pragma unroll
                for (int p = 0; p < NP; ++p)
#pragma unroll
                    for (int k = 0; k < 4; ++k)   // 16 k = 32 bytes further inside the swizzle atom
                        tc::tc_mma_bf16(tmem + (j & 1) * 64, flash_desc(sq + p * 2 * kTcPanel, 16, 1024) + 2 * k,
                                  flash_desc(sk + p * kTcPanel, 16, 1024) + 2 * k, id_s, p + k > 0 ? 1u : 0u);
                tc::tc_commit(bar(Sh::kFullS + (j & 1)));
                tc::tc_commit(bar(Sh::kEmptyK));
            }
            __syncwarp();
        };
        pdl_wait();   // the limit of a wait counts this kernel's own progress
        wait(Sh::kFullQ, 0);
        scores(0);
        for (int j = 0; j < tiles && !*abort_flag; ++j) {
            if (j > 0) wait(Sh::kDoneO + ((j - 1) & 1), ((j - 1) >> 1) & 1);
            if (j + 1 < tiles) scores(j + 1);
            wait(Sh::kFullP + (j & 1), (j >> 1) & 1);
            wait(Sh::kFullV, j & 1);
            tc::tc_fence_after();
            if (elected) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {   // 16 keys: two 8-row groups
                    const uint64_t v = flash_desc(sv, kTcPanel, 1024) + k * (2048 >> 4);
                    const uint32_t p = tmem + (j & 1) * 64 + 8 * k;
                    tc::tc_mma_bf16_ta(tmem + Sh::kOCol, p + 32, v, id_o, j + k > 0 ? 1u : 0u);
                    tc::tc_mma_bf16_ta(tmem + Sh::kOCol, p, v, id_o, 1u);
                }
                tc::tc_commit(bar(Sh::kDoneO + (j & 1)));
            }
            __syncwarp();
        }
        if (elected) tc::tc_commit(bar(Sh::kDrain));   // whatever became of the others: no MMA in flight when the tensor memory is freed
        __syncwarp();
        mbar_wait(bar(Sh::kDrain), 0);
    } else {
        const int q = q0 + t;                                  // this thread's query row
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        float m = 0.f, l = 0.f;
        pdl_wait();
        for (int j = 0; j < tiles && !*abort_flag; ++j) {
            uint32_t s[64];
            const uint32_t at = lanes + (j & 1) * 64;
            wait(Sh::kFullS + (j & 1), (j >> 1) & 1);
            if (j > 1) wait(Sh::kDoneO + (j & 1), ((j - 2) >> 1) & 1);   // long done; no phase of it goes by unseen
            tc::tc_fence_after();
            tmem_ld32(at, s);
            tmem_ld32(at + 32, s + 32);
            tc::tmem_wait_ld();
            if ((j + 1) * kTcFlashK > a.pos0 + q0 + 1) {       // some row of the block does not see all of these keys
                const int seen = a.pos0 + q + 1 - j * kTcFlashK;
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (i >= seen) s[i] = 0xFF800000u;
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(s[i]));
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.sl2;
            if (j == 0) {
                m = fmaxf(top, -1e30f);   // (finite, were all of these scores -inf)
            } else if (__any_sync(0xffffffffu, top - m > 8.f)) {
                wait(Sh::kDoneO + ((j - 1) & 1), ((j - 1) >> 1) & 1);   // O is complete up to the tile before
                tc::tc_fence_after();
                const float base = fmaxf(m, top), f = exp2_fast(m - base);
                m = base;
                l *= f;
#pragma unroll
                for (int c = 0; c < V; c += 32) {
                    uint32_t o[32];
                    tmem_ld32(lanes + Sh::kOCol + c, o);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                    tmem_st32(lanes + Sh::kOCol + c, o);
                }
            }
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 64; ++i) {
                const float p = exp2_fast(fmaf(__uint_as_float(s[i]), a.sl2, -m));
                sum[i & 3] += p;
                s[i] = __float_as_uint(p);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    split_bf16(__uint_as_float(s[2 * (c + i)]), __uint_as_float(s[2 * (c + i) + 1]), hi[i], lo[i]);
                tc::tmem_st16(at + c, hi);
                tc::tmem_st16(at + 32 + c, lo);
            }
            tc::tmem_wait_st();
            tc::tc_fence_before();
            __syncwarp();
            mbar_arrive_by(lane == 0, bar(Sh::kFullP + (j & 1)));
        }
        wait(Sh::kDoneO + ((tiles - 1) & 1), ((tiles - 1) >> 1) & 1);
        tc::tc_fence_after();
        if (!*abort_flag) {
            const float sink = a.sink[h] * 1.4426950408889634f, mm = fmaxf(m, sink), sc = exp2f(m - mm);
            const float f = q < a.T ? sc / (l * sc + exp2f(sink - mm)) * sigmoid_f(a.gate[(long)q * a.ld32 + h]) : 0.f;
            bf16* out = a.out + (long)q * a.ldout + h * a.v_head;
#pragma unroll
            for (int c = 0; c < V; c += 32) {
                uint32_t o[32];
                tmem_ld32(lanes + Sh::kOCol + c, o);
                tc::tmem_wait_ld();
                if (q < a.T) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint32_t v[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            v[e] = pack_bf16(__uint_as_float(o[i + 2 * e]) * f, __uint_as_float(o[i + 2 * e + 1]) * f);
                        *reinterpret_cast<uint4*>(out + c + i) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                }
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 256);
    }
    if (t == 0 && *abort_flag) atomicExch(a.status, kStatusMbarTimeout);
}

}  // namespace lm
}  // namespace bw
