// Launcher and kernels of the bf16 tcgen05 form of the W4A8 product.  See gemm_w4a8_wide.cuh for the arithmetic.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "../../include/blackwell_b200.h"
#include "act_prep.cuh"
#include "gemm_w4a8_wide.cuh"
#include "host_util.h"
#include "tensor_map.h"

namespace bw {
namespace wide {

// ----------------------------------------------------------------------------------------------------------
// Activation prep of the tensor-core kernel: quantizes every sequence once (int8 rule; plain / RMSNorm / SwiGLU, or int8 as
// it comes) and stores it in the layout of the MMA's B operand, chunk by chunk:
//   chunk c: [block 0..15][k half][NP rows x 16 B: eight bf16]   then   [block 0..15][NP] fp32 scales
// The eight elements of a half are in the order in which the unpack takes the nibbles of a word: 0 4 1 5 2 6 3 7.
// k-blocks >= K/16 of the last chunk are zero (their weights multiply as zero too); rows >= M are left as they are: an
// accumulator column is one sequence.  Zeroes the arrival counters of equal shares (`ncounters`, or 0).  Grid (ceil(chunks / 8), M),
// 256 threads of eight elements; starts early under programmatic dependent launch.
// ----------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) prep_x_kernel(unsigned char* xb, const GemvArgs a, int NP, int nchunks,
                                                     unsigned int* counters, int ncounters) {
    __shared__ float part[8];
    pdl_trigger();
    pdl_wait();   // the activations come from the kernel before
    zero_counters(counters, ncounters);
    const int m = blockIdx.y, t = threadIdx.x;
    const float rstd = a.xkind == kXFloatNorm ? row_rstd(a, m, t, part) : 1.f;
    const int e0 = (blockIdx.x * 256 + t) * 8;
    const bool valid = e0 < a.K;   // K % 16 == 0: the two threads of a block are valid or not together
    uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float sc = 0.f;
    if (a.xkind == kXInt8) {
        if (valid) {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(static_cast<const int8_t*>(a.x) + (size_t)m * a.K + e0));
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] = (i < 4 ? u.x : u.y) >> (8 * (i & 3));
            if ((t & 1) == 0) sc = __ldg(a.xsc + (size_t)m * (a.K / 16) + (e0 >> 4));
        }
    } else {
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (valid) load_elements<8>(a, m, e0, rstd, v);
        float am = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) am = fmaxf(am, fabsf(v[i]));
        am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
        if (valid) {
            sc = quant_scale_i8(am);
            round_elements<8>(v, am, sc, q);
        }
    }
    const int kb = e0 >> 4, c = kb / kBlocksPerChunk, b = kb % kBlocksPerChunk;
    if (c >= nchunks) return;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 p = __floats2bfloat162_rn((float)(int8_t)q[i], (float)(int8_t)q[i + 4]);
        o[i] = *reinterpret_cast<const uint32_t*>(&p);
    }
    unsigned char* chunk = xb + (size_t)c * xchunk_bytes(NP);
    *reinterpret_cast<uint4*>(chunk + ((size_t)(2 * b + (t & 1)) * NP + m) * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    if ((t & 1) == 0) reinterpret_cast<float*>(chunk + xop_bytes(NP))[b * NP + m] = sc;
}

// ----------------------------------------------------------------------------------------------------------
// Shape of an instantiation: NE sequences = columns of the MMA.
// ----------------------------------------------------------------------------------------------------------
template <int NE>
struct WideShape {
    static constexpr int NP = NE;                        // MMA N
    static constexpr int CW = NE / 4;                    // sequences per worker thread, for each of its two rows
    static constexpr bool kTight = NE > 48;              // two pairs of accumulators do not fit beside the A operand
    static constexpr int DB = kTight ? 1 : 2;            // k-blocks per accumulator stage
    static constexpr int DS = kTight ? 3 : 2;            // accumulator stages, of a pair or (kTight) of a block
    static constexpr int kDCols = DB * 2 * NP;           // tensor-memory columns of a stage: [block][row group][NP]
    static constexpr int kACol = DS * kDCols;            // first column of the two A slots: [row group][block of the pair][q sh, q sl][8]
    static constexpr int BYTES = kWBytes + xchunk_bytes(NP);
    static constexpr int S = (kMaxDynSmem - 2048) / BYTES < 5 ? (kMaxDynSmem - 2048) / BYTES : 5;
    static constexpr int kSmem = 2048 + S * BYTES;       // up to 1023 bytes of alignment, 1 KB of barriers and flags
    static_assert(BYTES % 1024 == 0 && kACol + 2 * 64 <= 512 && S >= 2, "shape");
    static_assert(NE * kRows * 4 <= S * BYTES, "the tile for the cluster reduction takes the place of the operand ring");
    // barriers
    static constexpr int kFullW = 0;             // + stage: nibbles landed
    static constexpr int kFullX = kFullW + S;    // + stage: activations and their scales landed
    static constexpr int kEmpty = kFullX + S;    // + stage: used up by the workers (and so by the MMAs before them)
    static constexpr int kFullA = kEmpty + S;    // + A slot: stored by the workers
    static constexpr int kFullD = kFullA + 2;    // + accumulator stage: its MMAs have completed
    static constexpr int kRead = kFullD + DS;    // kTight: the first block of a pair has been read
    static constexpr int kTeam = kRead + 1;      // all workers together, at the end of a tile
    static constexpr int kDrain = kTeam + 1;
    static constexpr int kNumBars = kDrain + 1;
    static_assert(kNumBars * 8 <= 512, "barriers");
};

// Place in a ring of three stages.
struct Stage {
    uint32_t at = 0, phase = 0;
    __device__ __forceinline__ void step() {
        if (++at == 3) { at = 0; phase ^= 1; }
    }
};

// Chunk range of a CTA, counted over (tile, chunk of the tile).
__device__ __forceinline__ void chunk_range(const WideArgs& a, int cta, int grid, int& w0, int& w1) {
    if (a.csize == 0) {         // whole tiles
        w0 = (int)((long long)a.tiles * cta / grid) * a.nchunks;
        w1 = (int)((long long)a.tiles * (cta + 1) / grid) * a.nchunks;
    } else if (a.csize > 1) {   // a cluster shares one tile
        const int tile = cta / a.csize, r = cta - tile * a.csize;
        w0 = tile * a.nchunks + (int)((long long)a.nchunks * r / a.csize);
        w1 = tile * a.nchunks + (int)((long long)a.nchunks * (r + 1) / a.csize);
    } else {                    // equal shares of everything; a share may begin and end inside a tile
        const long long all = (long long)a.tiles * a.nchunks;
        w0 = (int)(all * cta / grid);
        w1 = (int)(all * (cta + 1) / grid);
    }
}
// The CTA whose share holds chunk w (equal shares).
__device__ __forceinline__ int chunk_owner(const WideArgs& a, int w, int grid) {
    const long long all = (long long)a.tiles * a.nchunks;
    return (int)((((long long)w + 1) * grid - 1) / all);
}

template <int NE>
__global__ void __launch_bounds__(kThreads, 1)
gemm_w4a8_wide_kernel(const __grid_constant__ CUtensorMap map_w, const WideArgs a) {
    using Sh = WideShape<NE>;
    constexpr int NP = Sh::NP, CW = Sh::CW, DB = Sh::DB, DS = Sh::DS, S = Sh::S;
    constexpr bool kTight = Sh::kTight;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = smem + 1024;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(smem + 512);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 516);
    volatile int* last = reinterpret_cast<volatile int*>(smem + 520);
    const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;   // the warp index is uniform
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8 * i; };
    auto wait = [&](int i, uint32_t parity) {   // by a whole warp (whose lanes see the same) or by one lane
        if (mbar_wait_quick(bar(i), parity)) return true;
        *abort_flag = 1;
        return false;
    };
    if (t == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(bar(Sh::kFullW + i), 1);
            mbar_init(bar(Sh::kFullX + i), 1);
            mbar_init(bar(Sh::kEmpty + i), kWorkers);
        }
        for (int i = 0; i < 2; ++i) mbar_init(bar(Sh::kFullA + i), kWorkers);
        for (int i = 0; i < DS; ++i) mbar_init(bar(Sh::kFullD + i), 1);
        mbar_init(bar(Sh::kRead), kWorkers);
        mbar_init(bar(Sh::kTeam), kWorkers);
        mbar_init(bar(Sh::kDrain), 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(smem + 512), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
    pdl_trigger();

    int w0, w1;
    chunk_range(a, blockIdx.x, gridDim.x, w0, w1);
    const int total = w1 - w0;

    if (warp < 4) regs_fewer<kRegsFew>();
    if (warp == 0) {
        if (lane == 0) {
            // -------------------------------------------------------------------------------- producer
            auto load_w = [&](int n) {
                const int w = w0 + n, tile = w / a.nchunks, s = n % S;
                mbar_expect_tx(bar(Sh::kFullW + s), kWBytes);
                tma_load_2d(smem_u32(ring + s * Sh::BYTES), &map_w, (w - tile * a.nchunks) * (kKc / 2), tile * kRows, bar(Sh::kFullW + s));
            };
            const int ahead = min(total, S);
            for (int n = 0; n < ahead; ++n) load_w(n);   // the weights do not depend on the kernel before
            pdl_wait();
            int n = 0;
            for (; n < total; ++n) {
                const int s = n % S, c = (w0 + n) % a.nchunks;
                if (n >= S) {
                    if (!wait(Sh::kEmpty + s, ((n / S) & 1) ^ 1)) break;
                    load_w(n);
                }
                mbar_expect_tx(bar(Sh::kFullX + s), xchunk_bytes(NP));
                bulk_g2s_plain(smem_u32(ring + s * Sh::BYTES + kWBytes), a.xb + (size_t)c * xchunk_bytes(NP), xchunk_bytes(NP), bar(Sh::kFullX + s));
            }
            if (n < total)   // gave up: the copies in flight end before the block does
                for (int i = max(0, n - S); i < n; ++i) {
                    mbar_wait(bar(Sh::kFullW + i % S), (i / S) & 1);
                    mbar_wait(bar(Sh::kFullX + i % S), (i / S) & 1);
                }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------------------------ MMA issuer
        // The whole warp walks the loop, one elected lane issues (see elect_one).  Stored A operands of a pair also say that
        // every worker has read the accumulators of the pair before the last, whose stage this pair takes over; of three
        // single-block stages the second block of a pair takes over that of the first block of the pair before, whose reading it
        // waits for (before the first block's commit, so that the phase waited for cannot be followed by another unseen).
        constexpr uint32_t idesc = idesc_bf16(NP);
        const bool elected = elect_one();
        bool ok = true;
        uint32_t ph = 0;   // phase of the A slots
        pdl_wait();        // see the workers' first wait for activations
        Stage st;
        for (int n = 0; n < total && ok; ++n) {
            const int s = n % S;
            if (!(ok = wait(Sh::kFullX + s, (n / S) & 1))) break;
            const uint32_t xop = smem_u32(ring + s * Sh::BYTES + kWBytes);
#pragma unroll 1
            for (int p = 0; p < kPairs && ok; p += 2, ph ^= 1) {
#pragma unroll
                for (int as = 0; as < 2; ++as) {   // pair p + as
                    if (!(ok = wait(Sh::kFullA + as, ph))) break;
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t dst = kTight ? st.at : as;
                        if (elected) {
                            const uint64_t db = smem_desc(xop + (p + as + 8 * j) * NP * 32, NP * 16, 128);
#pragma unroll
                            for (int g = 0; g < 2; ++g) {
                                const uint32_t d = tmem + dst * Sh::kDCols + ((DB == 2 ? 2 * j : 0) + g) * NP;
                                const uint32_t av = tmem + Sh::kACol + as * 64 + g * 32 + j * 16;
                                tc_mma_bf16_ta(d, av, db, idesc, 0u);
                                tc_mma_bf16_ta(d, av + 8, db, idesc, 1u);
                            }
                        }
                        __syncwarp();
                        if (kTight && j == 0 && (as > 0 || n + p > 0)) {
                            if (!(ok = wait(Sh::kRead, as ^ 1))) break;   // the pair before
                            tc_fence_after();
                        }
                        if (elected && (kTight || j == 1)) tc_commit(bar(Sh::kFullD + dst));
                        st.step();
                        __syncwarp();
                    }
                    if (!ok) break;
                }
            }
        }
        if (!ok) {   // gave up: the MMAs in flight end before the tensor memory is freed
            if (elected) tc_commit(bar(Sh::kDrain));
            __syncwarp();
            mbar_wait(bar(Sh::kDrain), 0);
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------------------------ workers
        regs_more<kRegsWork>();
        const int wt = t - 128, q = warp & 3, cg = (warp - 4) >> 2;   // TMEM lanes 32 q ..; one of four warps on them
        // unpack: row group `ug`, block p + 8 uj of the pair; scaling: rows `row` and `row + 128`, sequences [cg CW, cg CW + CW)
        const int ug = cg & 1, uj = cg >> 1, urow = ug * 128 + q * 32 + lane, row = q * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        const uint32_t a_addr = lanes + Sh::kACol + ug * 32 + uj * 16, d_addr = lanes + cg * CW;
        // This row's eight scales of a chunk (blocks 8 uj ..), in the largest accesses that the row pitch allows; zero past the
        // end of the row.
        auto load_scales = [&](int w, uint32_t (&v)[4]) {
            const int tile = w / a.nchunks, b0 = (w - tile * a.nchunks) * kBlocksPerChunk + 8 * uj, left = a.nkb - b0;
            const __half* p = a.Wsc + (size_t)min(tile * kRows + urow, a.N - 1) * a.nkb + b0;
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = 0;
            if (a.sc_gran == 16) {
                if (left > 0)
                    asm volatile("ld.global.nc.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p));
            } else if (a.sc_gran == 8) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (left > 4 * i) asm volatile("ld.global.nc.L2::256B.v2.u32 {%0, %1}, [%2];" : "=r"(v[2 * i]), "=r"(v[2 * i + 1]) : "l"(p + 4 * i));
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (left > 2 * i) asm volatile("ld.global.nc.L2::256B.u32 %0, [%1];" : "=r"(v[i]) : "l"(p + 2 * i));
            }
        };
        float acc[2][CW];
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int j = 0; j < CW; ++j) acc[g][j] = 0.f;
        auto store = [&](int m, int n, float v) {
            const size_t yi = (size_t)m * a.y_stride + n;
            a.y[yi] = a.residual ? v + a.residual[yi] : v;
        };
        // acc += accumulators of a block whose scales are at x
        auto scale = [&](const uint32_t (&v)[2][CW], const float* x) {
#pragma unroll
            for (int i = 0; i < CW; i += 4) {
                float xv[4];
                *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(x + i);
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int g = 0; g < 2; ++g) acc[g][i + j] = fmaf(__uint_as_float(v[g][i + j]), xv[j], acc[g][i + j]);
            }
        };
        int team = 0;
        auto team_sync = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(Sh::kTeam));
            return wait(Sh::kTeam, team++ & 1);
        };
        // The tile of chunk `wlast` is finished (or this CTA's share of it): results out, accumulators back to zero.
        auto finish = [&](int wlast) -> bool {
            const int tile = wlast / a.nchunks, first = tile * a.nchunks, begin = max(w0, first);
            const int row0 = tile * kRows + row;
            if (a.csize > 1) {   // one tile per cluster: this CTA's share goes where the ring was, once all have left it
                if (!team_sync()) return false;
                float* sm = reinterpret_cast<float*>(ring) + row;
#pragma unroll
                for (int j = 0; j < CW; ++j) {
                    sm[(cg * CW + j) * kRows] = acc[0][j];
                    sm[(cg * CW + j) * kRows + 128] = acc[1][j];
                }
                return true;
            }
            // (y may still be read, the partial tiles still be summed by the kernels before: past the dependency wait since chunk 0)
            if (begin == first && wlast == first + a.nchunks - 1) {
#pragma unroll
                for (int j = 0; j < CW; ++j) {
                    const int m = cg * CW + j;
                    if (m < a.M) {
                        if (row0 < a.N) store(m, row0, acc[0][j]);
                        if (row0 + 128 < a.N) store(m, row0 + 128, acc[1][j]);
                    }
                }
            } else {
                // a share that begins or ends inside the tile: the last CTA to arrive adds all shares in the order of K
                float* mine = a.partial + (size_t)(2 * blockIdx.x + (begin == w0 ? 0 : 1)) * NE * kRows + row;
#pragma unroll
                for (int j = 0; j < CW; ++j)
                    if (cg * CW + j < a.M) {
                        mine[(cg * CW + j) * kRows] = acc[0][j];
                        mine[(cg * CW + j) * kRows + 128] = acc[1][j];
                    }
                __threadfence();
                if (!team_sync()) return false;
                const int grid = gridDim.x, i0 = chunk_owner(a, first, grid), i1 = chunk_owner(a, first + a.nchunks - 1, grid);
                if (wt == 0) *last = (atomicAdd(&a.tickets[tile], 1u) == (unsigned)(i1 - i0)) ? 1 : 0;
                if (!team_sync()) return false;
                if (*last) {
                    __threadfence();
                    int b0, b1;
                    chunk_range(a, i0, grid, b0, b1);
                    const int head = b0 / a.nchunks == tile ? 0 : 1;   // which of its two shares the first CTA left here
                    const float* p0 = a.partial + (size_t)(2 * i0 + head) * NE * kRows + row;
                    const float* p1 = a.partial + (size_t)(2 * i0 + 2) * NE * kRows + row;
                    // share by share, every column's load of a share in flight together
                    auto add = [&](const float* p, bool first_share) {
#pragma unroll
                        for (int j = 0; j < CW; ++j)
#pragma unroll
                            for (int g = 0; g < 2; ++g) {
                                const float v = cg * CW + j < a.M ? __ldcg(p + (cg * CW + j) * kRows + 128 * g) : 0.f;
                                acc[g][j] = first_share ? v : acc[g][j] + v;
                            }
                    };
                    add(p0, true);
#pragma unroll 1
                    for (int i = 0; i < i1 - i0; ++i) add(p1 + (size_t)i * 2 * NE * kRows, false);
#pragma unroll
                    for (int j = 0; j < CW; ++j)
                        if (cg * CW + j < a.M) {
                            if (row0 < a.N) store(cg * CW + j, row0, acc[0][j]);
                            if (row0 + 128 < a.N) store(cg * CW + j, row0 + 128, acc[1][j]);
                        }
                }
                if (!team_sync()) return false;   // `last` is written again
            }
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int j = 0; j < CW; ++j) acc[g][j] = 0.f;
            return true;
        };

        uint32_t cur[4], next[4];
        load_scales(w0, next);
        bool ok = true;
        Stage st;
        const float* xs = nullptr;   // scales of the chunk whose accumulators are being read
        // Unpack this thread's block of a pair into A slot `as` and hand it to the MMA issuer.  The MMAs that read the slot
        // before are those of the pair before the last, whose accumulators this warp has seen.
        auto unpack = [&](int as, uint32_t wlo, uint32_t whi, float sc) {
            const ScaleParts sp = split_scale(sc);
            uint32_t v[16];
            unpack_word(wlo, sp, v, v + 8);
            unpack_word(whi, sp, v + 4, v + 12);
            tmem_st16(a_addr + as * 64, v);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(Sh::kFullA + as));
        };
        // Scale the accumulators of a pair (slot `as`, phase ph): blocks at xs + x and 8 blocks further.
        auto take = [&](int as, uint32_t ph, const float* x) -> bool {
            if constexpr (DB == 2) {
                if (!wait(Sh::kFullD + as, ph)) return false;
                tc_fence_after();
                uint32_t v0[2][CW], v1[2][CW];
#pragma unroll
                for (int g = 0; g < 2; ++g) tmem_ld<CW>(d_addr + as * Sh::kDCols + g * NP, v0[g]);
#pragma unroll
                for (int g = 0; g < 2; ++g) tmem_ld<CW>(d_addr + as * Sh::kDCols + (2 + g) * NP, v1[g]);
                tmem_wait_ld();
                scale(v0, x);
                scale(v1, x + 8 * NP);
            } else {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (!wait(Sh::kFullD + st.at, st.phase)) return false;
                    tc_fence_after();
                    uint32_t v0[2][CW];
#pragma unroll
                    for (int g = 0; g < 2; ++g) tmem_ld<CW>(d_addr + st.at * Sh::kDCols + g * NP, v0[g]);
                    st.step();
                    tmem_wait_ld();
                    if (j == 0) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(Sh::kRead));
                    }
                    scale(v0, x + 8 * j * NP);
                }
            }
            tc_fence_before();   // read before the next pair's arrival lets the MMAs write there
            return true;
        };
        uint32_t ph = 0;   // phase of the pairs of this loop iteration
        for (int n = 0; n <= total && ok; ++n) {
            const int s = n % S;
            const unsigned char* src = ring + s * Sh::BYTES + urow * 128;
            if (n < total) {
#pragma unroll
                for (int i = 0; i < 4; ++i) cur[i] = next[i];
                if (n + 1 < total) load_scales(w0 + n + 1, next);
                if (!(ok = wait(Sh::kFullW + s, (n / S) & 1))) break;
            }
#pragma unroll 1
            for (int p = 0; p < kPairs; p += 2, ph ^= 1) {
                uint4 w4;
                float2 f;
                if (n < total) {
                    w4 = *reinterpret_cast<const uint4*>(src + (((4 * uj + p / 2) ^ (urow & 7)) << 4));
                    f = __half22float2(*reinterpret_cast<const __half2*>(&cur[0]));
                    cur[0] = cur[1]; cur[1] = cur[2]; cur[2] = cur[3];
                    unpack(0, w4.x, w4.y, f.x);
                }
                if (n + p > 0 && !(ok = take(1, ph ^ 1, xs + (p == 0 ? kPairs - 1 : p - 1) * NP))) break;
                if (p == 0) {
                    if (n > 0) {   // that was the last pair of chunk n - 1
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(Sh::kEmpty + (n - 1) % S));
                        if ((n == total || (w0 + n) % a.nchunks == 0) && !(ok = finish(w0 + n - 1))) break;
                    }
                    if (n == total) break;
                    // The limit of a wait counts this kernel's own progress, not the time until the activations' producers are done
                    // (an exchange before them may wait longer for a late rank).
                    if (n == 0) pdl_wait();
                    if (!(ok = wait(Sh::kFullX + s, (n / S) & 1))) break;
                    xs = reinterpret_cast<const float*>(ring + s * Sh::BYTES + kWBytes + xop_bytes(NP)) + cg * CW;
                }
                unpack(1, w4.z, w4.w, f.y);
                if (!(ok = take(0, ph, xs + p * NP))) break;
            }
        }
        if (a.csize > 1) {
            __syncwarp();
            cluster_sync_all();   // every CTA's share of the tile is in its shared memory
            const int tile = w0 / a.nchunks, rank = blockIdx.x % a.csize;
            const int r0 = kRows * rank / a.csize, nr = kRows * (rank + 1) / a.csize - r0;
            const uint32_t base = smem_u32(ring);
            if (!*abort_flag)
                for (int i = wt; i < nr * a.M; i += kWorkers * 32) {
                    const int m = i / nr, r = r0 + i - m * nr, n = tile * kRows + r;
                    float p[8];
#pragma unroll
                    for (int c = 0; c < 8; ++c) p[c] = c < a.csize ? ld_dsmem(base + (m * kRows + r) * 4, c) : 0.f;
                    // neighbours first: eight sums in a row had 2 % more error (2048 x 5632, against 64 bits)
                    const float sum = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
                    if (n < a.N) store(m, n, sum);
                }
            __syncwarp();
            cluster_sync_all();   // nobody leaves while its share may still be read
        }
    }
    if (warp < 4 && a.csize > 1) {
        __syncwarp();
        cluster_sync_all();
        cluster_sync_all();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (t == 0 && *abort_flag) atomicExch(a.status, kStatusMbarTimeout);
}

// ----------------------------------------------------------------------------------------------------------
// Host side
// ----------------------------------------------------------------------------------------------------------
static std::atomic<int> g_split{0};
void set_split(int v) { g_split = v; }

// Sequences an instantiation handles: those of M rounded up.
static int cols_of(int M) { return M <= 32 ? 32 : M <= 48 ? 48 : 64; }

// Makes an instance launchable on the current device, once.  The roles' register shares are drawn from what the launch allocates.
template <int NE>
static cudaError_t prepare() {
    static std::once_flag once[kMaxDevices];
    static cudaError_t usable[kMaxDevices];
    const int dev = current_device();
    std::call_once(once[dev], [&] {
        cudaFuncAttributes fa;
        cudaError_t e = cudaFuncSetAttribute(gemm_w4a8_wide_kernel<NE>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideShape<NE>::kSmem);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, gemm_w4a8_wide_kernel<NE>);
        if (e == cudaSuccess && fa.numRegs < 96) e = cudaErrorInvalidConfiguration;
        if (e != cudaSuccess) cudaGetLastError();
        usable[dev] = e;
    });
    return usable[dev];
}
static bool usable(int NE) { return (NE == 32 ? prepare<32>() : NE == 48 ? prepare<48>() : prepare<64>()) == cudaSuccess; }

// Clusters of `csize` CTAs that are resident at once on the current device, at most (the SMs of a cluster share a GPC).
static int max_clusters(int csize) {
    static std::atomic<int> cached[kMaxDevices][9];
    std::atomic<int>& c = cached[current_device()][csize];
    int n = c.load();
    if (n > 0) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(csize);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = WideShape<64>::kSmem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = csize;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (prepare<64>() != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_w4a8_wide_kernel<64>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    c = n;
    return n;
}

// Launch geometry and scratch layout of one call: [tickets][activation chunks][partial tiles].
struct WideLayout {
    int NE, nchunks, tiles, csize, grid;
    float us;   // estimate of the call's time
    size_t xb_off, part_off, part_bytes;
};
// Equal shares of all chunks, or a cluster per tile: whichever the estimate says.  Measured (us, prep included; 4096 x 4096,
// 6144 x 4096, 21888 x 4096, 4096 x 10944): a chunk of a tile takes 5.1 / 5.9 / 8.2 at 32 / 48 / 64 sequences; a cluster adds 6
// to its longest share, equal shares add 10 and about 0.9 (at 32) for every share that the last CTA of a tile adds up.  Clusters of
// 2 to 8 resident at once on a B200: 74, 45, 33, 26, 22, 15, 15.
static WideLayout layout_of(int M, int N, int K) {
    WideLayout l;
    l.NE = cols_of(M);
    l.nchunks = (K + kKc - 1) / kKc;
    l.tiles = (N + kRows - 1) / kRows;
    const int sms = sm_count(current_device()), force = g_split.load();
    const long long all = (long long)l.tiles * l.nchunks;
    const float chunk = l.NE == 32 ? 5.1f : l.NE == 48 ? 5.9f : 8.2f;
    l.csize = 1;
    l.grid = (int)(all < sms ? all : sms);
    l.us = chunk * (float)((all + l.grid - 1) / l.grid) + 10.f + 0.9f * (float)l.NE / 32.f * (float)(l.grid / l.tiles + 1);
    for (int cs = 8; cs > 1; --cs)
        if (cs <= l.nchunks && l.tiles <= max_clusters(cs)) {   // the largest that is resident at once
            const float us = 6.f + chunk * (float)((l.nchunks + cs - 1) / cs);
            if (us < l.us) { l.us = us; l.csize = cs; }
            break;
        }
    if (force > 8) l.csize = 1;
    else if (force > 1 && force <= l.nchunks) l.csize = force;
    else if (force == 1) l.csize = 0;
    // The arrival counters own a region of fixed size at the front of the block.  Matrices with more tiles than counters are dealt out by whole tiles.
    if (l.csize == 1 && (size_t)l.tiles * sizeof(unsigned int) > tc::kTicketBytes) l.csize = 0;
    if (l.csize == 0) l.grid = l.tiles < sms ? l.tiles : sms;
    if (l.csize > 1) l.grid = l.tiles * l.csize;
    l.part_bytes = l.csize == 1 ? (size_t)l.grid * 2 * l.NE * kRows * sizeof(float) : 0;
    l.xb_off = tc::kTicketBytes;
    l.part_off = (l.xb_off + (size_t)l.nchunks * xchunk_bytes(l.NE) + 255) & ~(size_t)255;
    return l;
}
static std::atomic<int> g_force{0};
void set_force(int v) { g_force = v; }
// Whether a call of 17 to 64 sequences is faster here than in the int8 form (gemm_w4a8_tc.cu), by the estimates of both.  That
// one takes 2.27 us for a chunk of 128 rows up to 32 sequences and 3.33 above (it computes 64 columns then), its tiles come in
// whole rounds of one per SM, and a K split adds 2.2 / 3.6 us per part.  Measured, this form / that one: 6144 x 4096 26 / 31 at 32
// sequences, 31 / 46 at 48, 40 / 47 at 64; 21888 x 4096 62 / 80, 72 / 115, 95 / 115; 3072 x 2048 11 / 26, 13 / 42, 16 / 42;
// 4096 x 10944 42 / 41, 48 / 58, 65 / 59; 4096 x 12288 46 / 42, 54 / 60, 72 / 60; 32768 x 2048 47 / 45, 55 / 64, 71 / 64;
// 151643 x 4096 327 / 329, 383 / 480, 526 / 482: the rule takes the faster one in each but the last at 32, where they are level.
// And whether every sum is a shorter chain of chunks than there, or neither splits K: a narrow matrix of very long rows is split
// finer by the int8 form (300 x 32768, 64 chunks: 4 against 16 in a cluster of eight), and its error against 64 bits was 1.8e-7
// where this form had 2.9e-7.  With the shorter chains here it is 0.6 to 0.99 of that form's (2048 to 24576 rows of 2048 to 12288,
// 17 to 64 sequences; 1.02 at most over 60 random sizes, 1.15 where the chains were equal).
bool preferred(int M, int N, int K) {
    if (M <= 16 || !usable(cols_of(M))) return false;   // the int8 form takes the same operands
    if (g_force.load() != 0) return g_force.load() > 0;
    const int sms = sm_count(current_device()), tiles = (N + 127) / 128, nchunks = (K + kKc - 1) / kKc;
    const int ks = std::max(1, std::min(sms / tiles, nchunks));
    const int boxes = ((nchunks + 1) / 2 + ks - 1) / ks, rounds = (tiles * ks + sms - 1) / sms;
    const float chunks = (float)(std::min(2 * boxes, nchunks) * rounds);
    const float us = M <= 32 ? 2.27f * chunks + (ks > 1 ? 8.f + 2.2f * ks : 6.f) : 3.33f * chunks + (ks > 1 ? 10.f + 3.6f * ks : 6.f);
    const WideLayout l = layout_of(M, N, K);
    const int share = (int)(((long long)l.tiles * l.nchunks + l.grid - 1) / l.grid);
    const int chain = l.csize == 0 ? nchunks : std::min(share, nchunks);
    const int theirs = std::min(2 * boxes, nchunks);
    return l.us < us && (chain < theirs || theirs == nchunks);
}
// Enough for every batch up to M.
size_t scratch_bytes(int M, int N, int K) {
    if (M <= 16 || N < 1 || K < 32) return 0;
    size_t most = 0;
    for (int m = 32; m <= cols_of(std::min(M, 64)); m += 16) {
        const WideLayout l = layout_of(m, N, K);
        most = std::max(most, l.part_off + l.part_bytes);
    }
    return most;
}

template <int NE>
static cudaError_t launch_n(const CUtensorMap& map_w, const WideArgs& t, int grid, cudaStream_t st) {
    auto kern = gemm_w4a8_wide_kernel<NE>;
    const cudaError_t e0 = prepare<NE>();
    if (e0 != cudaSuccess) return e0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = WideShape<NE>::kSmem;
    cfg.stream = st;
    cudaLaunchAttribute la[2];
    la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    la[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    la[1].id = cudaLaunchAttributeClusterDimension;
    la[1].val.clusterDim.x = t.csize > 1 ? t.csize : 1;
    la[1].val.clusterDim.y = la[1].val.clusterDim.z = 1;
    cfg.attrs = la;
    cfg.numAttrs = t.csize > 1 ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map_w, t);
    count_launch(1);
    return e != cudaSuccess ? e : cudaPeekAtLastError();
}

// y = W . q8(prologue(x)) for up to 64 sequences; what tc::eligible accepts.  `a` carries the operands as for the streaming
// kernel (x kinds int8 / f16 / f32 / f32+norm / swiglu; binary16 weight scales).
cudaError_t launch(const GemvArgs& a, int M, cudaStream_t st) {
    const WideLayout lay = layout_of(M, a.N, a.K);
    unsigned char* scratch = nullptr;
    cudaError_t e = tc::scratch(lay.part_off + lay.part_bytes, st, &scratch);
    if (e != cudaSuccess) return e;

    CUtensorMap map_w;
    const cuuint64_t dims[2] = {(cuuint64_t)(a.K / 2), (cuuint64_t)a.N};
    const cuuint64_t strides[1] = {(cuuint64_t)(a.K / 2)};
    const cuuint32_t box[2] = {(cuuint32_t)(kKc / 2), (cuuint32_t)kRows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = lm::encode_fn()(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(a.W), dims, strides,
                                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;

    e = launch_pdl(prep_x_kernel, dim3((lay.nchunks + 7) / 8, M), dim3(256), 0, st, scratch + lay.xb_off, a, lay.NE, lay.nchunks,
                   reinterpret_cast<unsigned int*>(scratch), lay.csize == 1 ? lay.tiles : 0);
    count_launch(1);
    if (e != cudaSuccess) return e;

    WideArgs t{};
    t.y = a.y; t.residual = a.residual; t.y_stride = a.y_stride;
    t.xb = scratch + lay.xb_off;
    t.Wsc = static_cast<const __half*>(a.Wsc);
    t.nkb = a.K / 16;
    const uintptr_t sc = reinterpret_cast<uintptr_t>(a.Wsc) | (uintptr_t)(2 * t.nkb);
    t.sc_gran = sc % 16 == 0 ? 16 : sc % 8 == 0 ? 8 : 4;
    t.partial = reinterpret_cast<float*>(scratch + lay.part_off);
    t.tickets = reinterpret_cast<unsigned int*>(scratch);
    t.status = a.status;
    t.N = a.N; t.M = M; t.nchunks = lay.nchunks; t.tiles = lay.tiles; t.csize = lay.csize;
    switch (lay.NE) {
        case 32: return launch_n<32>(map_w, t, lay.grid, st);
        case 48: return launch_n<48>(map_w, t, lay.grid, st);
        default: return launch_n<64>(map_w, t, lay.grid, st);
    }
}

}  // namespace wide
}  // namespace bw
