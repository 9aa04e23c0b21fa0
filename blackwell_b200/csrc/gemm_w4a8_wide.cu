// Launcher and kernels of the bf16 tcgen05 form of the W4A8 product.  See gemm_w4a8_wide.cuh for the arithmetic.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
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
// it comes) and stores x = xq x_sc as three bf16 parts in units of u (gemm_w4a8_wide.cuh; `six`: for six products) in the layout of the MMA's B operand:
//   chunk c: [half 0..1][block 0..7][k half][x1, x2, x3][NP rows x 16 B: eight bf16]   then   [NP] units u
// Half h holds the chunk's blocks whose index has bit 2 equal to h, in order.  The eight elements of a k half are in the order in
// which the unpack takes the nibbles of a word: 0 4 1 5 2 6 3 7.  k-blocks >= K/16 of the last chunk are zero (their weights
// multiply as zero too); rows >= M are left as they are: an accumulator column is one sequence.  An infinite or NaN scale makes its
// sequence's results non-finite.  Zeroes the arrival counters of equal shares (`ncounters`, or 0).  Grid (ceil(chunks / 8), M), 256
// threads of eight elements, a warp per chunk; starts early under programmatic dependent launch.
// ----------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) prep_x_kernel(unsigned char* xb, const GemvArgs a, int NP, int nchunks, int six,
                                                     unsigned int* counters, int ncounters) {
    __shared__ float part[8];
    pdl_trigger();
    pdl_wait();   // the activations come from the kernel before
    zero_counters(counters, ncounters);
    const int m = blockIdx.y, t = threadIdx.x, lane = t & 31;
    const float rstd = a.xkind == kXFloatNorm ? row_rstd(a, m, t, part) : 1.f;
    const int e0 = (blockIdx.x * 256 + t) * 8;
    const bool valid = e0 < a.K;   // K % 16 == 0: the two threads of a block are valid or not together
    uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float sc = 0.f;
    if (a.xkind == kXInt8) {
        if (valid) {
            const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const int8_t*>(a.x) + (size_t)m * a.K + e0);
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] = (i < 4 ? u.x : u.y) >> (8 * (i & 3));
            sc = a.xsc[(size_t)m * (a.K / 16) + (e0 >> 4)];
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
    // u = 2^e with e the exponent of the chunk's largest |x| / 128 (so |x| < 256 u), within what has a normal reciprocal or 2^-127
    float f[8], big = 0.f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        f[i] = (float)(int8_t)q[i];
        big = fmaxf(big, fabsf(f[i]));
        sum += fabsf(f[i]);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);   // of the block
    if (big == 0.f && fabsf(sc) < INFINITY) sc = 0.f;   // (0 times a scale far above the chunk's)
    float top = big * (fabsf(sc) * 0.0078125f);
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, i));
    const uint32_t eb = min(max(__float_as_uint(top) & 0x7F800000u, 0x00800000u), 0x7F000000u);
    const float ru = __uint_as_float(eb == 0x7F000000u ? 0x00400000u : 0x7F000000u - eb), rs = sc * ru;   // 1 / u; x_sc / u: exact
    // x1's places (see kFine) times 1.5 * 2^23: adding and taking that away rounds to them
    const float mean = __uint_as_float(__float_as_uint(sum * (fabsf(sc) * 0.0625f)) & 0x7F800000u) * ru;
    const float places = (six ? 1.f : fminf(mean * kFine, 1.f)) * kMagicFloat;
    const int c = e0 / kKc, b = (e0 >> 4) % kBlocksPerChunk;
    if (c >= nchunks) return;
    uint32_t o[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float p[3][2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float v = f[i + 4 * j];
            p[0][j] = __bfloat162float(__float2bfloat16_rn(__fadd_rn(__fmul_rn(v, rs), places) - places));
            const float r = fmaf(v, rs, -p[0][j]);   // exact: the product's upper bits are gone
            p[1][j] = __bfloat162float(__float2bfloat16_rn(r));
            p[2][j] = r - p[1][j];
        }
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(p[n][0], p[n][1]);
            o[n][i] = *reinterpret_cast<const uint32_t*>(&h);
        }
    }
    unsigned char* chunk = xb + (size_t)c * xchunk_bytes(NP);
    const int half = (b >> 2) & 1, at = (b >> 3) * 4 + (b & 3);
    unsigned char* row = chunk + half * xhalf_bytes(NP) + ((size_t)(2 * at + (t & 1)) * 3 * NP + m) * 16;
#pragma unroll
    for (int n = 0; n < 3; ++n) *reinterpret_cast<uint4*>(row + n * NP * 16) = make_uint4(o[n][0], o[n][1], o[n][2], o[n][3]);
    if (lane == 0) reinterpret_cast<float*>(chunk + 2 * xhalf_bytes(NP))[m] = __uint_as_float(eb) * 0.125f;   // the operand A is eight times the weights
}

// ----------------------------------------------------------------------------------------------------------
// Shape of an instantiation: NE sequences = columns of the MMA.
// ----------------------------------------------------------------------------------------------------------
template <int NE>
struct WideShape {
    static constexpr int NP = NE;                        // columns of an MMA
    static constexpr int CW = NE / 2;                    // sequences per worker thread
    static constexpr int LD = NE == 32 ? 16 : 8;         // of them read from tensor memory together
    static constexpr bool kTwice = NE <= 32;             // two sets of accumulators
    static constexpr int kDCols = 4 * NP;                // tensor memory: sets of [row group][sum of q sh x1, sum of the rest][NP], then
    static constexpr int kACol = (kTwice ? 2 : 1) * kDCols;   // A: [row group][slot][half of its workers][two blocks][q sh, q sl][8]
    // stages of weights (of a chunk) and of activations (of half a chunk): with few sequences the weights in flight matter, with many
    // the tensor pipe takes its time over a chunk
    static constexpr int SW = NE == 16 ? 4 : NE == 32 ? 3 : 2;
    static constexpr int SX = NE == 16 ? 5 : NE == 64 ? 3 : 4;
    static constexpr int kSmem = 1024 + 2048 + SW * kStageBytes + SX * xhalf_bytes(NP);   // alignment; barriers, flags, units; the rings
    static_assert(kACol + 2 * kSlots * 64 <= 512 && kSmem <= kMaxDynSmem, "shape");
    static_assert(NE * kRows * 4 <= SW * kStageBytes, "the tile for the cluster reduction takes the place of the weights");
    static_assert(kScaleSlots * NP * 4 <= 1024 && SX <= 6, "units");   // see the activation producer
    // barriers
    static constexpr int kFullW = 0;             // + stage: nibbles and scales landed
    static constexpr int kEmptyW = kFullW + SW;  // + stage: unpacked
    static constexpr int kFullX = kEmptyW + SW;  // + stage: activations landed
    static constexpr int kEmptyX = kFullX + SX;  // + stage: multiplied
    static constexpr int kFullU = kEmptyX + SX;  // + slot: units of a chunk landed
    static constexpr int kFullA = kFullU + kScaleSlots;   // + A slot: stored by the row group's workers, who have read what its unit will overwrite
    static constexpr int kDone = kFullA + 2 * kSlots;     // + A slot: its MMAs have completed
    static constexpr int kTeam = kDone + 2 * kSlots;      // all workers have left the ring, at the end of a cluster's tile
    static constexpr int kDrain = kTeam + 1;
    static constexpr int kNumBars = kDrain + 2;
    static_assert(kNumBars * 8 <= 512, "barriers");
};

// Place in a ring.
template <int N>
struct Ring {
    uint32_t at = 0, phase = 0;
    __device__ __forceinline__ void step() {
        if (++at == N) { at = 0; phase ^= 1; }
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

// The scales of chunk c of a tile's rows, B bytes a copy, by one warp: neighbouring lanes take neighbouring pieces of a row.  One
// addition and one copy per 32 pieces: a loop with a product per row was the slowest part of the kernel (44 against 36 us, 16 tiles
// of 16 chunks on a CTA each, 32 sequences).
template <int B>
__device__ __forceinline__ void copy_scales(const WideArgs& a, uint32_t to, int tile, int c, int lane) {
    constexpr int kStep = B / 2, kPer = kBlocksPerChunk / kStep, kAtOnce = 32 / kPer;   // blocks a piece, pieces a row, rows at once
    const int piece = lane % kPer, r0 = lane / kPer, at = c * kBlocksPerChunk + piece * kStep, row0 = tile * kRows + r0;
    const uint32_t dst = to + (piece * kStep >> 3) * kRows * 16 + (piece * kStep & 7) * 2 + r0 * 16, src = at < a.nkb ? B : 0;
    const char* p = reinterpret_cast<const char*>(a.Wsc + min(at, a.nkb - kStep));
    const size_t pitch = (size_t)a.nkb * 2;
    if (tile * kRows + kRows <= a.N) {
        p += row0 * pitch;
#pragma unroll
        for (int i = 0; i < kRows / kAtOnce; ++i, p += kAtOnce * pitch) cp_async<B>(dst + i * kAtOnce * 16, p, src);
    } else {   // the last tile: rows past the end take the last one's scales, nothing reads what comes of them
#pragma unroll 1
        for (int i = 0; i < kRows / kAtOnce; ++i) cp_async<B>(dst + i * kAtOnce * 16, p + min(row0 + i * kAtOnce, a.N - 1) * pitch, src);
    }
}

template <int NE>
__global__ void __launch_bounds__(kThreads, 1)
gemm_w4a8_wide_kernel(const __grid_constant__ CUtensorMap map_w, const WideArgs a) {
    using Sh = WideShape<NE>;
    constexpr int NP = Sh::NP, CW = Sh::CW, SW = Sh::SW, SX = Sh::SX;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    float* units = reinterpret_cast<float*>(smem + 1024);   // [slot][NP]
    unsigned char* ring = smem + 2048;                      // nibbles and scales
    unsigned char* xring = ring + SW * kStageBytes;         // activations
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(smem + 512);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 516);
    const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;   // the warp index is uniform
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8 * i; };
    const uint32_t flag = smem_u32(const_cast<int*>(abort_flag));
    auto wait = [&](int i, uint32_t parity) { mbar_wait_or_abort(bar(i), parity, flag); };   // by a converged warp or by one lane
    if (t == 0) {
        for (int i = 0; i < SW; ++i) {
            mbar_init(bar(Sh::kFullW + i), 1 + 32);
            mbar_init(bar(Sh::kEmptyW + i), kWorkers);
        }
        for (int i = 0; i < SX; ++i) {
            mbar_init(bar(Sh::kFullX + i), 1);
            mbar_init(bar(Sh::kEmptyX + i), 2);
        }
        for (int i = 0; i < kScaleSlots; ++i) mbar_init(bar(Sh::kFullU + i), 1);
        for (int i = 0; i < 2 * kSlots; ++i) {
            mbar_init(bar(Sh::kFullA + i), kWorkers / 2);
            mbar_init(bar(Sh::kDone + i), 1);
        }
        mbar_init(bar(Sh::kTeam), kWorkers);
        for (int i = 0; i < 2; ++i) mbar_init(bar(Sh::kDrain + i), 1);
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
    if (warp == 3) {
        // ------------------------------------------------------------------------------------ weights
        // Nibbles by TMA, scales (32 bytes of a row and chunk, zeros past the end of the row) in the largest copies that the row pitch
        // allows.  Loaded into registers by the workers a chunk ahead, the scales held up every wait for shared memory behind them (12 %
        // of the time at 32 sequences, 19 % at 64).
        bool waited = false;
        int n = 0;
        for (; n < total; ++n) {
            const int w = w0 + n, tile = w / a.nchunks, c = w - tile * a.nchunks, s = n % SW;
            if (n >= SW) {
                if (!waited) pdl_wait();   // the weights do not depend on the kernel before; see the workers' first wait
                waited = true;
                wait(Sh::kEmptyW + s, ((n / SW) & 1) ^ 1);
                if (*abort_flag) break;
            }
            const uint32_t stage = smem_u32(ring + s * kStageBytes);
            if (lane == 0) {
                mbar_expect_tx(bar(Sh::kFullW + s), kWBytes);
                tma_load_2d(stage, &map_w, c * (kKc / 2), tile * kRows, bar(Sh::kFullW + s));
            }
            if (a.sc_gran == 16) copy_scales<16>(a, stage + kWBytes, tile, c, lane);
            else if (a.sc_gran == 8) copy_scales<8>(a, stage + kWBytes, tile, c, lane);
            else copy_scales<4>(a, stage + kWBytes, tile, c, lane);
            tc::cp_async_arrive(bar(Sh::kFullW + s));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (*abort_flag && lane == 0)   // gave up: the copies in flight end before the block does
            for (int i = max(0, n - SW); i < n; ++i) mbar_wait(bar(Sh::kFullW + i % SW), (i / SW) & 1);
    } else if (warp == 2) {
        if (lane == 0) {
            // -------------------------------------------------------------------------------- activations
            // The units of chunk n take the slot of chunk n - 4.  They follow the chunk's second half, which is let in by the MMAs of half
            // 2 n + 1 - SX: of chunk n - 3 or later, and the workers read the sums (and units) of chunk n - 4 before they store the operands of
            // that one's second half.
            pdl_wait();
            int h = 0;
            for (; h < 2 * total; ++h) {
                const int s = h % SX, n = h >> 1;
                wait(Sh::kEmptyX + s, ((h / SX) & 1) ^ 1);   // (at once the first time round)
                if (*abort_flag) break;
                const unsigned char* chunk = a.xb + (size_t)((w0 + n) % a.nchunks) * xchunk_bytes(NP);
                mbar_expect_tx(bar(Sh::kFullX + s), xhalf_bytes(NP));
                bulk_g2s_plain(smem_u32(xring + s * xhalf_bytes(NP)), chunk + (h & 1) * xhalf_bytes(NP), xhalf_bytes(NP), bar(Sh::kFullX + s));
                if (h & 1) {
                    const int u = n % kScaleSlots;
                    mbar_expect_tx(bar(Sh::kFullU + u), NP * 4);
                    bulk_g2s_plain(smem_u32(units + u * NP), chunk + 2 * xhalf_bytes(NP), NP * 4, bar(Sh::kFullU + u));
                }
            }
            if (*abort_flag) {   // gave up
                for (int i = max(0, h - SX); i < h; ++i) mbar_wait(bar(Sh::kFullX + i % SX), (i / SX) & 1);
                for (int n = max(0, h / 2 - kScaleSlots); n < h / 2; ++n) mbar_wait(bar(Sh::kFullU + n % kScaleSlots), (n / kScaleSlots) & 1);
            }
        }
    } else if (warp < 2) {
        // ------------------------------------------------------------------------------------ MMA issuers, one for each row group
        // The whole warp walks the loop, one elected lane issues (see elect_one).
        constexpr uint32_t idesc = idesc_bf16(NP);
        const int g = warp;
        const bool elected = elect_one(), six = NE == 16 || a.six;
        pdl_wait();        // see the workers' first wait
        Ring<SX> xs;
        for (int n = 0; n < total && !*abort_flag; ++n) {
            const uint32_t d1 = tmem + (Sh::kTwice ? (n & 1) * Sh::kDCols : 0) + g * 2 * NP, d2 = d1 + NP;
#pragma unroll 1
            for (int h = 0; h < 2; ++h, xs.step()) {
                wait(Sh::kFullX + xs.at, xs.phase);
                const uint64_t db0 = smem_desc(smem_u32(xring) + xs.at * xhalf_bytes(NP), 3 * NP * 16, 128);
#pragma unroll
                for (int z = 0; z < kSlots; ++z) {
                    const int slot = g * kSlots + z;
                    wait(Sh::kFullA + slot, h);
                    tc_fence_after();
                    if (elected) {
#pragma unroll
                        for (int b = 0; b < 4; ++b) {   // blocks 2 z, 2 z + 1 of a thread's four, of either half of the workers
                            const uint32_t hi = tmem + Sh::kACol + slot * 64 + b * 16, lo = hi + 8, more = z + b > 0 ? 1u : (uint32_t)h;
                            const uint64_t x1 = db0 + (b / 2 * 4 + z * 2 + b % 2) * (2 * 3 * NP), x2 = x1 + NP, x3 = x2 + NP;   // (in 16 bytes)
                            tc_mma_bf16_ta(d2, hi, x3, idesc, more);
                            if (six) tc_mma_bf16_ta(d2, lo, x3, idesc, 1u);
                            tc_mma_bf16_ta(d2, lo, x2, idesc, 1u);
                            tc_mma_bf16_ta(d2, hi, x2, idesc, 1u);
                            tc_mma_bf16_ta(d2, lo, x1, idesc, 1u);
                            tc_mma_bf16_ta(d1, hi, x1, idesc, more);
                        }
                        tc_commit(bar(Sh::kDone + slot));
                        if (z == 1) tc_commit(bar(Sh::kEmptyX + xs.at));
                    }
                    __syncwarp();
                }
            }
        }
        if (elected) tc_commit(bar(Sh::kDrain + g));   // whatever became of the others: no MMA in flight when the tensor memory is freed
        __syncwarp();
        mbar_wait(bar(Sh::kDrain + g), 0);
    } else if (warp >= 4) {
        // ------------------------------------------------------------------------------------ workers
        regs_more<kRegsWork>();
        // Row group g; TMEM lanes 32 q ..; blocks 8 cg .. 8 cg + 7 of a chunk to unpack, sequences [cg CW, cg CW + CW) to add up.
        const int wt = t - 128, g = (warp - 4) >> 3, cg = ((warp - 4) >> 2) & 1, q = warp & 3, row = g * 128 + q * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        const uint32_t a_addr = lanes + Sh::kACol + g * 128 + cg * 32, d_addr = lanes + g * 2 * NP + cg * CW;
        float acc[CW];
#pragma unroll
        for (int j = 0; j < CW; ++j) acc[j] = 0.f;
        auto store = [&](int m, int n, float v) {
            const size_t yi = (size_t)m * a.y_stride + n;
            a.y[yi] = a.residual ? v + a.residual[yi] : v;
        };
        // The tile of chunk `wlast` is finished (or this CTA's share of it): results out, accumulators back to zero.
        auto finish = [&](int wlast) {
            const int tile = wlast / a.nchunks, first = tile * a.nchunks, begin = max(w0, first);
            const int row0 = tile * kRows + row;
            if (a.csize > 1) {   // one tile per cluster: this CTA's share goes where the ring was, once all have left it
                __syncwarp();
                mbar_arrive_by(lane == 0, bar(Sh::kTeam));
                wait(Sh::kTeam, 0);
                float* sm = reinterpret_cast<float*>(ring) + row;
#pragma unroll
                for (int j = 0; j < CW; ++j) sm[(cg * CW + j) * kRows] = acc[j];
                return;
            }
            if (*abort_flag) return;
            // (y may still be read, the partial tiles still be summed by the kernels before: past the dependency wait since chunk 0)
            if (begin == first && wlast == first + a.nchunks - 1) {
#pragma unroll
                for (int j = 0; j < CW; ++j)
                    if (cg * CW + j < a.M && row0 < a.N) store(cg * CW + j, row0, acc[j]);
            } else {
                // A share that begins or ends inside the tile: every warp leaves its part of it (32 rows x CW sequences), and the last
                // CTA's warp to arrive there adds all shares in the order of K.  (One counter per tile, with the workers in step: 34.2
                // against 32.3 us, 2,048 x 5,632 at 64 sequences in equal shares.)
                float* mine = a.partial + (size_t)(2 * blockIdx.x + (begin == w0 ? 0 : 1)) * NE * kRows + row;
#pragma unroll
                for (int j = 0; j < CW; ++j)
                    if (cg * CW + j < a.M) mine[(cg * CW + j) * kRows] = acc[j];
                __threadfence();
                __syncwarp();
                const int grid = gridDim.x, i0 = chunk_owner(a, first, grid), i1 = chunk_owner(a, first + a.nchunks - 1, grid);
                unsigned int before = 0;
                if (lane == 0) before = atomicAdd(&a.tickets[tile * kWorkers + warp - 4], 1u);
                before = __shfl_sync(0xffffffffu, before, 0);
                if (before == (unsigned)(i1 - i0)) {
                    __threadfence();
                    int b0, b1;
                    chunk_range(a, i0, grid, b0, b1);
                    const int head = b0 / a.nchunks == tile ? 0 : 1;   // which of its two shares the first CTA left here
                    const float* p0 = a.partial + (size_t)(2 * i0 + head) * NE * kRows + row;
                    const float* p1 = a.partial + (size_t)(2 * i0 + 2) * NE * kRows + row;
                    // share by share, every column's load of a share in flight together
                    auto add = [&](const float* p, bool first_share) {
#pragma unroll
                        for (int j = 0; j < CW; ++j) {
                            const float v = cg * CW + j < a.M ? __ldcg(p + (cg * CW + j) * kRows) : 0.f;
                            acc[j] = first_share ? v : acc[j] + v;
                        }
                    };
                    add(p0, true);
#pragma unroll 1
                    for (int i = 0; i < i1 - i0; ++i) add(p1 + (size_t)i * 2 * NE * kRows, false);
#pragma unroll
                    for (int j = 0; j < CW; ++j)
                        if (cg * CW + j < a.M && row0 < a.N) store(cg * CW + j, row0, acc[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < CW; ++j) acc[j] = 0.f;
        };

        // acc += the sums over chunk n, which have been waited for
        auto take = [&](int n) {
            wait(Sh::kFullU + n % kScaleSlots, (n / kScaleSlots) & 1);
            const float* u = units + n % kScaleSlots * NP + cg * CW;
            const uint32_t d = d_addr + (Sh::kTwice ? (n & 1) * Sh::kDCols : 0);
#pragma unroll
            for (int j0 = 0; j0 < CW; j0 += Sh::LD) {
                uint32_t d1[Sh::LD], d2[Sh::LD];
                tmem_ld<Sh::LD>(d + j0, d1);
                tmem_ld<Sh::LD>(d + NP + j0, d2);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < Sh::LD; ++j)
                    acc[j0 + j] = fmaf(__uint_as_float(d1[j]) + __uint_as_float(d2[j]), u[j0 + j], acc[j0 + j]);
            }
        };
        Ring<SW> ws;
        const uint32_t row_off = row * 128, sc_off = kWBytes + cg * kRows * 16 + row * 16;
        int left = a.nchunks - w0 % a.nchunks;   // chunks of the tile, from chunk n on
        for (int n = 0; n < total && !*abort_flag; ++n) {
            const unsigned char* stage = ring + ws.at * kStageBytes;
            wait(Sh::kFullW + ws.at, ws.phase);
            uint32_t sc[4];
            *reinterpret_cast<uint4*>(sc) = *reinterpret_cast<const uint4*>(stage + sc_off);
#pragma unroll
            for (int j = 0; j < 4; ++j) {   // blocks 2 j, 2 j + 1 of the thread's eight: half j / 2, slot j % 2
                const int slot = g * kSlots + j % 2;
                uint32_t v[32];
                const uint4 w4 = *reinterpret_cast<const uint4*>(stage + row_off + (((4 * cg + j) ^ (row & 7)) << 4));
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&sc[j]));
                const ScaleParts s0 = split_scale(f.x), s1 = split_scale(f.y);
                unpack_word(w4.x, s0, v, v + 8);
                unpack_word(w4.y, s0, v + 4, v + 12);
                unpack_word(w4.z, s1, v + 16, v + 24);
                unpack_word(w4.w, s1, v + 20, v + 28);
                // The limit of a wait counts this kernel's own progress, not the time until the activations' producers are done (an
                // exchange before them may wait longer for a late rank).
                if (n == 0 && j == 2) pdl_wait();
                wait(Sh::kDone + slot, j < 2);   // the slot's last MMAs (at once the first time)
                tc_fence_after();
                tmem_st16(a_addr + j % 2 * 64, v);
                tmem_st16(a_addr + j % 2 * 64 + 16, v + 16);
                if (!Sh::kTwice && j == 0 && n > 0) {   // the next MMAs take the place of the sums over the chunk before
                    wait(Sh::kDone + g * kSlots + 1, 1);
                    tc_fence_after();
                    take(n - 1);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                mbar_arrive_by(lane == 0, bar(Sh::kFullA + slot));
                if (j == 3) mbar_arrive_by(lane == 0, bar(Sh::kEmptyW + ws.at));
                if (j == (Sh::kTwice ? 1 : 0) && n > 0) {
                    if (Sh::kTwice) take(n - 1);   // (complete: its last MMAs read the slot that was waited for)
                    if (left == a.nchunks) finish(w0 + n - 1);
                }
            }
            ws.step();
            if (--left == 0) left = a.nchunks;
        }
        wait(Sh::kDone + g * kSlots + 1, 1);
        tc_fence_after();
        take(total - 1);
        finish(w0 + total - 1);
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
static int cols_of(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 48 ? 48 : 64; }

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
static bool usable(int NE) {
    return (NE == 16 ? prepare<16>() : NE == 32 ? prepare<32>() : NE == 48 ? prepare<48>() : prepare<64>()) == cudaSuccess;
}

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
    size_t xb_off, part_off, part_bytes;
};
// A cluster per tile, equal shares of all chunks or whole tiles: whichever the estimate says.  Measured (us, prep included; 21
// geometries of the matrices of three models, one CTA to 148): a chunk takes 2.0 / 2.3 / 3.1 / 4.0 at 16 / 32 / 48 / 64 sequences; a
// cluster adds 6 to 8 to its longest share; whole tiles 6; equal shares 12 and 0.5 to 0.9 for every share of a tile.  4096 x 4096,
// cluster of six / equal shares / whole tiles: 14.1 / 21.3 / 34.0 at 32 sequences; 21888 x 4096 (six, equal, whole): 56 / 36 / 36;
// 32768 x 2048: 68 / 30 / 23.  Clusters of 2 to 8 resident at once on a B200: 74, 45, 33, 26, 22, 15, 15.
static WideLayout layout_of(int M, int N, int K) {
    WideLayout l;
    l.NE = cols_of(M);
    l.nchunks = (K + kKc - 1) / kKc;
    l.tiles = (N + kRows - 1) / kRows;
    const int sms = sm_count(current_device()), force = g_split.load(), at = l.NE / 16 - 1;
    const long long all = (long long)l.tiles * l.nchunks;
    const float chunk = std::array<float, 4>{2.0f, 2.3f, 3.1f, 4.0f}[at], share = std::array<float, 4>{0.4f, 0.5f, 0.7f, 0.9f}[at];
    l.csize = 1;
    l.grid = (int)(all < sms ? all : sms);
    float best = chunk * (float)((all + l.grid - 1) / l.grid) + 12.f + share * (float)(l.grid / l.tiles + 1);
    const float whole = chunk * (float)l.nchunks * (float)((l.tiles + sms - 1) / sms) + 5.5f;
    if (whole < best) { best = whole; l.csize = 0; }
    for (int cs = 8; cs > 1; --cs)
        if (cs <= l.nchunks && l.tiles <= max_clusters(cs)) {   // the largest that is resident at once
            if (6.f + 0.6f * (float)at + chunk * (float)((l.nchunks + cs - 1) / cs) < best) l.csize = cs;
            break;
        }
    if (force > 8) l.csize = 1;
    else if (force > 1 && force <= l.nchunks) l.csize = force;
    else if (force == 1) l.csize = 0;
    // The arrival counters own a region of fixed size at the front of the block.  Matrices with more tiles than counters are dealt out by whole tiles.
    if (l.csize == 1 && (size_t)l.tiles * kWorkers * sizeof(unsigned int) > tc::kTicketBytes) l.csize = 0;
    if (l.csize == 0) l.grid = l.tiles < sms ? l.tiles : sms;
    if (l.csize > 1) l.grid = l.tiles * l.csize;
    l.part_bytes = l.csize == 1 ? (size_t)l.grid * 2 * l.NE * kRows * sizeof(float) : 0;
    l.xb_off = tc::kTicketBytes;
    l.part_off = (l.xb_off + (size_t)l.nchunks * xchunk_bytes(l.NE) + 255) & ~(size_t)255;
    return l;
}
static std::atomic<int> g_force{0};
void set_force(int v) { g_force = v; }
// Whether a call of 9 to 64 sequences comes here.  From 17 on the int8 form (gemm_w4a8_tc.cu) takes the same operands.  Measured (us, prep
// included, this form / that one at 17, 32, 48 and 64 sequences): 6144 x 4096 17 / 32, 18 / 33, 23 / 48, 28 / 48; 21888 x 4096
// 37 / 81, 38 / 81, 46 / 116, 55 / 117; 4096 x 12288 25 / 42, 28 / 43, 35 / 61, 41 / 61; 2048 x 2048 9.7 / 22, 10 / 22, 12 / 32,
// 13 / 33; 633 x 64 7.4 / 8.9, 7.4 / 8.8, 8.7 / 11, 10 / 12: this one is faster at every one of 24 shapes, by 0.16 to 0.9.
// It does not come here where its chains of chunks would be longer than that form's, unless neither splits K: a narrow matrix of very
// long rows (300 x 32768), which that form splits finer.
// Error against 64 bits (2-norm, three seeds, normal activations and scales; others in the .cuh file; five products / six / the forms that these calls took before): 633 x 64
// 8.9e-8 / 2.8e-8 / 4.0e-8, 2481 x 1024 1.0e-7 / 4.9e-8 / 8.3e-8, 3072 x 2048 1.04e-7 / 5.6e-8 / 8.8e-8, 2048 x 5632 1.09e-7 / 6.6e-8 /
// 1.30e-7, 4096 x 4096 1.08e-7 / 6.4e-8 / 1.28e-7, 21888 x 4096 1.12e-7 / 7.1e-8 / 2.0e-7, 4096 x 12288 1.17e-7 / 7.8e-8 / 2.1e-7 to
// 2.5e-7.  Hence six products up to kSixK, where five would lose more than those did; above, the sixth costs 5 to 10 % of the time.
// At 9 to 16 sequences the other form is the mma.sync kernel.  Measured (us, binary16 input, this form / that one at 9 and at 16
// sequences): 6144 x 4096 14.6 / 18.4, 15.2 / 20.6; 21888 x 4096 32.3 / 33.2, 32.8 / 35.7; 4096 x 10944 21 / 32, 22 / 32; 2048 x 5632 12 / 24,
// 12 / 24; 32768 x 2048 21 / 26, 21 / 28; 2048 x 2048 8.4 / 8.7, 8.8 / 10.2; 28683 x 704 11 / 18, 11 / 18; 5558 x 736 8.4 / 8.7, 9.0 / 8.8;
// 2481 x 1024 7.9 / 6.9, 8.4 / 7.6; 700 x 256 5.9 / 4.8, 6.1 / 5.4: the line lies at rows of 2,048 or 8 million weights.  Always six
// products (1 to 3 % of the time), error 0.32 to 0.68 of that kernel's.  Up to eight sequences that one is faster (151,643 x 4096:
// 114 against 127).
constexpr int kSixK = 3072;
bool preferred(int M, int N, int K) {
    if (M <= 8 || !usable(cols_of(M))) return false;
    if (g_force.load() != 0) return g_force.load() > 0;
    if (M <= 16) return K >= 2048 || (long long)N * K >= 8000000;
    const int sms = sm_count(current_device()), tiles = (N + 127) / 128, nchunks = (K + kKc - 1) / kKc;
    const int ks = std::max(1, std::min(sms / tiles, nchunks));
    const int theirs = std::min(2 * (((nchunks + 1) / 2 + ks - 1) / ks), nchunks);
    const WideLayout l = layout_of(M, N, K);
    const int share = (int)(((long long)l.tiles * l.nchunks + l.grid - 1) / l.grid);
    const int chain = l.csize == 0 ? nchunks : std::min(share, nchunks);
    return chain < theirs || theirs == nchunks;
}
// Whether a call can have its scratch: unless it would have to grow while the stream is captured.
bool scratch_at_hand(int M, int N, int K, cudaStream_t st) {
    const WideLayout l = layout_of(M, N, K);
    return tc::scratch_at_hand(l.part_off + l.part_bytes, st);
}
// Enough for every batch up to M.
size_t scratch_bytes(int M, int N, int K) {
    if (M <= 8 || N < 1 || K < 32) return 0;
    size_t most = 0;
    for (int m = 16; m <= cols_of(std::min(M, 64)); m += 16) {
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

    const int six = lay.NE == 16 || a.K <= kSixK;
    e = launch_pdl(prep_x_kernel, dim3((lay.nchunks + 7) / 8, M), dim3(256), 0, st, scratch + lay.xb_off, a, lay.NE, lay.nchunks, six,
                   reinterpret_cast<unsigned int*>(scratch), lay.csize == 1 ? lay.tiles * kWorkers : 0);
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
    t.N = a.N; t.M = M; t.nchunks = lay.nchunks; t.tiles = lay.tiles; t.csize = lay.csize; t.six = six;
    switch (lay.NE) {
        case 16: return launch_n<16>(map_w, t, lay.grid, st);
        case 32: return launch_n<32>(map_w, t, lay.grid, st);
        case 48: return launch_n<48>(map_w, t, lay.grid, st);
        default: return launch_n<64>(map_w, t, lay.grid, st);
    }
}

}  // namespace wide
}  // namespace bw
