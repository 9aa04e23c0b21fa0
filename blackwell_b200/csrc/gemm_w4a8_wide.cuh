// INT4-weight x INT8-activation block-16 GEMM for batches of up to 64 sequences on the 5th-generation tensor cores
// (tcgen05.mma kind::f16, A and accumulators in tensor memory).  Device side.
//
//   y[m][n] = sum_kb (sum_{k in kb} W[n,k] * w_sc[n,kb] * xq[m,k]) * x_sc[m,kb]
//
// The weight scale goes into the MMA's A operand without rounding: a binary16 scale s (11 significant bits) is the sum of
// two bf16 numbers of five significant bits each, s = sh + sl (sh = s rounded to five bits, |s - sh| <= 32 units of s's last
// place), a nibble q in [-8, 7] has three, so q * sh and q * sl are bf16 numbers exactly.  An int8 activation is a bf16 number
// exactly.  One k-block is the K = 16 of one MMA: two MMAs (q sh, then += q sl) leave w_sc * dot16 in the accumulator.  All
// products of an MMA are integer multiples of one unit with sums below 2^19, and w_sc * dot16 has 25 bits at the most
// (11 + 14), so what the accumulator holds is exact but for its last bit in extreme blocks.  What remains per (row, sequence,
// block) is ONE fp32 FMA with the activation scale.
//
// Against the int8 form (gemm_w4a8_tc.cuh: exact int32 dots, two FMAs per value in the epilogue) this moves half of the scaling
// to the operand, where it is done once per weight and not once per weight and sequence.
//
// A tile is 256 weight rows: two MMA row groups that share the activations and their scales.  Roles in a CTA of 20 warps:
//   warp 0       producer: TMA boxes of 256 rows x 128 bytes of nibbles, bulk copies of activations and their scales
//   warp 1       MMA issuer
//   warps 4-19   workers, all alike: a worker unpacks one k-block of one row per thread and pair of blocks (nibbles -> q sh, q sl
//                by packed bf16 FMAs, stored straight to tensor memory: through shared memory the A operand alone would take a
//                third of its bandwidth), then scales the accumulators of the pair before, two rows x a quarter of the sequences
//                per thread.  Unpack and scaling in the same warps: four independent warps per scheduler hide each other's
//                tensor-memory and barrier latencies (eight unpack and eight epilogue warps measured 594 us where this takes
//                530: 151,643 x 4096, 64 sequences).
// A pair is the blocks (p, p + 8) of a chunk, so that a thread's eight blocks are consecutive: its scales are 16 bytes, its
// nibbles come two blocks per 16-byte load.  Scalar FMAs, not packed ones: the packed form goes to half of the FMA pipe, which
// the bf16 FMAs of the unpack already fill (708 against 517 us, same case).
// What bounds it (75,776 x 4096, 32 / 48 / 64 sequences): issue slots 63 / 68 / 68 % busy with five warps per scheduler, then the
// latency chain of a worker's step; HBM 15 / 13 / 10 %, tensor pipe 11 / 14 / 14 % active.  Spilled by ptxas at 32 / 48 columns:
// 12 / 56 bytes stored, 56 loaded; none at 64.
// All waits are bounded; a wait that gives up raises an abort flag.
#pragma once
#include <cuda_bf16.h>

#include "gemm_w4a8_tc.cuh"

namespace bw {
namespace wide {

using tc::bulk_g2s_plain;
using tc::elect_one;
using tc::smem_desc;
using tc::tc_commit;
using tc::tc_fence_after;
using tc::tc_fence_before;
using tc::tma_load_2d;
using tc::tmem_alloc;
using tc::tmem_dealloc;
using tc::tmem_relinquish;
using tc::tmem_wait_ld;

constexpr int kKc = 256;          // k per chunk = 16 k-blocks
constexpr int kBlocksPerChunk = 16;
constexpr int kPairs = 8;         // block pairs (p, p + 8) of a chunk
constexpr int kRows = 256;        // weight rows per tile: two MMA row groups of 128
constexpr int kWBytes = kRows * (kKc / 2);           // nibbles of a tile's chunk: 128 bytes a row, 128-byte swizzle
constexpr int kWorkers = 16;                         // worker warps
constexpr int kThreads = 128 + kWorkers * 32;        // warp 0 producer, warp 1 MMA issuer, two idle warps, workers
// Registers by role: the launch gives every thread 96; the first four warps keep 32, the workers take 112.
constexpr int kRegsFew = 32, kRegsWork = 112;
static_assert(4 * kRegsFew + kWorkers * kRegsWork <= (4 + kWorkers) * 96, "register shares above the launch's total wait forever");

struct WideArgs {
    float* y;                 // [M][y_stride]
    const float* residual;    // optional, same layout as y
    long y_stride;
    const unsigned char* xb;  // activations in chunk layout (see prep kernel)
    const __half* Wsc;        // [N][nkb] weight scales
    int nkb;                  // K / 16
    int sc_gran;              // largest of 16, 8, 4 bytes that divides scale base and row pitch
    float* partial;           // [CTA][2][sequences][256] partial tiles of K ranges that begin or end inside a tile
    unsigned int* tickets;    // [tiles], zero at the start (see the prep kernel)
    int* status;              // device status word
    int N, M;
    int nchunks;              // ceil(K / 256)
    int tiles;                // ceil(N / 256)
    int csize;                // > 1: the CTAs of a cluster share one tile's K range; 1: chunks of all tiles dealt out
                              // evenly; 0: whole tiles dealt out
};

// bytes of one activation chunk: [block 0..15][k half][NP sequences x 16 B bf16], then 16 x NP fp32 block scales
__host__ __device__ constexpr int xop_bytes(int NP) { return kBlocksPerChunk * NP * 32; }
__host__ __device__ constexpr int xchunk_bytes(int NP) { return xop_bytes(NP) + kBlocksPerChunk * NP * 4; }

// Bounded wait of a converged warp whose common case is a probe and a branch; false after about a second.
__device__ __forceinline__ bool mbar_wait_quick(uint32_t bar, uint32_t parity) {
    uint32_t tries;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmov.u32 %0, 0;\n"
        "W%=:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra D%=;\n\t"
        "add.u32 %0, %0, 1;\n\tsetp.lt.u32 p, %0, 64;\n\t@p bra W%=;\nD%=:\n\t}"
        : "=&r"(tries) : "r"(bar), "r"(parity) : "memory");
    return tries < 64 || mbar_wait(bar, parity);
}
// D = A * B (accumulate == 0) or D += A * B; A (bf16, row = lane, two k per column) in tensor memory, B in shared memory.
__device__ __forceinline__ void tc_mma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// C accumulator columns of this warp's 32 lanes.
template <int C>
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t* v);
template <>
__device__ __forceinline__ void tmem_ld<4>(uint32_t addr, uint32_t* v) { tc::tmem_ld4(addr, *reinterpret_cast<uint32_t(*)[4]>(v)); }
template <>
__device__ __forceinline__ void tmem_ld<8>(uint32_t addr, uint32_t* v) { tc::tmem_ld8(addr, *reinterpret_cast<uint32_t(*)[8]>(v)); }
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t addr, uint32_t* v) { tc::tmem_ld16(addr, *reinterpret_cast<uint32_t(*)[16]>(v)); }
template <>
__device__ __forceinline__ void tmem_ld<12>(uint32_t addr, uint32_t* v) {
    tmem_ld<8>(addr, v);
    tmem_ld<4>(addr + 8, v + 8);
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <int R>
__device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

// Instruction descriptor: D = fp32, A = B = bf16, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}

// ------------------------------------------------------------------ weight unpack
// What the unpack of one k-block needs of its scale s = sh + sl, each as a bf16 number in both halves of a word.
struct ScaleParts {
    uint32_t sh8, sh24, sl8, sl24;   // sh / 8, -24 sh, sl / 8, -24 sl: exact (24 has two significant bits)
};
// In the fp32 form of a binary16 number mantissa bits 12..0 are zero: bits 22..19 stay in sh (rounded), what is left is a
// multiple of bit 13 of magnitude at most 2^5 such units.  Both parts and their multiples end above bit 16 of the word.
__device__ __forceinline__ ScaleParts split_scale(float s) {
    const float h = __uint_as_float((__float_as_uint(s) + 0x00040000u) & 0xFFF80000u), l = s - h;
    uint32_t sh, sl;
    asm("prmt.b32 %0, %1, 0, 0x3232;" : "=r"(sh) : "r"(__float_as_uint(h)));
    asm("prmt.b32 %0, %1, 0, 0x3232;" : "=r"(sl) : "r"(__float_as_uint(l)));
    auto mul = [](uint32_t v, uint32_t by) {
        uint32_t r;
        asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(by));
        return r;
    };
    return ScaleParts{mul(sh, 0x3E003E00u), mul(sh, 0xC1C0C1C0u), mul(sl, 0x3E003E00u), mul(sl, 0xC1C0C1C0u)};
}
__device__ __forceinline__ uint32_t bfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// Four words of A: nibbles (i, i + 4) of w, i = 0..3, as bf16 pairs q sh (hi) and q sl (lo).  A nibble n at bits 6..3 under
// the exponent of 128 is 8 (16 + n) in bf16, and 8 (16 + n) * s / 8 - 24 s = (n - 8) s: one FMA, exact.
__device__ __forceinline__ void unpack_word(uint32_t w, const ScaleParts& s, uint32_t* hi, uint32_t* lo) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t n;
        const uint32_t sft = i == 0 ? w << 3 : w >> (4 * i - 3);
        asm("lop3.b32 %0, %1, 0x00780078, 0x43004300, 0xEA;" : "=r"(n) : "r"(sft));   // (a & b) | c
        hi[i] = bfma2(n, s.sh8, s.sh24);
        lo[i] = bfma2(n, s.sl8, s.sl24);
    }
}

}  // namespace wide
}  // namespace bw
