// INT4-weight x INT8-activation block-16 GEMM for batches of up to 64 sequences on the 5th-generation tensor cores
// (tcgen05.mma kind::f16, A and accumulators in tensor memory).  Device side.
//
//   y[m][n] = sum_kb (sum_{k in kb} W[n,k] * w_sc[n,kb] * xq[m,k]) * x_sc[m,kb]
//
// Both block scales go into the MMA's operands, as sums of bf16 numbers, so that an accumulator runs over a whole chunk of 256 k
// and one fp32 FMA per (row, sequence, chunk) is left of the scaling.
//   Weights: a binary16 scale s (11 significant bits) is sh + sl, two numbers of five significant bits each (sh = s rounded to
//   five bits, |s - sh| <= 32 units of s's last place); a nibble q in [-8, 7] has three, so q sh and q sl are bf16 numbers: exact.
//   Activations: x = xq x_sc is cut into x1 + x2 + x3 in units of a power of two u per (sequence, chunk), u the place of the eighth
//   bit of the chunk's largest |x|: x1 = x rounded to whole units (|x1| <= 256), x2 the rest as a bf16 number, x3 what is still
//   left as another.  Of an element 2^-19 u is lost at most, 2^-26 of the chunk's largest |x|, and never more than 2^-18 of itself.
// Products: q sh x1 | q sh x2, q sh x3, q sl x1, q sl x2, and q sl x3 where the chains of sums are short (WideArgs::six).  Without
// it up to 2^-15 u |w| more would be lost; x1 then has finer places where its block is far below the chunk's largest (kFine), so that it
// is 2^-20 of the block's mean |x| and 2^-23 of the element at most.
// So this is fixed point over 256 k of a sequence, not 24 bits of every block.  On what the path meets it loses less than the sums of
// the other forms do (beside kFine and preferred()).  Where one block of a chunk is f times the others and meets zero weights, the
// others' bits are what counts: 4,096 x 4096, 2-norm against 64 bits, five products / six (12 sequences) / every block scaled by itself:
// f = 64 1.2e-7 / 5.5e-7 / 1.7e-7, f = 1,024 1.2e-7 / 2.6e-6 / 1.7e-7; one element of every block 64 times the others 5e-7 / 5e-7 / 1.7e-7
// (quantizing to int8 loses 5e-3).  Finer places help there and cost where blocks of very different sizes all count: the first sum is
// then no longer exact (below).  bw_set_tuning key 24 < 0 chooses the forms that scale every block by itself.
// The first product has an accumulator of its own: x1 (in whole units) and, where the scales of a row's chunk share an exponent, q sh are whole
// numbers of one unit below 2^8 in magnitude, so its sum over 256 k stays below 2^24 units and is exact -- the tensor core cuts off
// what an addition shifts out, which in one accumulator would cost up to a unit of the last place at every step, always towards
// zero.  The others are 2^-5 to 2^-22 of the first; what is cut off there does not count.  The sum of both times u joins the fp32
// result.  Errors against 64 bits: beside preferred() in the .cu file.
//
// Against the int8 form (gemm_w4a8_tc.cuh: exact int32 dots, two FMAs per row, sequence and block in the epilogue) and an earlier
// bf16 form (weight scale in A, activation scale by one FMA per row, sequence and block) this trades CUDA-core work and
// tensor-memory reads for 2.5 to 3 times the MMAs; the tensor pipe had been 11 to 14 % busy.  151,643 x 4096 at 32 / 48 / 64 sequences,
// prep included: int8 form 329 / 480 / 482 us, earlier bf16 form 327 / 383 / 526, this one 170 / 225 / 280.
//
// A tile is 256 weight rows: two MMA row groups that share the activations.  Roles in a CTA of 20 warps:
//   warps 0, 1   MMA issuers, one for each row group: between two A slots an issuer needs some 150 cycles, which the other's MMAs
//                fill (65,536 x 4096 at 32 / 64 sequences: 101 / 139 us with one issuer for both, 94 / 131 with two)
//   warp 2       activations: bulk copies of half a chunk's operand
//   warp 3       nibbles: TMA boxes of 256 rows x 128 bytes; weight scales: 32 bytes of a row and chunk by cp.async
//   warps 4-19   workers: a worker thread unpacks k-blocks of one row (nibbles -> q sh, q sl by packed bf16 FMAs, stored straight to
//                tensor memory: through shared memory the A operand alone would take its whole bandwidth) and, once per chunk,
//                adds up the accumulators of that row x half of the sequences.
// Eight workers serve each row group, so that one group's waiting falls into the other's unpacking and MMAs.  A thread's eight blocks
// of a chunk are consecutive, four to each half: half h of a chunk is the blocks whose index has bit 2 equal to h, and the
// activations are laid out the same way.
// What bounds it (65,536 x 4096): at 64 sequences the tensor pipe, 81 % busy at the 1.55 GHz that the power limit leaves (five products
// of 64 columns take 161 cycles per k-block and group; 48 / 32 / 16 columns 121 / 83 / 53, measured); at 32 and 16 the workers' issue
// slots (63 % used at 32; bf16 FMAs, shifts and logic operations take two cycles of their pipes each): with one MMA in five the same
// kernel takes 74 us of 80 there, with two thirds of the activation traffic left out 79.
// All waits are bounded; a wait that gives up raises an abort flag.
#pragma once
#include <cuda_bf16.h>

#include "gemm_w4a8_tc.cuh"

namespace bw {
namespace wide {

using tc::bulk_g2s_plain;
using tc::elect_one;
using tc::idesc_bf16;
using tc::smem_desc;
using tc::tc_commit;
using tc::tc_fence_after;
using tc::tc_fence_before;
using tc::tc_mma_bf16_ta;
using tc::tma_load_2d;
using tc::tmem_alloc;
using tc::tmem_dealloc;
using tc::tmem_relinquish;
using tc::tmem_st16;
using tc::tmem_wait_ld;
using tc::tmem_wait_st;

constexpr int kKc = 256;          // k per chunk = 16 k-blocks
constexpr int kBlocksPerChunk = 16;
constexpr int kRows = 256;        // weight rows per tile: two MMA row groups of 128
constexpr int kWBytes = kRows * (kKc / 2);           // nibbles of a tile's chunk: 128 bytes a row, 128-byte swizzle
constexpr int kWorkers = 16;                         // worker warps
constexpr int kStageBytes = kWBytes + kRows * 32;    // and the scales: [blocks 0-7, 8-15][row][16 bytes]
constexpr int kThreads = 128 + kWorkers * 32;        // two MMA issuers, activations, weights, workers
constexpr int kScaleSlots = 4;    // chunks whose units u are in shared memory
// Five products: x1 has places of kFine times the power of two below its block's mean |x|, where that is less than u.  Error against 64 bits
// (2-norm, 1e-8; 5,632 x 2048, whole units / this / 2^-6, 2^-7 in a numpy restatement / every block scaled by itself): silu(g) u of normal g and
// u 23 / 10 / 8, 8 / 13, one channel in 200 30 times the others 46 / 9 / 8, 8 / 13, block sizes spread evenly over 2^12 with such weights 21 / 27 /
// 28, 30 / 13.  With six products the error is 5 to 9 on all but the last (11) without it, and the finer places would cost the last.
constexpr float kFine = 0.03125f;
constexpr int kSlots = 2;         // A slots of a row group, four k-blocks each (eight in one slot, at 32 sequences: 86 against 78 us)
// Registers by role: the launch gives every thread 96; the first four warps keep 32, the workers take 112.
constexpr int kRegsFew = 32, kRegsWork = 112;
static_assert(4 * kRegsFew + kWorkers * kRegsWork <= (4 + kWorkers) * 96, "register shares above the launch's total wait forever");

struct WideArgs {
    float* y;                 // [M][y_stride]
    const float* residual;    // optional, same layout as y
    long y_stride;
    const unsigned char* xb;  // activations in chunk layout (see the prep kernel)
    const __half* Wsc;        // [N][nkb] weight scales
    int nkb;                  // K / 16
    int sc_gran;              // largest of 16, 8, 4 bytes that divides scale base and row pitch
    float* partial;           // [CTA][2][sequences][256] partial tiles of K ranges that begin or end inside a tile
    unsigned int* tickets;    // [tiles][worker warps], zero at the start (see the prep kernel)
    int* status;              // device status word
    int N, M;
    int nchunks;              // ceil(K / 256)
    int tiles;                // ceil(N / 256)
    int csize;                // > 1: the CTAs of a cluster share one tile's K range; 1: chunks of all tiles dealt out
                              // evenly; 0: whole tiles dealt out
    int six;                  // all six products, not five
};

// bytes of half an activation chunk: [block 0..7][k half][x1, x2, x3][NP sequences x 16 B bf16]; of a chunk: two halves, then NP units u
__host__ __device__ constexpr int xhalf_bytes(int NP) { return 8 * 2 * 3 * NP * 16; }
__host__ __device__ constexpr int xchunk_bytes(int NP) { return 2 * xhalf_bytes(NP) + NP * 4; }

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
// Asynchronous copy of B bytes global -> shared; src_bytes 0 writes zeros.
template <int B>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, uint32_t src_bytes) {
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(src_bytes), "n"(B) : "memory");
}

template <int R>
__device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

// ------------------------------------------------------------------ weight unpack
// What the unpack of one k-block needs of its scale s = sh + sl, each as a bf16 number in both halves of a word.
struct ScaleParts {
    uint32_t sh, sh192, sl, sl192;   // sh, -192 sh, sl, -192 sl: exact (192 has two significant bits)
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
    return ScaleParts{sh, mul(sh, 0xC340C340u), sl, mul(sl, 0xC340C340u)};
}
__device__ __forceinline__ uint32_t bfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// Four words of A: nibbles (i, i + 4) of w, i = 0..3, as bf16 pairs 8 q sh (hi) and 8 q sl (lo).  A nibble n at bits 6..3 under
// the exponent of 128 is 128 + 8 n in bf16, and (128 + 8 n) s - 192 s = 8 (n - 8) s: one FMA, exact.  (The eight is in u.)
__device__ __forceinline__ void unpack_word(uint32_t w, const ScaleParts& s, uint32_t* hi, uint32_t* lo) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t n;
        const uint32_t sft = i == 0 ? w << 3 : w >> (4 * i - 3);
        asm("lop3.b32 %0, %1, 0x00780078, 0x43004300, 0xEA;" : "=r"(n) : "r"(sft));   // (a & b) | c
        hi[i] = bfma2(n, s.sh, s.sh192);
        lo[i] = bfma2(n, s.sl, s.sl192);
    }
}

}  // namespace wide
}  // namespace bw
