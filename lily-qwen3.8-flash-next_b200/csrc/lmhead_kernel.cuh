// The quantised LM head that feeds the sampler: logits[t, n] = sum over column groups g
// of scale[n, g] * (sum over the group's 64 columns of w[n, c] * h[t, c]), w int8
// (symmetric), scale bf16 per 64 columns, h bf16, everything summed in binary32. It
// stands where the reference projects the hidden state through its quantised head
// before sampling (gemv_quant, src/kernels/quant.rs:141-175, called from
// src/qwen4exp/model.rs:2999-3006). The reference's own storage, MLX affine
// (src/weights.rs:21-36; gemv_q8, src/kernels/metal/quant.metal:124-160; 4 bits:
// :44-66), is w = scale * q + bias: the converters widen q - 128 (4 bits: q), and the
// epilogue adds (128 * scale + bias) * (sum of the group's hidden values).
//
// The weights are the only large operand, so the kernel is a stream of them through
// the tensor cores, one persistent block per SM, warps specialised:
//
//   * one thread asks the copy engine (TMA, 128-byte swizzle) for 256 rows x 128 bytes
//     of weights per stage, another for each group's slice of the hidden states (a
//     ready image, see prepare_hidden_kernel); two warps copy the rows' scales and biases,
//     eight groups of them at a time;
//   * converter warps own one tile row per thread: they widen a group's 64 weights
//     exactly to 16 bits and store them with tcgen05.st into TENSOR MEMORY, where the
//     multiplier reads its A operand (lane = row, two values per column);
//   * four warps, two per 128 rows, issue 4 tcgen05.mma each per group (M = 128, N =
//     tokens, K = 16) into an accumulator that starts from zero: products of two
//     8-bit significands are exact in binary32;
//   * epilogue warps read each group's sums back with tcgen05.ld, multiply by the
//     row's scale of that group and add into registers: the sums cannot stay in
//     tensor memory across groups because each has its own scale.
//
// The two halves of a tile are pipelines of their own (barriers, accumulators, operand
// slots): one converts while the other multiplies.
//
// Binary16 or bf16. Widening a byte to binary16 costs two or three integer
// instructions per four weights, to bf16 (whose significand does not hold 128 + 255)
// six; the integer pipe was the busiest one. A 4-bit code takes a mask: alone in 16
// bits it is a subnormal binary16, which the multiplier takes exactly. A bf16 hidden
// value times a power of two per token fits binary16 exactly if it lies within 2^32
// (4-bit codes: 2^28) of the token's largest, which hidden states do; a call in which one
// does not is multiplied in bf16, same results.
//
// Measured at 262144 x 4096, 64 tokens (before: bf16 only, one pipeline for both
// halves, N = 64 always, the affine term in a kernel of its own): see the figures at
// launch_head.
//
// Every wait on an mbarrier is bounded in time; a wait that runs out sets an
// abort word, after which no wait blocks any more: the block runs to its end
// (results are garbage, TMEM is freed) and the status word tells the host.
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "lmhead_args.cuh"

namespace lily_head {

// Warps: four that multiply, four that load (weights, hidden states, two for the scales), then
// converters, then the epilogue.
constexpr int MMA_WARPS = 4;
constexpr int WARP_LOAD_W = 4;
constexpr int WARP_LOAD_H = 5;
constexpr int WARP_LOAD_S0 = 6;
constexpr int WARP_CONV0 = 8;

constexpr uint32_t RAW_STAGE_BYTES = TILE_ROWS * 128u;  // 32 KB
constexpr uint32_t TMEM_COLS = 512;

// What depends on the (padded) number of tokens and the format. Tensor memory per half:
// ACC_BUFS times PG accumulators of N columns, A_SLOTS times PG operand tiles of 32. The
// converters are two teams of eight warps, which share the groups; one team where the
// epilogue of 64 tokens needs the registers.
template <uint32_t N, int FMT>
struct Shape {
    static constexpr uint32_t TEAMS = N == 64u && FMT != FMT_S8 ? 1u : 2u;
    static constexpr bool LEAN = TEAMS == 2u;  // converters of few registers
    static constexpr uint32_t CONV_WARPS = 8u * TEAMS;
    static constexpr uint32_t EPI_WARPS = EPILOGUE_WARPS;
    static constexpr uint32_t THREADS = 32u * (8u + CONV_WARPS + EPI_WARPS);
    // Registers a thread: at launch, then as the roles share them out (setmaxnreg; the
    // shares add up to what the block was launched with, launch_one checks that).
    static constexpr uint32_t REGS = TEAMS == 2u ? 64u : 80u;
    static constexpr uint32_t REGS_CTRL = 40u;
    static constexpr uint32_t REGS_CONV = TEAMS == 1u ? 64u : N == 64u ? 48u : 56u;
    static constexpr uint32_t REGS_EPI = TEAMS == 1u ? 136u : N == 64u ? 120u : 104u;
    static_assert(32u * (8u * REGS_CTRL + CONV_WARPS * REGS_CONV + EPI_WARPS * REGS_EPI) <= THREADS * REGS, "register shares");
    // Groups per hand-over (of operands, of accumulators): a hand-over costs each of its two
    // sides some 200 to 300 clocks, whatever goes through it.
    static constexpr uint32_t PG = N == 64u ? 1u : 2u;
    static constexpr uint32_t ACC_BUFS = 2u;                              // of PG groups
    static constexpr uint32_t A_SLOTS = N == 64u ? 4u : N == 32u ? 2u : 3u;  // of PG groups
    static constexpr uint32_t RAW_STAGES = N == 64u ? 3u : N == 32u ? 4u : 5u;
    static constexpr uint32_t H_SLOTS = 8u;                             // hidden slices in shared memory
    static constexpr uint32_t DONE_SLOTS = H_SLOTS / PG;                // ring of "has been multiplied" barriers
    static constexpr uint32_t SUM_SLOTS = 2u * H_SLOTS;                 // the slices' sums: the epilogue may be that far behind
    // Units of scales (and biases) in shared memory, so that they are there when the epilogue, which
    // is the slowest of the roles, comes to them. (Loaded by the epilogue, its warps waited some
    // 40 to 100 clocks of a group's 700 to 1200 for them: 4 bits, 32 tokens 61.5 -> 58.4 us, affine
    // bytes, 64 tokens 296 -> 293, 4 tokens 173.6 -> 171.4; sizes at launch_head.)
    static constexpr uint32_t S_SLOTS = 4u;
    static_assert(BLOCK_GROUPS * 2u == 16u, "a row's scales of a unit are one copy");
    static constexpr uint32_t S_ARRAY_BYTES = TILE_ROWS * 16u;          // 16 bytes a row
    static constexpr uint32_t S_SLOT_BYTES = (FMT != FMT_S8 ? 2u : 1u) * S_ARRAY_BYTES;
    static constexpr uint32_t H_BYTES = N * 128u;
    static constexpr uint32_t A_COL0 = ACC_BUFS * PG * N;                    // within a half's 256 columns
    static_assert(A_COL0 + A_SLOTS * PG * 32u <= TMEM_COLS / 2u, "tensor memory columns of a half");
    static_assert(ACC_BUFS <= DONE_SLOTS && A_SLOTS <= DONE_SLOTS, "the rings' phases");
    static constexpr int WARP_EPI0 = WARP_CONV0 + (int)CONV_WARPS;

    // Offsets from a 1024-byte aligned base.
    static constexpr uint32_t HID = 0;
    static constexpr uint32_t RAW = HID + H_SLOTS * H_BYTES;
    static constexpr uint32_t SUMS = RAW + RAW_STAGES * RAW_STAGE_BYTES;
    static constexpr uint32_t SCALES = SUMS + SUM_SLOTS * N * 4u;
    static constexpr uint32_t UNSCALE = SCALES + S_SLOTS * S_SLOT_BYTES;
    static constexpr uint32_t BARS = UNSCALE + N * 4u;
    static constexpr uint32_t RAW_FULL = BARS;                          // [RAW_STAGES]
    static constexpr uint32_t RAW_EMPTY = RAW_FULL + 8 * RAW_STAGES;
    static constexpr uint32_t H_FULL = RAW_EMPTY + 8 * RAW_STAGES;      // [H_SLOTS / 2]
    static constexpr uint32_t A_FULL = H_FULL + 8 * H_SLOTS;            // [2][A_SLOTS]
    // DONE[half][..]: a half of PG groups has been multiplied. One commit tells the
    // converters (slot free), the hidden loader and the epilogue (sums ready).
    static constexpr uint32_t DONE = A_FULL + 2 * 8 * A_SLOTS;          // [2][DONE_SLOTS]
    static constexpr uint32_t ACC_EMPTY = DONE + 2 * 8 * DONE_SLOTS;    // [2][ACC_BUFS]
    static constexpr uint32_t FINAL = ACC_EMPTY + 2 * 8 * ACC_BUFS;     // [MMA_WARPS] an issuing warp's last commit
    static constexpr uint32_t S_FULL = FINAL + 8 * MMA_WARPS;            // [S_SLOTS]
    static constexpr uint32_t S_EMPTY = S_FULL + 8 * S_SLOTS;            // [S_SLOTS]
    static constexpr uint32_t TMEM_ADDR = S_EMPTY + 8 * S_SLOTS;
    static constexpr uint32_t ABORT = TMEM_ADDR + 4;
    static constexpr uint32_t BYTES = ABORT + 4 + 1024;                  // room to align the base
    static_assert(BYTES <= 227u * 1024u, "shared memory of one block");
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Whether the phase with the given parity is complete; waits for a while if it is not.
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0u;
}

// Waits for the phase with the given parity to complete, for at most
// `limit_ns`; once any wait of the block has run out, none blocks any more.
// Returns true if it gave up (this wait ran out, or another had): the caller
// then leaves its loop. A phase that is complete at the first look returns
// false without reading the abort word, so the path that never waits pays
// nothing for the bound.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort_word,
                                          uint64_t limit_ns) {
    uint64_t t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        if (mbar_try(bar, parity)) {
            return false;
        }
        if ((spin & 15u) == 15u) {
            if (*abort_word) {
                return true;
            }
            const uint64_t now = global_ns();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > limit_ns) {
                *abort_word = 1u;
                return true;
            }
        }
    }
}

// The same for a whole warp, whose lanes go on together: most waits find their phase complete,
// or complete while the first look waits, and then cost a look, a vote and a branch that no
// lane takes alone. (The kernel is bound by what its warps issue, and a group has some 36 waits: 12
// instructions each with the vote behind a loop of each lane's own, 8 so; a group's 2525 became
// 2383. 64 tokens, symmetric 248 -> 243.5 us, affine bytes 288.5 -> 283, 4 bits, 32 tokens 58.4 -> 57.3;
// sizes at launch_head.)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort_word,
                                          uint64_t limit_ns) {
    if (__all_sync(0xFFFFFFFFu, mbar_try(bar, parity))) {
        return false;
    }
    return __any_sync(0xFFFFFFFFu, mbar_wait(bar, parity, abort_word, limit_ns));
}

// The same wait for the way out of a block that has given up: it does not look
// at the abort word (which is set by then), only at its own clock. Used to let
// copies and multiplies that are still in flight land before the block frees
// its tensor memory and returns.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    const uint64_t t0 = global_ns();
    for (uint32_t spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done || ((spin & 15u) == 15u && global_ns() - t0 > limit_ns)) {
            return;
        }
    }
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// One tile of a 2-D tensor map into shared memory; its bytes complete `bar`.
// x (the inner coordinate) times the element size is a multiple of 16 bytes
// at every call site.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t x,
                                            int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

// K-major operand in shared memory, 128-byte swizzle, rows 128 bytes apart,
// 8-row groups 1024 bytes apart; the start address may be advanced by 32
// bytes per K = 16 step inside the (1024-byte aligned) atom.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}

// Every warp of a warpgroup gives registers back or takes more.
template <uint32_t REGS, bool MORE>
__device__ __forceinline__ void set_registers() {
    if (MORE) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
    }
}

// A plain copy into shared memory (addresses and size multiples of 16 bytes); its bytes complete `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// A thread's copy of 16 bytes into shared memory (the 128 bytes they lie in are asked into L2).
__device__ __forceinline__ void copy_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// kind::f16: D binary32, A and B both binary16 or both bf16, both K-major, M = 128.
template <uint32_t N>
__device__ __forceinline__ uint32_t instr_desc(bool bf16) {
    return (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | ((N >> 3) << 17) | ((128u >> 4) << 24);
}

// D[tmem] (+)= A[tmem] * B[smem]^T.
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t is;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(is));
    return is != 0u;
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
          "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]),
          "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]),
          "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Two binary32 values in one 64-bit register, and the packed fused
// multiply-add on them (each half rounds as a scalar fma does).
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    uint32_t a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
    lo = __uint_as_float(a);
    hi = __uint_as_float(b);
}

// 16 bytes in registers -> 64 weights' worth of A operand words (two values each).
// Bytes: word w gives columns (4w, 4w + 2), (4w + 1, 4w + 3); nibbles: columns
// (0, 4), (1, 5), (2, 6), (3, 7) of the word's eight. The hidden states' image has its
// columns in the same order.
//
// Binary16: a byte b under the exponent of 1024 (0x6400 | b) is 1024 + b; the even
// bytes take one masking, the odd ones one byte permute, and a subtraction makes
// the value exact. Signed bytes have their top bit flipped first: (b ^ 0x80) - 128.
// bf16: with c = 0x43 in the high byte, (0x4300 | b) & 0xFF7F is 128 + (b & 127) and
// (0x4300 | b) & 0xFF80 is 128 or 256: their difference is the signed byte, and with the
// subtrahend's top bit flipped q - 128.
template <int FMT, bool BF16>
__device__ __forceinline__ void widen_bytes(uint32_t x, uint32_t &even, uint32_t &odd) {
    if (!BF16) {
        const uint32_t y = FMT == FMT_S8 ? x ^ 0x80808080u : x;
        const uint32_t e = (y & 0x00FF00FFu) | 0x64006400u, o = __byte_perm(y, 0x64646464u, 0x4341);
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(even) : "r"(e), "r"(0x64806480u));
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(odd) : "r"(o), "r"(0x64806480u));
    } else {
        constexpr uint32_t FLIP = FMT == FMT_S8 ? 0u : 0x00800080u;
        const uint32_t e = (x & 0x00FF00FFu) | 0x43004300u, o = __byte_perm(x, 0x43434343u, 0x4341);
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(even) : "r"(e & 0xFF7FFF7Fu), "r"((e ^ FLIP) & 0xFF80FF80u));
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(odd) : "r"(o & 0xFF7FFF7Fu), "r"((o ^ FLIP) & 0xFF80FF80u));
    }
}

template <bool BF16>
__device__ __forceinline__ void widen_nibbles(uint32_t x, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d) {
    if (!BF16) {
        // A code alone in 16 bits is a subnormal binary16: 2^-24 times its value, or 2^-20
        // where it is the upper half of a byte (the hidden image makes up for both).
        const uint32_t y = x >> 8;
        a = x & 0x000F000Fu;
        b = x & 0x00F000F0u;
        c = y & 0x000F000Fu;
        d = y & 0x00F000F0u;
    } else {
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(a) : "r"((x & 0x000F000Fu) | 0x43004300u), "r"(0x43004300u));
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(b) : "r"(((x >> 4) & 0x000F000Fu) | 0x43004300u), "r"(0x43004300u));
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(c) : "r"(((x >> 8) & 0x000F000Fu) | 0x43004300u), "r"(0x43004300u));
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(((x >> 12) & 0x000F000Fu) | 0x43004300u), "r"(0x43004300u));
    }
}

// Grid (padded tokens): a token's images and sums. Padded tokens are zeros.
__global__ void __launch_bounds__(256) prepare_hidden_kernel(const Prepared p, const __nv_bfloat16 *hidden, uint64_t ld,
                                                             uint32_t tokens, uint32_t groups, int nibbles, uint32_t *flags,
                                                             uint32_t n_flags) {
    __shared__ uint32_t top_s;
    const uint32_t t = blockIdx.x, padded = gridDim.x, tid = threadIdx.x;
    if (tid == 0) {
        top_s = 0;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (uint32_t i = blockIdx.x * 256u + tid; i < n_flags; i += gridDim.x * 256u) {
        flags[i] = 0;
    }
    // (Whatever this stream did before is complete now: the head kernel may read weights.)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr uint32_t HOLD = CHUNK_K / 8u / 256u;
    uint4 v[HOLD];
    uint32_t top = 0;  // the largest magnitude's bits
#pragma unroll
    for (uint32_t j = 0; j < HOLD; ++j) {
        const uint32_t i = tid + j * 256u;
        v[j] = t < tokens && i < groups * 8u ? __ldg(reinterpret_cast<const uint4 *>(hidden + (uint64_t)t * ld) + i)
                                             : make_uint4(0, 0, 0, 0);
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            top = max(top, max((w[e] << 16) & 0x7FFF0000u, w[e] & 0x7FFF0000u));
        }
    }
    __syncthreads();
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    if ((tid & 31u) == 0u) {
        atomicMax(&top_s, top);
    }
    __syncthreads();
    // The token's largest magnitude goes to [2^15, 2^16).
    const int exponent = (int)(top_s >> 23);
    const int shift = top_s == 0u ? 0 : min(142 - exponent, 126);
    const float scale = __uint_as_float((uint32_t)(shift + 127) << 23);
    // (4-bit codes: the odd columns' stand for 16 times their value, all for 2^-24 times.)
    const float scale_odd = nibbles ? __fmul_rn(scale, 0.0625f) : scale;
    const int codes = nibbles ? 24 : 0;
    // (A token of extreme size stays as it is: a scaled sum might overflow where its own does not.)
    uint32_t lost = shift < -40 || shift > 40 ? 1u : 0u;
#pragma unroll
    for (uint32_t j = 0; j < HOLD; ++j) {
        const uint32_t i = tid + j * 256u, g = i >> 3, chunk = i & 7u;
        if (g >= groups) {
            continue;  // (whole warps: groups come in eights)
        }
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        uint32_t h[4];
        float sum = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float lo = __uint_as_float(w[e] << 16), hi = __uint_as_float(w[e] & 0xFFFF0000u);
            sum += lo;
            sum += hi;
            const __half a = __float2half_rn(__fmul_rn(lo, scale)), b = __float2half_rn(__fmul_rn(hi, scale_odd));
            lost |= __half2float(a) == __fmul_rn(lo, scale) && __half2float(b) == __fmul_rn(hi, scale_odd) ? 0u : 1u;
            h[e] = (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        }
        const size_t at = ((size_t)g * padded + t) * 8u + (chunk ^ (t & 7u));
        auto ordered = [&](const uint32_t (&x)[4]) -> uint4 {
            return nibbles ? make_uint4(__byte_perm(x[0], x[2], 0x5410), __byte_perm(x[0], x[2], 0x7632),
                                        __byte_perm(x[1], x[3], 0x5410), __byte_perm(x[1], x[3], 0x7632))
                           : make_uint4(__byte_perm(x[0], x[1], 0x5410), __byte_perm(x[0], x[1], 0x7632),
                                        __byte_perm(x[2], x[3], 0x5410), __byte_perm(x[2], x[3], 0x7632));
        };
        p.image[0][at] = ordered(h);
        p.image[1][at] = ordered(w);
        if (chunk == 0u) {
            p.sums[0][g * padded + t] = __fmul_rn(sum, __uint_as_float((uint32_t)(shift - codes + 127) << 23));
            p.sums[1][g * padded + t] = sum;
        }
    }
    const int any = __syncthreads_or((int)lost);
    if (tid == 0) {
        p.unscale[t] = __uint_as_float((uint32_t)(127 - shift + codes) << 23);
        p.inexact[t] = any ? 1u : 0u;
    }
}

template <uint32_t N, int FMT>
__global__ void __launch_bounds__(Shape<N, FMT>::THREADS, 1) lmhead_kernel(const __grid_constant__ Args a) {
    using S = Shape<N, FMT>;
    constexpr bool AFFINE = FMT != FMT_S8;
    constexpr uint32_t RG = FMT == FMT_U4 ? 4u : 2u;  // groups per stage
    constexpr unsigned FULL = 0xFFFFFFFFu;
    extern __shared__ uint8_t smem_unaligned[];
    const uint32_t base = (smem_u32(smem_unaligned) + 1023u) & ~1023u;
    uint8_t *base_ptr = smem_unaligned + (base - smem_u32(smem_unaligned));
    volatile uint32_t *abort_word = reinterpret_cast<volatile uint32_t *>(base_ptr + S::ABORT);
    volatile uint32_t *tmem_word = reinterpret_cast<volatile uint32_t *>(base_ptr + S::TMEM_ADDR);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint64_t wait_ns = a.wait_ns;

    // This block's work, in units of BLOCK_GROUPS groups, numbered through all tiles: an
    // even share of them, [lo, hi), cut where it ends. A tile that two blocks work on is
    // one chain of sums all the same (a row's logit must not depend on how many rows the
    // head has): its second block goes on from the first one's sums. So the beginning of
    // a tile at the share's end comes first, then whole tiles, and the rest of the tile
    // that the block before began comes last, when that block has long left its sums.
    // With fewer tiles than blocks a block would wait for all of its predecessor's work:
    // every block takes one whole tile (units of `grain`).
    const uint32_t per_tile = a.groups / BLOCK_GROUPS;
    const uint32_t n_tiles = (a.rows + TILE_ROWS - 1u) / TILE_ROWS;
    const uint32_t grain = n_tiles <= gridDim.x ? per_tile : 1u, shares = n_tiles * per_tile / grain;
    auto share_begin = [&](uint32_t b) { return (uint32_t)((uint64_t)b * shares / gridDim.x) * grain; };
    const uint32_t lo = share_begin(blockIdx.x), hi = share_begin(blockIdx.x + 1u), n_blocks = hi - lo;
    const uint32_t begun = hi % per_tile;                                  // units of the tile it begins
    const uint32_t rest = (per_tile - lo % per_tile) % per_tile;           // units of the tile it ends
    auto unit_at = [&](uint32_t n) -> uint32_t {                           // its n-th unit
        return n < begun ? hi - begun + n : n < n_blocks - rest ? lo + rest + (n - begun) : lo + (n - (n_blocks - rest));
    };
    constexpr uint32_t STAGES_PER_BLOCK = BLOCK_GROUPS / RG;
    const uint32_t n_stages = n_blocks * STAGES_PER_BLOCK, total_groups = n_blocks * BLOCK_GROUPS;
    // (Wait's results: true means that the block has given up.)
    auto wait = [&](uint32_t bar, uint32_t phase) -> bool { return mbar_wait(base + bar, phase & 1u, abort_word, wait_ns); };
    auto wait_all = [&](uint32_t bar, uint32_t phase) -> bool { return warp_wait(base + bar, phase & 1u, abort_word, wait_ns); };

    if (tid == 0) {
        for (uint32_t s = 0; s < S::RAW_STAGES; ++s) {
            mbar_init(base + S::RAW_FULL + 8 * s, 1);
            mbar_init(base + S::RAW_EMPTY + 8 * s, S::CONV_WARPS);
        }
        for (uint32_t s = 0; s < S::H_SLOTS / 2u; ++s) {
            mbar_init(base + S::H_FULL + 8 * s, 1);
        }
        for (uint32_t s = 0; s < 2u * S::A_SLOTS; ++s) {
            mbar_init(base + S::A_FULL + 8 * s, 4 * S::PG);
        }
        for (uint32_t s = 0; s < 2u * S::DONE_SLOTS; ++s) {
            mbar_init(base + S::DONE + 8 * s, 1);
        }
        for (uint32_t b = 0; b < 2u * S::ACC_BUFS; ++b) {
            mbar_init(base + S::ACC_EMPTY + 8 * b, 4);
        }
        for (int w = 0; w < MMA_WARPS; ++w) {
            mbar_init(base + S::FINAL + 8 * w, 1);
        }
        for (uint32_t s = 0; s < S::S_SLOTS; ++s) {
            mbar_init(base + S::S_FULL + 8 * s, 64);
            mbar_init(base + S::S_EMPTY + 8 * s, S::EPI_WARPS);
        }
        *abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0u) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + S::TMEM_ADDR),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_word;

    // The weights and scales do not come from the launch before this one, and what came before
    // that has completed (see prepare_hidden_kernel): their loads start at once.
    bool bf16 = false;
    if (warp != WARP_LOAD_W && (warp & ~1u) != WARP_LOAD_S0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t inexact = 0;
        for (uint32_t t = lane; t < N; t += 32u) {
            inexact |= __ldcg(a.prep.inexact + t);
        }
        bf16 = __any_sync(FULL, inexact != 0u);
    }

    if (warp < (uint32_t)WARP_CONV0) {
        set_registers<S::REGS_CTRL, false>();
        if (warp < MMA_WARPS) {
            // ---- four issuing warps: one per 128 rows of the tile and parity of the group (a
            // group's waits, multiplies and commit take one warp longer than the group's
            // weights take to arrive). The whole warp goes through
            // the loop and one elected lane issues: everything the instruction takes is then
            // the same in all lanes and lives in uniform registers. (Issued from a branch of
            // lane 0 alone a multiply cost that thread 110 clocks, whatever its size.)
            const uint32_t mw = __shfl_sync(FULL, warp, 0), half = mw & 1u;
            const bool leader = elect_one();
            const uint32_t idesc = instr_desc<N>(bf16);
            const uint32_t acc0 = tmem + half * 256u, a0 = acc0 + S::A_COL0;
            for (uint32_t q = mw >> 1; q < total_groups / S::PG; q += MMA_WARPS / 2) {
                const uint32_t as = q % S::A_SLOTS, hs = q * S::PG % S::H_SLOTS, b = q % S::ACC_BUFS;
                if (wait_all(S::H_FULL + 8 * (hs / 2u), q * S::PG / S::H_SLOTS) ||
                    wait_all(S::A_FULL + 8 * (half * S::A_SLOTS + as), q / S::A_SLOTS) ||
                    wait_all(S::ACC_EMPTY + 8 * (half * S::ACC_BUFS + b), (q / S::ACC_BUFS) ^ 1u)) {
                    break;
                }
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (uint32_t g = 0; g < S::PG; ++g) {
                        const uint64_t bdesc = operand_desc(base + S::HID + (hs + g) * S::H_BYTES);
#pragma unroll
                        for (uint32_t k4 = 0; k4 < 4; ++k4) {
                            mma_ts(acc0 + (b * S::PG + g) * N, a0 + (as * S::PG + g) * 32u + k4 * 8u, bdesc + k4 * 2u, idesc, k4);
                        }
                    }
                    mma_commit(base + S::DONE + 8 * (half * S::DONE_SLOTS + q % S::DONE_SLOTS));
                }
                __syncwarp();
            }
            // The multiplies that were issued must have run before the tensor memory they
            // use is freed. On the normal way out the epilogue has seen to that already and
            // this wait finds its phase complete; it matters when the block has given up.
            if (leader) {
                mma_commit(base + S::FINAL + 8 * mw);
                mbar_drain(base + S::FINAL + 8 * mw, 0u, wait_ns);
            }
            __syncwarp();
        } else if (warp == WARP_LOAD_W) {
            // ---- one thread asks for every stage of weights, as far ahead as slots are free
            if (lane == 0) {
                // The copies asked for last, per slot (bit s: slot s has one; its phase's
                // parity beside it): what the way out has to wait for if the block gives up.
                uint32_t asked = 0, parity = 0;
                uint32_t tile = 0, stage = 0;
                for (uint32_t i = 0; i < n_stages; ++i) {
                    if (i % STAGES_PER_BLOCK == 0u) {
                        const uint32_t unit = unit_at(i / STAGES_PER_BLOCK);
                        tile = unit / per_tile;
                        stage = unit % per_tile * STAGES_PER_BLOCK;
                    }
                    const uint32_t st = i % S::RAW_STAGES, use = i / S::RAW_STAGES;
                    if (wait(S::RAW_EMPTY + 8 * st, use ^ 1u)) {
                        break;
                    }
                    if (!(i == a.lost_stage && blockIdx.x == 0)) {  // (test hook: the stage never fills)
                        asked |= 1u << st;
                        parity = (parity & ~(1u << st)) | ((use & 1u) << st);
                        mbar_expect_tx(base + S::RAW_FULL + 8 * st, RAW_STAGE_BYTES);
                        tma_load_2d(base + S::RAW + st * RAW_STAGE_BYTES, &a.w_map, base + S::RAW_FULL + 8 * st,
                                    (int32_t)(a.byte0 + stage * 128u), (int32_t)(tile * TILE_ROWS));
                    }
                    ++stage;
                }
                asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
                if (*abort_word) {
                    // The block has given up: the copies asked for land in this block's
                    // shared memory, so it stays until they have.
                    for (uint32_t s2 = 0; s2 < S::RAW_STAGES; ++s2) {
                        if ((asked >> s2) & 1u) {
                            mbar_drain(base + S::RAW_FULL + 8 * s2, (parity >> s2) & 1u, wait_ns);
                        }
                    }
                }
            }
            __syncwarp();
        } else if (warp == WARP_LOAD_H) {
            // ---- another warp asks for the hidden states' images (and their sums), two
            // groups per copy. (One group at a time, two waits and two copies by one thread
            // took longer than a group of 4-bit codes.)
            uint32_t asked = 0, parity = 0;
            const uint8_t *image = reinterpret_cast<const uint8_t *>(a.prep.image[bf16 ? 1 : 0]);
            const float *sums = a.prep.sums[bf16 ? 1 : 0];
            uint32_t g = 0;
            static_assert(S::H_SLOTS == S::DONE_SLOTS * S::PG, "the hidden ring and the done ring share their indexing");
            for (uint32_t q = 0; q < total_groups; q += 2u) {
                if (q % BLOCK_GROUPS == 0u) {
                    g = unit_at(q / BLOCK_GROUPS) % per_tile * BLOCK_GROUPS;
                }
                const uint32_t pair = (q / 2u) % (S::H_SLOTS / 2u), use = q / S::H_SLOTS;
                bool gave_up = false;
                if (q >= S::H_SLOTS && lane < 4u / S::PG) {  // the slot's previous two groups have been multiplied, by both halves
                    gave_up = wait(S::DONE + 8 * ((lane & 1u) * S::DONE_SLOTS + (q / S::PG + (lane >> 1)) % S::DONE_SLOTS), use ^ 1u);
                }
                if (__any_sync(FULL, gave_up)) {
                    break;
                }
                asked |= 1u << pair;
                parity = (parity & ~(1u << pair)) | ((use & 1u) << pair);
                if (lane == 0) {
                    const uint32_t bar = base + S::H_FULL + 8 * pair;
                    mbar_expect_tx(bar, 2u * S::H_BYTES + (AFFINE ? 2u * N * 4u : 0u));
                    bulk_load(base + S::HID + 2u * pair * S::H_BYTES, image + (size_t)g * S::H_BYTES, 2u * S::H_BYTES, bar);
                    if (AFFINE) {
                        bulk_load(base + S::SUMS + (q % S::SUM_SLOTS) * N * 4u, sums + (size_t)g * N, 2u * N * 4u, bar);
                    }
                }
                g += 2u;
            }
            if (lane == 0 && *abort_word) {
                for (uint32_t s2 = 0; s2 < S::H_SLOTS / 2u; ++s2) {
                    if ((asked >> s2) & 1u) {
                        mbar_drain(base + S::H_FULL + 8 * s2, (parity >> s2) & 1u, wait_ns);
                    }
                }
            }
            __syncwarp();
        } else {
            // ---- two warps ask for the scales (and biases) of every unit, a row's 16 bytes a copy
            const uint32_t r0 = tid - 32u * (uint32_t)WARP_LOAD_S0;
            for (uint32_t n = 0; n < n_blocks; ++n) {
                const uint32_t slot = n % S::S_SLOTS, unit = unit_at(n), to = base + S::SCALES + slot * S::S_SLOT_BYTES;
                if (wait_all(S::S_EMPTY + 8 * slot, (n / S::S_SLOTS) ^ 1u)) {
                    break;
                }
                const uint32_t tile = unit / per_tile, first = unit % per_tile * BLOCK_GROUPS;
#pragma unroll
                for (uint32_t i = 0; i < TILE_ROWS / 64u; ++i) {
                    const uint32_t trow = r0 + 64u * i;
                    const uint64_t at = (uint64_t)min(tile * TILE_ROWS + trow, a.rows - 1u) * a.scale_ld + first;
                    copy_async16(to + trow * 16u, a.scales + at);
                    if (AFFINE) {
                        copy_async16(to + S::S_ARRAY_BYTES + trow * 16u, a.biases + at);
                    }
                }
                // (The barrier counts this thread once its copies are there.)
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(base + S::S_FULL + 8 * slot) : "memory");
            }
            // (Whether or not the block has given up: nothing is on its way when it ends.)
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
    } else if (warp < (uint32_t)S::WARP_EPI0) {
        set_registers<S::REGS_CONV, false>();
        // ---- bytes in; one thread per tile row widens them into tensor memory. With two
        // teams of eight warps the groups alternate between them.
        const uint32_t cw = warp - WARP_CONV0, team = cw >> 3;
        const uint32_t quad = warp & 3u;            // the TMEM lanes this warp may write
        const uint32_t half = (cw >> 2) & 1u;       // which 128 rows of the tile
        const uint32_t trow = half * 128u + quad * 32u + lane;
        const uint32_t a_base = tmem + ((quad * 32u) << 16) + half * 256u + S::A_COL0;
        auto convert = [&](auto wide_exponent) {
            constexpr bool BF16 = decltype(wide_exponent)::value;
            for (uint32_t i = 0; i < n_stages; ++i) {
                const uint32_t st = i % S::RAW_STAGES;
                if (wait_all(S::RAW_FULL + 8 * st, i / S::RAW_STAGES)) {
                    return;
                }
                const uint32_t raw_row = base + S::RAW + st * RAW_STAGE_BYTES + trow * 128u;
#pragma unroll 1
                for (uint32_t gg = team; gg < RG; gg += S::TEAMS) {
                    const uint32_t q = (i * RG + gg) / S::PG, as = q % S::A_SLOTS;
                    static_assert(S::PG == 1u || S::TEAMS == 2u, "each team converts one group of a hand-over");
                    constexpr uint32_t CHUNKS = FMT == FMT_U4 ? 2u : 4u;  // of 16 bytes
                    constexpr uint32_t CW = 32u / CHUNKS;                 // words of a chunk
                    auto load_chunk = [&](uint32_t c, uint32_t (&x)[4]) {
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3])
                                     : "r"(raw_row + (((gg * CHUNKS + c) ^ (trow & 7u)) << 4)));
                    };
                    auto widen_chunk = [&](const uint32_t (&x)[4], uint32_t *o) {
#pragma unroll
                        for (uint32_t w = 0; w < 4; ++w) {
                            if (FMT == FMT_U4) {
                                widen_nibbles<BF16>(x[w], o[4u * w], o[4u * w + 1u], o[4u * w + 2u], o[4u * w + 3u]);
                            } else {
                                widen_bytes<FMT, BF16>(x[w], o[2u * w], o[2u * w + 1u]);
                            }
                        }
                    };
                    auto bytes_read = [&]() {  // the stage's bytes are in registers: the slot may be refilled
                        if (gg + S::TEAMS >= RG) {
                            __syncwarp();
                            if (lane == 0) {
                                mbar_arrive(base + S::RAW_EMPTY + 8 * st);
                            }
                        }
                    };
                    auto slot_free = [&]() -> bool {  // the slot's last user has been multiplied
                        const uint32_t before = q - S::A_SLOTS;
                        return q < S::A_SLOTS || !wait_all(S::DONE + 8 * (half * S::DONE_SLOTS + before % S::DONE_SLOTS), before / S::DONE_SLOTS);
                    };
                    const uint32_t to = a_base + (as * S::PG + (S::PG == 2u ? team : 0u)) * 32u;
                    if (!S::LEAN) {
                        // Widen first (it needs no slot), then wait for the slot: the
                        // conversion overlaps the multiplies still reading the slot.
                        uint32_t x[CHUNKS][4], o[32];
#pragma unroll
                        for (uint32_t c = 0; c < CHUNKS; ++c) {
                            load_chunk(c, x[c]);
                        }
#pragma unroll
                        for (uint32_t c = 0; c < CHUNKS; ++c) {
                            widen_chunk(x[c], o + CW * c);
                        }
                        bytes_read();
                        if (!slot_free()) {
                            return;
                        }
                        tc_fence_after();
                        tmem_st32(to, o);
                    } else {
                        // Few registers: the slot first, then half a group at a time.
                        uint32_t x[CHUNKS][4];
#pragma unroll
                        for (uint32_t c = 0; c < CHUNKS; ++c) {
                            load_chunk(c, x[c]);
                        }
                        if (!slot_free()) {
                            return;
                        }
                        tc_fence_after();
#pragma unroll
                        for (uint32_t h = 0; h < 2u; ++h) {
                            uint32_t o[16];
#pragma unroll
                            for (uint32_t c = 0; c < CHUNKS / 2u; ++c) {
                                widen_chunk(x[h * (CHUNKS / 2u) + c], o + CW * c);
                            }
                            tmem_st16(to + 16u * h, o);
                        }
                        bytes_read();
                    }
                    tmem_st_wait();
                    tc_fence_before();
                    // One arrival per warp: arrivals on one barrier are serialised.
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(base + S::A_FULL + 8 * (half * S::A_SLOTS + as));
                    }
                }
            }
        };
        if (bf16) {
            convert(std::true_type());
        } else {
            convert(std::false_type());
        }
    } else {
        set_registers<S::REGS_EPI, true>();
        // ---- scale each group's sums and add them up; write the tile
        const uint32_t e = warp - S::WARP_EPI0;
        const uint32_t quad = warp & 3u;      // the TMEM lanes this warp may read
        const uint32_t half = (e >> 2) & 1u;  // which 128 rows of the tile
        const uint32_t trow = half * 128u + quad * 32u + lane;
        const uint32_t acc_base = tmem + ((quad * 32u) << 16) + half * 256u;
        constexpr uint32_t P = N / 2u;  // tokens come in pairs
        constexpr float OFFSET = FMT == FMT_U8 ? 128.0f : 0.0f;  // (8-bit codes are widened less 128)
        float *unscale = reinterpret_cast<float *>(base_ptr + S::UNSCALE);
        const uint32_t et = tid - 32u * (uint32_t)S::WARP_EPI0, epi_threads = 32u * S::EPI_WARPS;
        auto epi_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(32 * (int)S::EPI_WARPS) : "memory"); };
        for (uint32_t t = et; t < N; t += epi_threads) {
            unscale[t] = bf16 ? 1.0f : __ldcg(a.prep.unscale + t);
        }
        epi_sync();
        uint64_t acc[P];
#pragma unroll
        for (uint32_t m = 0; m < P; ++m) {
            acc[m] = 0ull;
        }
        // (At 16 tokens, where the weights' stream is the bound, the look by itself is the faster form here:
        // affine bytes, 4 tokens, 171.2 us against 174.5.)
        auto gave_up_on = [&](uint32_t bar, uint32_t phase) -> bool {
            return N == 16u ? __any_sync(FULL, wait(bar, phase)) != 0 : wait_all(bar, phase);
        };
        auto write_out = [&](uint32_t row) {
            if (row < a.rows) {
#pragma unroll
                for (uint32_t m = 0; m < P; ++m) {
                    float v[2];
                    unpack2(acc[m], v[0], v[1]);
#pragma unroll
                    for (uint32_t h = 0; h < 2u; ++h) {
                        const uint32_t t = 2u * m + h;
                        if (t < a.tokens) {
                            float *to = a.out + (uint64_t)t * a.ldo + row;
                            const float x = __fmul_rn(v[h], unscale[t]);
                            *to = a.accumulate ? __fadd_rn(*to, x) : x;
                        }
                    }
                }
            }
        };
        // The sums of a tile's beginning, left for the next thread block's warp of the same rows: where
        // the tile's logits will be, unless something to add to lies there.
        const uint64_t part_ld = a.part ? (uint64_t)TILE_ROWS : a.ldo;
        auto part_of = [&](uint32_t block, uint32_t row) {
            return a.part ? a.part + (size_t)block * N * TILE_ROWS + trow : a.out + row;
        };
        auto flag_of = [&](uint32_t block) { return a.flags + block * S::EPI_WARPS + e; };
        uint32_t tile = unit_at(0) / per_tile, blk = unit_at(0) % per_tile, q = 0;
        for (uint32_t n = 0; n < n_blocks; ++n) {
            const uint32_t row = tile * TILE_ROWS + trow;
            uint32_t sw[4], bw[4] = {0, 0, 0, 0};
            {
                const uint32_t slot = n % S::S_SLOTS;
                if (wait_all(S::S_FULL + 8 * slot, n / S::S_SLOTS)) {
                    goto epilogue_out;
                }
                const uint4 *from = reinterpret_cast<const uint4 *>(base_ptr + S::SCALES + slot * S::S_SLOT_BYTES) + trow;
                const uint4 sc = from[0];
                sw[0] = sc.x;
                sw[1] = sc.y;
                sw[2] = sc.z;
                sw[3] = sc.w;
                if (AFFINE) {
                    const uint4 bi = from[TILE_ROWS];
                    bw[0] = bi.x;
                    bw[1] = bi.y;
                    bw[2] = bi.z;
                    bw[3] = bi.w;
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(base + S::S_EMPTY + 8 * slot);
                }
            }
            if (n == n_blocks - rest) {  // (rest = 0: never) on from where the block before stopped
                const uint64_t t0 = global_ns();
                for (uint32_t there = 0; !there;) {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(there) : "l"(flag_of(blockIdx.x - 1u)) : "memory");
                    if (__any_sync(FULL, !there && (*abort_word != 0u || global_ns() - t0 > wait_ns))) {
                        *abort_word = 1u;
                        goto epilogue_out;
                    }
                    there = __all_sync(FULL, there);
                }
                if (row < a.rows) {
                    const float *theirs = part_of(blockIdx.x - 1u, row);
#pragma unroll
                    for (uint32_t m = 0; m < P; ++m) {
                        acc[m] = pack2(2u * m < a.tokens ? __float_as_uint(__ldcg(theirs + (2u * m) * part_ld)) : 0u,
                                       2u * m + 1u < a.tokens ? __float_as_uint(__ldcg(theirs + (2u * m + 1u) * part_ld)) : 0u);
                    }
                }
            }
#pragma unroll
            for (uint32_t gi = 0; gi < BLOCK_GROUPS; ++gi, ++q) {
                const uint32_t p = q / S::PG, b = p % S::ACC_BUFS;
                const float s = __uint_as_float((gi & 1u) ? (sw[gi >> 1] & 0xFFFF0000u) : (sw[gi >> 1] << 16));
                const uint64_t s2 = pack2(__float_as_uint(s), __float_as_uint(s));
                if (gi % S::PG == 0u) {
                    if (gave_up_on(S::DONE + 8 * (half * S::DONE_SLOTS + p % S::DONE_SLOTS), p / S::DONE_SLOTS)) {
                        goto epilogue_out;  // the block has given up: nothing more is read or written
                    }
                    tc_fence_after();
                }
                const uint32_t taddr = acc_base + (b * S::PG + gi % S::PG) * N;
#pragma unroll
                for (uint32_t c = 0; c < N / 16u; ++c) {
                    uint32_t v[16];
                    tmem_ld16(taddr + 16u * c, v);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t m = 0; m < 8u; ++m) {
                        fma2(acc[8u * c + m], s2, pack2(v[2u * m], v[2u * m + 1u]));
                    }
                }
                if (gi % S::PG == S::PG - 1u) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(base + S::ACC_EMPTY + 8 * (half * S::ACC_BUFS + b));
                    }
                }
                if (AFFINE) {
                    const float bias = __uint_as_float((gi & 1u) ? (bw[gi >> 1] & 0xFFFF0000u) : (bw[gi >> 1] << 16));
                    const float add = __fmaf_rn(OFFSET, s, bias);
                    const uint64_t add2 = pack2(__float_as_uint(add), __float_as_uint(add));
                    const ulonglong2 *hs = reinterpret_cast<const ulonglong2 *>(
                        base_ptr + S::SUMS + (q % S::SUM_SLOTS) * N * 4u);
#pragma unroll
                    for (uint32_t m = 0; m < P / 2u; ++m) {
                        const ulonglong2 h = hs[m];
                        fma2(acc[2u * m], add2, h.x);
                        fma2(acc[2u * m + 1u], add2, h.y);
                    }
                }
            }
            ++blk;
            if (blk != per_tile && n + 1u != begun) {
                continue;
            }
            if (blk == per_tile) {
                write_out(row);
            } else {
                if (row < a.rows) {
                    float *mine = part_of(blockIdx.x, row);
#pragma unroll
                    for (uint32_t m = 0; m < P; ++m) {
                        float v0, v1;
                        unpack2(acc[m], v0, v1);
                        if (2u * m < a.tokens) {
                            __stcg(mine + (2u * m) * part_ld, v0);
                        }
                        if (2u * m + 1u < a.tokens) {
                            __stcg(mine + (2u * m + 1u) * part_ld, v1);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    __threadfence();
                    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag_of(blockIdx.x)), "r"(1u) : "memory");
                }
            }
#pragma unroll
            for (uint32_t m = 0; m < P; ++m) {
                acc[m] = 0ull;
            }
            tile = unit_at(n + 1u) / per_tile;
            blk = unit_at(n + 1u) % per_tile;
        }
    epilogue_out:;
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0u) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
    if (tid == 0 && *abort_word) {
        atomicOr(a.status_word, 1u << STATUS_TIMEOUT_BIT);
    }
}

}  // namespace lily_head
