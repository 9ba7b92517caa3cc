// What the row kernel (split_kernel.cuh) and its host side share: constants, the
// kernel's arguments, the sizes of its shared memory.
#pragma once

#include <math.h>

#include "sample_kernel.cuh"

namespace lily {

constexpr uint32_t SPL_NT = 256;         // threads that read the logits; the block's other half marks the row's history
constexpr uint32_t SPL_WARPS = SPL_NT / 32;
constexpr uint32_t SPL_LOG_NT = 8;
static_assert(1u << SPL_LOG_NT == SPL_NT, "");
// Vectors of a bucket: a thread's loads in flight (with two blocks per SM as many
// as 64 registers a thread hold).
__host__ __device__ constexpr uint32_t split_u(int bps) { return bps == 1 ? 10u : 6u; }
constexpr uint32_t SPL_MAX_BLOCKS = 8;   // blocks of a cluster (the portable size)
constexpr uint32_t SPL_SMALL_K = 64;     // up to here a row's bound comes from the pool and one warp draws (split_finalize)
constexpr uint32_t SPL_POOL = 256;       // keys in the pool a narrow row's bound is taken from
constexpr uint32_t SPL_HITS = 512;       // vectors of a block that may reach the bound
constexpr uint32_t SPL_FLAGGED = 2048;   // buckets that may reach the bound
constexpr uint32_t HELD_MIN = 320;       // a row of two buckets that keeps more does not read the second one again
constexpr uint32_t SPL_SORTED = 2048;    // candidates of a wide row
// Pieces of a block, at least: half of its warps have one. (With a piece for every warp, and
// so fewer blocks, 4096 bf16 that keep 64 took 14.2 us instead of 12.9.)
constexpr uint32_t SPL_MIN_TILES = SPL_WARPS / 2u;
constexpr uint32_t SPL_NAN_KEY = 0xFFFFFFFFu;  // a candidate that came out a NaN

// How a block keeps the history ids of its share.
enum { MARK_BITS = 0, MARK_BYTES = 1, MARK_COUNTS = 2 };
// Flags of a mark: the id is on the bias or ban list; it has been looked at already (a row
// whose penalties can raise a logit). MARK_MAX: the largest count beside them.
constexpr uint32_t BYTE_LISTED = 0x80u, BYTE_CLAIMED = 0x40u, BYTE_MAX = 0x3Fu;
constexpr uint32_t HALF_LISTED = 0x8000u, HALF_CLAIMED = 0x4000u, MARK_MAX = 0x3FFFu;

template <typename T>
struct Piece {
    static constexpr uint32_t PER = 16u / (uint32_t)sizeof(T);    // logits per vector
    static constexpr uint32_t SHIFT = sizeof(T) == 4 ? 7u : 8u;   // log2 of the logits per piece (32 vectors)
    static constexpr uint32_t LOGITS = 1u << SHIFT;
};

// A row's parameters as the kernel uses them.
struct RowIn {
    float temp, rep, presence, frequency, top_p, min_p;
    uint32_t k, flags;
    float u;        // the row's uniform, unless the caller gave an array of them
    uint32_t step;
    uint64_t seed;
};
enum { ROW_GREEDY = 1, ROW_PEN = 2, ROW_COUNTS = 4, ROW_RAISES = 8, ROW_BAD = 16 };

__host__ __device__ inline bool split_finite(float x) { return x - x == 0.0f; }

__host__ __device__ inline RowIn row_in(const lily_sampling_params_t &P, uint32_t step) {
    RowIn r;
    // src/kernels/sample.rs:57-79 validate, :83-94 effective.
    const bool ok = split_finite(P.temperature) && split_finite(P.top_p) && split_finite(P.min_p) &&
                    split_finite(P.repetition_penalty) && split_finite(P.presence_penalty) &&
                    split_finite(P.frequency_penalty) && P.temperature >= 0.0f && P.top_p > 0.0f &&
                    P.top_p <= 1.0f && P.min_p >= 0.0f && P.min_p <= 1.0f && P.repetition_penalty > 0.0f;
    const bool greedy = P.temperature <= 0.0f || P.top_k == 1u;
    const bool pen = P.presence_penalty != 0.0f || P.frequency_penalty != 0.0f || P.repetition_penalty != 1.0f;
    // (A negative zero counts as "can raise", as the general code has it.)
    const bool raises = P.repetition_penalty < 1.0f || signbit(P.presence_penalty) || signbit(P.frequency_penalty);
    r.temp = greedy ? 1.0f : P.temperature;
    r.rep = P.repetition_penalty;
    r.presence = P.presence_penalty;
    r.frequency = P.frequency_penalty;
    r.top_p = P.top_p;
    r.min_p = P.min_p;
    r.k = greedy ? 1u : (P.top_k == 0u || P.top_k > KCAP ? KCAP : P.top_k);
    r.flags = (greedy ? ROW_GREEDY : 0) | (pen ? ROW_PEN : 0) | (P.frequency_penalty != 0.0f ? ROW_COUNTS : 0) |
              (pen && raises ? ROW_RAISES : 0) | (ok ? 0 : ROW_BAD);
    r.u = uniform_for(P.seed, step);
    r.step = step;
    r.seed = P.seed;
    return r;
}

// The barriers at which the blocks of a row meet.
enum {
    MEET_POOL = 0,    // every block's keys have arrived
    MEET_CANDIDATES,  // first block: every block's candidates have arrived
    MEET_LISTS,       // wide rows: the sorted lists of all blocks have arrived
    MEET_SUMS,        // first block: every block's sums of exponentials have arrived
    MEET_GONE,        // wide rows: this block's list has arrived in every block
    MEETS
};

struct alignas(16) SplitSmem {
    unsigned long long mbar[MEETS];
    uint4 head[SPL_MAX_BLOCKS];      // first block: a block's number of candidates, flag, bound
    uint2 sums[SPL_MAX_BLOCKS * SPL_WARPS];  // first block, a shard's record: (reference, sum) of every warp
    union {
        struct {
            alignas(16) uint32_t pool[SPL_POOL];  // the best keys of every warp of the cluster
            // Buckets that reach the bound. (The maxima have served by then, and a block that waited for them in vain
            // lists none; the pool may still be read. By itself this list kept a second block of 151937 f32 logits off an SM: 256 rows 77 us, so 48.)
            uint16_t flagged[SPL_FLAGGED];
        };
        uint32_t tmax[SPL_MAX_BLOCKS * SPL_NT];  // wide rows: the keys of all its threads
    };
    uint32_t hit_at[SPL_HITS];       // vectors that reach the bound: the id of their first logit (mod 2^32)
    uint32_t n_flagged;
    uint32_t n_hits;
    uint32_t n_listed;               // ids on the row's bias list that are this block's
    uint32_t n_sent;
    uint32_t n_live;
    uint32_t hard;                   // the row goes to the general code
    uint32_t bin;
    uint32_t verdict[2];             // what the waiting warps of the first block learn
    uint32_t bound_key;
    uint32_t record_key;             // a shard's largest adjusted logit
    float least;                     // what an adjusted logit has to reach
    uint32_t late;                   // a wait of this block ran out: others may still store into it
};
static_assert(sizeof(SplitSmem) % 16u == 0u, "the arrays behind it are 16-byte aligned");

// Parameters of up to MAXR rows travel in the kernel's own arguments: no staging
// copy sits in front of the launch.
template <uint32_t MAXR>
struct SplitArgs {
    KArgs a;
    uint32_t log_blocks;      // log2 of the blocks per row
    uint32_t log_live;        // log2 of the warps of a block that have pieces, at least (2 or 3)
    uint32_t two_per_sm;      // more rows than SMs: the instantiation of which two blocks fit
    uint32_t mark_mode;
    uint32_t mark_words;      // 32-bit words of the marks, a multiple of four
    uint32_t inline_params;   // `in` below is valid (else a.params / a.steps)
    uint32_t inline_slots;    // `slots` below is (both only with inline_params)
    uint32_t inline_history;  // 1 + the history length of every row (0: a.history_len)
    // Test hook: block lost >> 8 of every cluster waits for one arrival too many at its
    // barrier (lost & 255) - 1, so that the wait runs out (0: none).
    uint32_t lost;
    uint64_t wait_ns;         // the bound of every wait of a block for the others (wait_first_phase: a row's
                              // earlier meetings have a part of it)
    RowIn in[MAXR];
    // Keys that a warp gives to the pool of a row that keeps k: so much above its share
    // that all but some three of the best k are in the pool. (What is missing there
    // lowers the bound by as many places. Shares of all warps where half of them have nothing
    // left the pool with fewer than k keys, and the row to the general code: 1 x 520, 20 kept, 25 us.)
    __device__ __forceinline__ uint32_t rounds_of(uint32_t k) const {
        const uint32_t share10 = (k * 10u) >> (log_live + log_blocks);  // tenths
        static_assert(SPL_WARPS == 8u && SPL_MIN_TILES == 4u, "");
        return min((share10 * 13u + 170u) / 100u, SPL_POOL / (SPL_WARPS << log_blocks));
    }
    uint32_t slots[MAXR];
};

// Pieces of a row, and the most of them a block has.
__host__ __device__ inline uint32_t split_pieces(uint32_t vocab, uint32_t skip, uint32_t per) {
    const uint32_t piece = 32u * per;
    return (vocab + skip + piece - 1u) / piece;
}

__host__ __device__ inline uint32_t split_buckets(uint32_t pieces_of_block, uint32_t u) {
    return (pieces_of_block + SPL_WARPS * u - 1u) / (SPL_WARPS * u);
}

// What the rows of a launch may bring beside a narrow draw: rows that keep more than SPL_SMALL_K; shards' records
// in place of draws; bias or ban lists; penalties that can raise a logit; a proposal to verify. The kernel is
// compiled for some sets of these and for everything; a launch takes a variant that has what its rows bring, as
// far as the host knows them. (With parameters on the device it does not know what they keep, nor whether
// they raise a logit.) Code that a row never runs slows down the chain of steps it does run: with everything, with
// nothing of this, and so for rows over several blocks alone, 1 x 151936 f32 8.75, 7.66 and 7.44 us, with 4096 ids
// 9.26, 8.18 and 7.96; 3 x 151936 bf16 with ids 8.82, 7.48 and 7.32; 8 x 248320 f32 11.4, 10.2 and 10.0.
enum : uint32_t {
    HAS_WIDE = 1, HAS_SHARD = 2, HAS_LISTS = 4, HAS_RAISES = 8, HAS_SPEC = 16, HAS_ALL = 31,
    HAS_ARGMAX = 32  // (nothing but: parameters, lists, slots and forced ids are not looked at)
};
// Parameters on the device, no lists; and of up to 8 rows what else needs no more than this: rows whose penalties
// raise a logit (4 x 151936 bf16, 4096 ids: 14.85 us with everything, 13.45 so; 8 x 151936 f32 12.7, 11.95), and rows in
// one block (1 x 1000 f32: 8.24, 7.60).
constexpr uint32_t HAS_UNKNOWN = HAS_WIDE | HAS_RAISES;
// Rows whose parameters travel in the kernel's arguments: sizes of the argument block (a
// larger one takes longer to launch), the last one as many rows as the chip has SMs.
constexpr uint32_t INLINE_ROWS = 8, INLINE_ROWS_MID = 64, INLINE_ROWS_MAX = 148;
// Variants whose rows' parameters all lie in the arguments, and those of them whose rows all lie over two blocks or
// more: not of the largest argument block, whose launches have one block a row from 75 rows on. (No launch of
// other rows takes them: split_takes in split_launch.cuh.)
__host__ __device__ constexpr bool variant_inline(uint32_t has) {
    return has != HAS_ALL && has != HAS_ARGMAX && has != HAS_UNKNOWN;
}
__host__ __device__ constexpr bool variant_many(uint32_t has, uint32_t max_rows) {
    return variant_inline(has) && max_rows != INLINE_ROWS_MAX;
}

// Launches the kernel for a.a.rows rows from row0 on: logits of `dtype`, `smem` bytes of
// dynamic shared memory (at most what split_ready was given); `has`: what the rows may bring, HAS_ALL if that is not
// known. Instantiated in split*.cu.
template <uint32_t MAXR>
cudaError_t split_launch(const SplitArgs<MAXR> &a, uint32_t has, uint32_t rows, uint32_t dtype, size_t smem,
                         cudaStream_t stream);

// Loads every variant that launches of up to max_rows rows can take on the current device, and lets it have max_smem
// bytes of shared memory. (Left to the launches, the first request of another kind would wait 0.2 to 1 ms for
// its kernel in the middle of serving, or 4 to 19 where it is the first of its translation unit.)
cudaError_t split_ready(uint32_t max_rows, uint32_t sms, int max_smem);

// The most rows that clusters of 1 << log_blocks blocks run at once, one block per SM. Less
// than the SMs would hold (15 clusters of eight on 148 SMs, 33 of four): a cluster lies in
// one group of SMs, and those do not divide evenly.
uint32_t split_rows_at_once(int device, int sm_count, int max_smem, uint32_t log_blocks);

// The merge of the shards' records (merge_kernel.cuh). a.params set: the rows' parameters
// and steps are there, else in `in`.
struct MergeArgs {
    KArgs a;
    RowIn in[INLINE_ROWS_MID];
};
cudaError_t merge_launch(const MergeArgs &a, uint32_t rows, cudaStream_t stream);
cudaError_t merge_ready();

}  // namespace lily
