// What the LM-head kernel (lmhead_kernel.cuh) and its host side share.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lily_head {

constexpr uint32_t TOK = 64;          // the most hidden rows per launch
constexpr uint32_t GROUP_K = 64;      // columns per scale
constexpr uint32_t TILE_ROWS = 256;   // two M = 128 accumulators
constexpr uint32_t BLOCK_GROUPS = 8;  // groups of a block, the unit of the shares
constexpr uint32_t CHUNK_K = 8192;    // columns of one launch, at most: wider heads take several
constexpr uint32_t EPILOGUE_WARPS = 8;
constexpr uint32_t STATUS_TIMEOUT_BIT = 30;  // bit of the handle's status word

enum Format { FMT_S8 = 0, FMT_U8 = 1, FMT_U4 = 2 };  // symmetric bytes; affine, 8 and 4 bits

// The hidden states as the multiplier wants them: the B operand's shared-memory
// image per group (padded tokens x 64 columns of 16 bits, 128-byte swizzle, columns in
// the order the converters produce the weights in), once as binary16 scaled by a
// power of two per token, once as bf16.
struct Prepared {
    uint4 *image[2];       // [binary16, bf16]: [groups][padded tokens][8]
    float *sums[2];        // [groups][padded tokens]: sums of a group's (scaled) hidden values
    float *unscale;        // [TOK] what a token's binary16 results are multiplied by
    uint32_t *inexact;     // [TOK] the token's values do not all fit binary16 exactly
};

struct Args {
    // The weights' bytes [rows, row bytes] in boxes of 256 rows x 128 bytes (TMA,
    // 128-byte swizzle). Rows past the end read 0.
    CUtensorMap w_map;
    const __nv_bfloat16 *scales;  // [rows, groups of the whole head], from this launch's first group on
    const __nv_bfloat16 *biases;
    uint32_t scale_ld;          // groups of the whole head
    uint32_t byte0;             // first byte of a weight row that this launch takes
    uint32_t tokens;            // <= 64
    uint32_t groups;            // of this launch, a multiple of BLOCK_GROUPS
    uint32_t rows;              // vocabulary rows of this shard
    uint32_t accumulate;        // add to what `out` holds (the launches of a wide head after the first)
    float *out;                 // [tokens, ldo]
    uint64_t ldo;
    Prepared prep;
    // Every thread block takes an even share of the tiles, cut where it ends. The sums of a
    // tile that a block begins and the next one ends go through `out`, or through `part`
    // ([grid][padded tokens][TILE_ROWS]; launches that add to `out`), and are there once
    // `flags` ([grid][EPILOGUE_WARPS], cleared by launch_prepare) says so.
    float *part;
    uint32_t *flags;
    uint32_t *status_word;
    uint64_t wait_ns;           // the bound of every wait inside the kernel
    // Test hook: block 0 does not ask for the weights of this stage (~0: none),
    // so that the wait of their consumers runs out.
    uint32_t lost_stage;
};

__host__ __device__ inline uint32_t padded_tokens(uint32_t tokens) { return tokens <= 16u ? 16u : tokens <= 32u ? 32u : 64u; }

// Sizes of the workspaces: the hidden states' images, flags, and `part`.
inline size_t prepared_bytes(uint32_t padded) {
    return 2u * (size_t)padded * CHUNK_K * 2u + 2u * (size_t)padded * (CHUNK_K / GROUP_K) * 4u + 2u * TOK * 4u;
}
inline size_t part_bytes(uint32_t sms) { return (size_t)sms * TOK * TILE_ROWS * sizeof(float); }

inline size_t flag_bytes(uint32_t sms) { return (size_t)sms * EPILOGUE_WARPS * sizeof(uint32_t); }

Prepared prepared_at(void *base, uint32_t padded);

// The two launches of a head (or of 8192 columns of one): the hidden states' images,
// then the products. hidden: bf16 [tokens, hidden_ld], from the launch's first column on.
cudaError_t launch_prepare(const Prepared &p, const void *hidden, uint64_t hidden_ld, uint32_t tokens, uint32_t groups,
                           Format format, uint32_t *flags, uint32_t sms, cudaStream_t stream);
cudaError_t launch_head(const Args &a, Format format, uint32_t sms, cudaStream_t stream);

}  // namespace lily_head
