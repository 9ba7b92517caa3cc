// Host side of the C ABI declared in include/lily_sampler.h: argument
// checks, parameter staging, launch geometry. All device work is enqueued on
// the caller's stream; nothing here falls back to the CPU.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/lily_batch.h"
#include "../../include/lily_sampler.h"
#include "sample_kernel.cuh"
#include "stream_kernel.cuh"
#include "split_args.cuh"
#include "lmhead_args.cuh"

namespace {

constexpr int RING = 8;

struct StageLayout {
    size_t params, steps, slots, hist_len, total;
};

StageLayout stage_layout(uint32_t max_rows) {
    StageLayout l;
    size_t off = 0;
    l.params = off;
    off += sizeof(lily_sampling_params_t) * max_rows;
    l.steps = off;
    off += sizeof(uint32_t) * max_rows;
    l.slots = off;
    off += sizeof(uint32_t) * max_rows;
    l.hist_len = off;
    off += sizeof(uint32_t) * max_rows;
    l.total = (off + 255) & ~size_t(255);
    return l;
}

}  // namespace

struct lily_sampler {
    int device = 0;
    uint32_t vocab = 0, max_rows = 0, max_history = 0, max_list = 0, flags = 0;
    std::string last_error;
    int32_t fault = 0;
    uint64_t wait_ns = 1000000000ull;     // bound of the waits inside the kernels
    uint32_t lost_arrival = 0;            // test hook: what SplitArgs::lost of the next row-kernel launch is
    uint32_t lost_stage = 0xFFFFFFFFu;    // test hook: a weight copy the next head launch leaves out
    int sm_count = 0;
    int max_smem = 0;
    uint2 *part = nullptr;
    uint32_t *part_n = nullptr;
    uint32_t *tickets = nullptr;
    uint32_t *status_word = nullptr;
    char *arena = nullptr;  // the device workspaces below are places in it, the staging ring's host side lies behind h_status
    uint32_t *counts_scratch = nullptr;
    uint32_t *counts_table = nullptr;
    uint32_t *seen_table = nullptr;
    uint32_t seen_words = 0;
    StageLayout layout{};
    char *h_stage[RING] = {};
    char *d_stage[RING] = {};
    cudaEvent_t ev[RING] = {};
    int ring_pos = 0;
    uint32_t *h_status = nullptr;
    long long *phase_clocks = nullptr;
    // The parameters a sharded call staged last: a decode step stages the same
    // rows for its candidate call and its merge call, and usually again next step.
    uint64_t slot_serial[RING] = {};
    int shard_slot = -1;
    uint64_t shard_serial = 0;
    std::vector<char> shard_bytes;
    float *lm_logits = nullptr;  // LILY_FLAG_LMHEAD: F32 [64, lm_ld]
    uint64_t lm_ld = 0;
    // The LM head's workspaces: the hidden states' images (for lm_tokens padded tokens) and
    // the flags of sums handed on. lm_more: those of calls of more tokens than max_rows or of
    // more than CHUNK_K columns, made by the first of them.
    char *lm_prepared = nullptr, *lm_more = nullptr;
    uint32_t *lm_flags = nullptr;
    uint32_t lm_tokens = 0;
};

namespace {

int32_t fail(lily_sampler *h, int32_t code, const char *msg) {
    if (h) {
        h->last_error = msg;
    }
    return code;
}

int32_t cuda_fail(lily_sampler *h, cudaError_t e, const char *what) {
    if (h) {
        h->last_error = std::string(what) + ": " + cudaGetErrorString(e);
    }
    return LILY_ERR_CUDA;
}

#define CU(h, call)                              \
    do {                                         \
        cudaError_t e_ = (call);                 \
        if (e_ != cudaSuccess) {                 \
            return cuda_fail((h), e_, #call);    \
        }                                        \
    } while (0)

struct DeviceGuard {
    int prev = -1;
    bool ok = true, moved = false;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) {
            prev = -1;
        }
        if (prev != dev) {
            moved = true;
            ok = cudaSetDevice(dev) == cudaSuccess;
        }
    }
    ~DeviceGuard() {
        if (moved && prev >= 0) {
            cudaSetDevice(prev);
        }
    }
};

bool params_ok(const lily_sampling_params_t &p) {
    return std::isfinite(p.temperature) && p.temperature >= 0.0f && std::isfinite(p.top_p) &&
           p.top_p > 0.0f && p.top_p <= 1.0f && std::isfinite(p.min_p) && p.min_p >= 0.0f &&
           p.min_p <= 1.0f && std::isfinite(p.repetition_penalty) &&
           p.repetition_penalty > 0.0f && std::isfinite(p.presence_penalty) &&
           std::isfinite(p.frequency_penalty);
}

bool is_greedy(const lily_sampling_params_t &p) {
    return p.temperature <= 0.0f || p.top_k == 1u;
}

bool uses_penalties(const lily_sampling_params_t &p) {
    return p.presence_penalty != 0.0f || p.frequency_penalty != 0.0f ||
           p.repetition_penalty != 1.0f;
}

uint32_t effective_k(const lily_sampling_params_t &p) {
    if (is_greedy(p)) {
        return 1u;
    }
    return p.top_k == 0u ? LILY_K_CAP : (p.top_k < LILY_K_CAP ? p.top_k : LILY_K_CAP);
}

// A staging slot whose previous use has left the stream.
int32_t next_stage(lily_sampler *h, int *slot) {
    const int s = h->ring_pos;
    h->ring_pos = (h->ring_pos + 1) % RING;
    CU(h, cudaEventSynchronize(h->ev[s]));
    ++h->slot_serial[s];
    *slot = s;
    return LILY_OK;
}

size_t smem_bytes(uint32_t vocab, uint32_t n_slices) {
    // The largest slice a row can get is the whole row: a row that keeps many
    // candidates and takes the two-pass route is not cut, whatever n_slices is
    // (the kernel decides per row; the seen bitmap must fit either way).
    (void)n_slices;
    const uint32_t slice_len = (vocab + 255u) & ~255u;
    const size_t words = (slice_len + 31u) / 32u + 8u;
    return sizeof(lily::SmemFixed) + lily::RING_BYTES + words * sizeof(uint32_t);
}

// Programmatic stream serialisation: the grid may be set up and its blocks may
// start while the stream's previous kernel drains; the kernels wait
// (griddepcontrol.wait) before they read or write any global memory.
template <typename Kernel>
int32_t launch_serialised(lily_sampler *h, cudaStream_t stream, Kernel kernel, dim3 grid, size_t smem,
                          const lily::KArgs &a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(lily::NT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CU(h, cudaLaunchKernelEx(&cfg, kernel, a));
    return LILY_OK;
}

int32_t launch_accept(lily_sampler *h, cudaStream_t stream, const uint32_t *draws, const uint32_t *ids, uint32_t id_offset,
                      uint32_t m, uint32_t *ctrl, uint32_t pos0, uint32_t ratio, uint32_t chain, uint32_t stride) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, 1);
    cfg.blockDim = dim3(1, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CU(h, cudaLaunchKernelEx(&cfg, lily::spec_accept_kernel, draws, ids, id_offset, m, ctrl, pos0, ratio, chain, stride));
    return LILY_OK;
}

// Whether a call goes to the kernel of one block per row (see launch_one).
bool stream_route(const lily::KArgs &a, uint32_t rows, uint32_t dtype) {
    const size_t esize = dtype == LILY_F32 ? 4 : 2;
    const bool vec = (reinterpret_cast<uintptr_t>(a.logits) % 16u == 0u) && ((a.logits_ld * esize) % 16u == 0u);
    const uint32_t round = dtype == LILY_F32 ? lily::Geo<float>::ROUND : lily::Geo<__nv_bfloat16>::ROUND;
    return vec && a.vocab / round >= lily::STREAM_MIN_ROUNDS && a.merge_in == nullptr && a.spec.n_spec == 0u &&
           a.extra_len == 0u && rows >= lily::STREAM_MIN_ROWS && (a.cand_out == nullptr || a.shard_k <= lily::STREAM_K_MAX);
}

template <typename T, bool VEC>
int32_t launch_one(lily_sampler *h, cudaStream_t stream_, const lily::KArgs &a, uint32_t rows,
                   size_t smem) {
    // What the row kernel leaves (split_plan): aligned long rows, more of them than SMs, go to
    // the kernel of one block per row, which runs the general code itself, on the whole row,
    // for the rows it does not take; a vocabulary shard's candidate launch goes the same way
    // and ends in the rows' records. (16 rows and more of vocabularies whose marks do not fit a
    // block of the row kernel, beyond 700000, too.) Everything else, rows shorter than the row
    // kernel's least and the merge of shards among it: the general kernel, rows cut into slices.
    const bool stream = VEC && stream_route(a, rows, sizeof(T) == 4 ? LILY_F32 : LILY_BF16);
    if (stream) {
        lily::KArgs whole = a;
        whole.n_slices = 1;
        const size_t smem1 = smem_bytes(a.vocab, 1);
        const bool plain = a.cand_out == nullptr && a.count_slots == nullptr;
        const bool many = rows > (uint32_t)h->sm_count;
        auto kernel = plain ? (many ? lily::stream_rows_kernel<T, 2, true> : lily::stream_rows_kernel<T, 3, true>)
                            : (many ? lily::stream_rows_kernel<T, 2, false> : lily::stream_rows_kernel<T, 3, false>);
        return launch_serialised(h, stream_, kernel, dim3(rows, 1, 1), smem1, whole);
    }
    return launch_serialised(h, stream_, lily::sample_rows_kernel<T, VEC>, dim3(a.n_slices, rows, 1), smem, a);
}

// Parameters of more rows than a launch's own arguments take go to the device in the
// arguments of a launch of their own: stored first, then the stream's previous work is
// waited for, so that the launch behind it may trust its own wait. (A copy from pinned
// memory between two kernels cost some 10 us of the stream's time: 256 rows x 32768 took
// 25.9 us with it.)
template <uint32_t BYTES>
struct PutArgs {
    uint4 *to;
    uint32_t n;  // 16-byte words
    uint4 data[BYTES / 16u];
};

constexpr uint32_t PUT_THREADS = 64;

template <uint32_t BYTES>
__global__ void __launch_bounds__(PUT_THREADS) put_kernel(const __grid_constant__ PutArgs<BYTES> p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t i = blockIdx.x * PUT_THREADS + threadIdx.x;
    if (i < p.n) {
        p.to[i] = p.data[i];
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <uint32_t BYTES>
cudaError_t put(void *to, const void *from, size_t bytes, cudaStream_t stream) {
    PutArgs<BYTES> p;
    p.to = static_cast<uint4 *>(to);
    p.n = (uint32_t)(bytes / 16u);
    std::memcpy(p.data, from, bytes);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.n + PUT_THREADS - 1u) / PUT_THREADS, 1, 1);
    cfg.blockDim = dim3(PUT_THREADS, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, put_kernel<BYTES>, p);
}

// The first `bytes` (a multiple of 256) of a staging slot to the device. (A launch takes
// somewhat less than 32 KB of arguments.)
int32_t upload(lily_sampler *h, int slot, size_t bytes, cudaStream_t stream) {
    void *to = h->d_stage[slot];
    const void *from = h->h_stage[slot];
    CU(h, bytes <= 4096u    ? put<4096>(to, from, bytes, stream)
          : bytes <= 16384u ? put<16384>(to, from, bytes, stream)
          : bytes <= 32000u ? put<32000>(to, from, bytes, stream)
                            : cudaMemcpyAsync(to, from, bytes, cudaMemcpyHostToDevice, stream));
    return LILY_OK;
}

// How the row kernel is launched: the blocks a row is split over, and how each
// keeps the history ids of its share.
struct SplitPlan {
    bool take = false;
    bool sole = false;   // at most one block per SM
    uint32_t log_blocks = 0, log_live = 0, mark_mode = lily::MARK_BITS, mark_words = 0;
    size_t smem = 0;
};

using lily::INLINE_ROWS;
using lily::INLINE_ROWS_MAX;
using lily::INLINE_ROWS_MID;

// `lists`: rows may bring a list of ids (history, bias, ban, or ids drawn earlier
// in the step); `counts`: a history list with a frequency penalty.
SplitPlan split_plan(const lily_sampler *h, const lily::KArgs &a, uint32_t rows, uint32_t dtype, bool lists,
                     bool counts) {
    SplitPlan p;
    if (a.merge_in != nullptr || (a.cand_out != nullptr && a.shard_k > lily::SPL_SMALL_K)) {
        return p;
    }
    const uint32_t per = dtype == LILY_F32 ? lily::Piece<float>::PER : lily::Piece<__nv_bfloat16>::PER;
    const uint32_t logits = 32u * per;
    if (a.vocab / logits < lily::SPL_MIN_TILES) {
        return p;
    }
    const uint32_t pieces = lily::split_pieces(a.vocab, per - 1u, per);
    const size_t general = smem_bytes(a.vocab, 1);  // the first block may run the general row code
    // As many blocks per row as still run all rows at once (with a second wave of clusters
    // 16 rows took 15.6 us, with clusters of half the size 9.9).
    uint32_t lb = 3;
    while (lb > 0u && ((a.vocab / logits) >> lb < lily::SPL_MIN_TILES ||
                       rows > lily::split_rows_at_once(h->device, h->sm_count, h->max_smem, lb))) {
        --lb;
    }
    p.sole = rows <= lily::split_rows_at_once(h->device, h->sm_count, h->max_smem, lb);
    const uint32_t here = (pieces + (1u << lb) - 1u) >> lb, entries = here * logits;
    const size_t fixed = sizeof(lily::SmemFixed) + sizeof(lily::SplitSmem) +
                         (size_t)lily::split_buckets(here, lily::split_u(p.sole ? 1 : 2)) * lily::SPL_NT * 4u;
    p.log_blocks = lb;
    p.log_live = (a.vocab / logits) >> lb < lily::SPL_WARPS ? 2u : 3u;
    if (lists) {
        const size_t limit = p.sole ? (size_t)h->max_smem : 113u * 1024u;
        if (counts && fixed + (size_t)entries * 2u <= limit) {
            p.mark_mode = lily::MARK_COUNTS;
            p.mark_words = entries / 2u;
        } else if (fixed + entries <= limit) {
            p.mark_mode = lily::MARK_BYTES;
            p.mark_words = entries / 4u;
        } else {
            p.mark_mode = lily::MARK_BITS;
            p.mark_words = (entries / 32u + 3u) & ~3u;
        }
    }
    p.smem = fixed + (size_t)p.mark_words * 4u;
    p.smem = p.smem > general ? p.smem : general;
    // More rows than SMs: two blocks to an SM, unless the kernel of one block per row takes the
    // call (aligned logits), which reads further ahead. 256 rows x 151936 bf16 with 1024 ids a row: 31.0 us here,
    // 27.0 there; 200 x 100352 f32 33.7 and 26.2; 256 x 50304 f32 22.3 and 20.0. What only the general kernel took,
    // 256 rows: x 151937 bf16 with 4096 ids a row 31.0, with 32768 39.1; x 50257 f32 with 8192 ids 24.0
    // (the general kernel, by its first measurement, with ids of a power law: 122, 128 and 55.5).
    p.take = p.smem <= (size_t)h->max_smem && (p.sole || !stream_route(a, rows, dtype));
    return p;
}

template <uint32_t MAXR>
int32_t launch_split(lily_sampler *h, cudaStream_t stream, lily::SplitArgs<MAXR> &sa, const SplitPlan &p,
                     uint32_t has, uint32_t rows, uint32_t dtype) {
    sa.log_blocks = p.log_blocks;
    sa.log_live = p.log_live;
    sa.two_per_sm = p.sole ? 0u : 1u;
    sa.mark_mode = p.mark_mode;
    sa.mark_words = p.mark_words;
    sa.wait_ns = h->wait_ns;
    sa.lost = h->lost_arrival;
    h->lost_arrival = 0;  // one launch only
    CU(h, lily::split_launch<MAXR>(sa, has, rows, dtype, p.smem, stream));
    return LILY_OK;
}

// The row kernel with host parameters in its arguments. sa.a is complete but for
// params, steps and slots, which come as host arrays.
template <uint32_t MAXR>
int32_t launch_split_inline(lily_sampler *h, cudaStream_t stream, const lily::KArgs &a, const SplitPlan &p,
                            uint32_t rows, uint32_t dtype, const lily_sampling_params_t *params,
                            const uint32_t *steps, const uint32_t *slots, uint32_t inline_history = 0,
                            uint32_t grid_rows = 0) {
    lily::SplitArgs<MAXR> sa;
    sa.a = a;
    sa.a.params = nullptr;
    sa.a.steps = nullptr;
    sa.a.count_slots = nullptr;
    sa.inline_params = 1;
    sa.inline_slots = slots != nullptr ? 1u : 0u;
    sa.inline_history = inline_history;
    uint32_t has = (a.cand_out != nullptr ? lily::HAS_SHARD : 0u) | (a.spec.n_spec != 0u ? lily::HAS_SPEC : 0u) |
                   (a.bias_ids != nullptr || a.ban_ids != nullptr ? lily::HAS_LISTS : 0u);
    for (uint32_t r = 0; r < rows; ++r) {
        sa.in[r] = lily::row_in(params[r], steps != nullptr ? steps[r] : 0u);
        has |= (sa.in[r].k > lily::SPL_SMALL_K && a.cand_out == nullptr ? lily::HAS_WIDE : 0u) |
               (sa.in[r].flags & lily::ROW_RAISES ? lily::HAS_RAISES : 0u);
    }
    if (slots != nullptr) {
        std::memcpy(sa.slots, slots, sizeof(uint32_t) * rows);
    }
    return launch_split(h, stream, sa, p, has, grid_rows ? grid_rows : rows, dtype);
}

// The argument block that holds the rows' parameters.
int32_t launch_rows_inline(lily_sampler *h, cudaStream_t stream, const lily::KArgs &a, const SplitPlan &p, uint32_t rows,
                           uint32_t dtype, const lily_sampling_params_t *params, const uint32_t *steps,
                           const uint32_t *slots) {
    return rows <= INLINE_ROWS ? launch_split_inline<INLINE_ROWS>(h, stream, a, p, rows, dtype, params, steps, slots)
           : rows <= INLINE_ROWS_MID
               ? launch_split_inline<INLINE_ROWS_MID>(h, stream, a, p, rows, dtype, params, steps, slots)
               : launch_split_inline<INLINE_ROWS_MAX>(h, stream, a, p, rows, dtype, params, steps, slots);
}

int32_t launch(lily_sampler *h, cudaStream_t stream, const lily::KArgs &a, uint32_t rows,
               uint32_t dtype) {
    const size_t smem = smem_bytes(a.vocab, a.n_slices);
    if (smem > (size_t)h->max_smem) {
        return fail(h, LILY_ERR_CAPACITY, "vocabulary too large for the shared-memory bitmap");
    }
    // (Parameters on the device: their penalties are not known here.)
    const SplitPlan plan = split_plan(h, a, rows, dtype,
                                      (a.history_ids != nullptr && a.count_slots == nullptr) || a.extra_len != 0u ||
                                          a.bias_ids != nullptr || a.ban_ids != nullptr,
                                      !a.force_greedy);
    if (plan.take) {
        lily::SplitArgs<INLINE_ROWS> sa;
        sa.a = a;
        sa.inline_params = sa.inline_slots = sa.inline_history = 0;
        const bool plain = a.cand_out == nullptr && a.spec.n_spec == 0u && a.bias_ids == nullptr && a.ban_ids == nullptr;
        return launch_split(h, stream, sa, plan, !plain ? lily::HAS_ALL : a.force_greedy ? lily::HAS_ARGMAX : lily::HAS_UNKNOWN, rows,
                            dtype);
    }
    const size_t esize = dtype == LILY_F32 ? 4 : 2;
    const bool vec = (reinterpret_cast<uintptr_t>(a.logits) % 16u == 0u) &&
                     ((a.logits_ld * esize) % 16u == 0u);
    if (dtype == LILY_F32) {
        return vec ? launch_one<float, true>(h, stream, a, rows, smem)
                   : launch_one<float, false>(h, stream, a, rows, smem);
    }
    return vec ? launch_one<__nv_bfloat16, true>(h, stream, a, rows, smem)
               : launch_one<__nv_bfloat16, false>(h, stream, a, rows, smem);
}

// Every kernel that the handle's calls can come to is on the device, with its shared-memory limit raised, before the
// first of them: which one a call takes depends on what its rows bring, and loading it there (an allocation on
// the device) would hold up one step in the middle of serving, or fall into a capture. (Not the LM head's: its
// first call loads them.)
cudaError_t load_kernels(const lily_sampler *h) {
    cudaError_t e = lily::split_ready(h->max_rows, (uint32_t)h->sm_count, h->max_smem);
    if (e == cudaSuccess) {
        e = lily::merge_ready();
    }
    for (uint32_t log_blocks = 1; log_blocks <= 3u; ++log_blocks) {
        lily::split_rows_at_once(h->device, h->sm_count, h->max_smem, log_blocks);  // (asked of the device once)
    }
    auto load = [&](auto kernel, int smem) {
        cudaFuncAttributes fa;
        if (e == cudaSuccess) {
            e = cudaFuncGetAttributes(&fa, kernel);  // (this loads it)
        }
        if (e == cudaSuccess && smem != 0) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        }
    };
    auto of_type = [&](auto logit) {
        using T = decltype(logit);
        load(lily::sample_rows_kernel<T, true>, h->max_smem);
        load(lily::sample_rows_kernel<T, false>, h->max_smem);
        if (h->max_rows >= lily::STREAM_MIN_ROWS) {
            load(lily::stream_rows_kernel<T, 3, true>, h->max_smem);
            load(lily::stream_rows_kernel<T, 3, false>, h->max_smem);
        }
        if (h->max_rows > (uint32_t)h->sm_count) {
            load(lily::stream_rows_kernel<T, 2, true>, h->max_smem);
            load(lily::stream_rows_kernel<T, 2, false>, h->max_smem);
        }
        load(lily::shard_sums_kernel<T>, 0);
    };
    of_type(0.0f);
    of_type(__nv_bfloat16());
    load(put_kernel<4096>, 0);
    load(put_kernel<16384>, 0);
    load(put_kernel<32000>, 0);
    load(lily::spec_accept_kernel, 0);
    load(lily::shard_publish_kernel, 0);
    if (h->flags & LILY_FLAG_COUNTS_TABLE) {
        load(lily::uncount_kernel, 0);
        load(lily::rebuild_seen_kernel, 0);
    }
    return e;
}

uint32_t choose_slices(const lily_sampler *h, uint32_t rows) {
    const uint32_t target = 2u * (uint32_t)h->sm_count;
    uint32_t s = target / rows;
    if (s < 1u) {
        s = 1u;
    }
    if (s > lily::MAX_SLICES) {
        s = lily::MAX_SLICES;
    }
    // Short slices cost more in merging than they save.
    const uint32_t by_len = (h->vocab + lily::MIN_SLICE - 1u) / lily::MIN_SLICE;
    if (s > by_len) {
        s = by_len;
    }
    return s < 1u ? 1u : s;
}

void base_args(const lily_sampler *h, lily::KArgs *a) {
    std::memset(a, 0, sizeof(*a));
    a->vocab = h->vocab;
    a->counts_table = h->counts_table;
    a->seen_table = h->seen_table;
    a->seen_words = h->seen_words;
    a->counts_scratch = h->counts_scratch;
    a->max_history = h->max_history;
    a->max_list = h->max_list;
    a->part = h->part;
    a->part_n = h->part_n;
    a->tickets = h->tickets;
    a->status_word = h->status_word;
    a->phase_clocks = h->phase_clocks;
}

int32_t check_handle(lily_sampler *h) {
    if (h == nullptr) {
        return LILY_ERR_ARG;
    }
    if (h->fault != 0) {
        return fail(h, LILY_ERR_FAULT, "a fault is latched on this sampler");
    }
    return LILY_OK;
}

}  // namespace

extern "C" {

uint32_t lily_abi_version(void) { return LILY_ABI_VERSION; }

int32_t lily_params_validate(const lily_sampling_params_t *p) {
    if (p == nullptr) {
        return LILY_ERR_ARG;
    }
    return params_ok(*p) ? LILY_OK : LILY_ERR_PARAMS;
}

int32_t lily_params_is_greedy(const lily_sampling_params_t *p) { return p && is_greedy(*p); }

int32_t lily_params_uses_penalties(const lily_sampling_params_t *p) {
    return p && uses_penalties(*p);
}

void lily_params_effective(const lily_sampling_params_t *p, float *temperature, uint32_t *top_k) {
    if (p == nullptr) {
        return;
    }
    if (temperature) {
        *temperature = is_greedy(*p) ? 1.0f : p->temperature;
    }
    if (top_k) {
        *top_k = effective_k(*p);
    }
}

void lily_draft_params(const lily_sampling_params_t *p, lily_sampling_params_t *out) {
    if (p == nullptr || out == nullptr) {
        return;
    }
    *out = *p;
    out->presence_penalty = 0.0f;
    out->frequency_penalty = 0.0f;
    out->repetition_penalty = 1.0f;
}

float lily_uniform_for(uint64_t seed, uint32_t step) { return lily::uniform_for(seed, step); }

uint32_t lily_draft_step(uint32_t step) { return step | 0x40000000u; }

uint32_t lily_residual_step(uint32_t step) { return step | 0x80000000u; }

int32_t lily_sampler_create(int32_t device, uint32_t vocab, uint32_t max_rows,
                            uint32_t max_history, uint32_t max_list, uint32_t flags,
                            lily_sampler_t **out) {
    if (out == nullptr || vocab == 0u || max_rows == 0u || max_list > 512u ||
        vocab > (1u << 24)) {
        return LILY_ERR_ARG;
    }
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) {
        return LILY_ERR_CUDA;
    }
    DeviceGuard guard(device);
    if (!guard.ok) {
        return LILY_ERR_CUDA;
    }
    lily_sampler *h = new (std::nothrow) lily_sampler();
    if (h == nullptr) {
        return LILY_ERR_ARG;
    }
    h->device = device;
    h->vocab = vocab;
    h->max_rows = max_rows;
    h->max_history = max_history;
    h->max_list = max_list;
    h->flags = flags;
    h->seen_words = (vocab + 31u) / 32u;
    h->layout = stage_layout(max_rows);
    auto bail = [&](cudaError_t e, const char *what) {
        std::fprintf(stderr, "lily_sampler_create: %s: %s\n", what, cudaGetErrorString(e));
        lily_sampler_destroy(h);
        return (int32_t)LILY_ERR_CUDA;
    };
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, device)) !=
        cudaSuccess) {
        return bail(e, "sm count");
    }
    if ((e = cudaDeviceGetAttribute(&h->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                    device)) != cudaSuccess) {
        return bail(e, "shared memory limit");
    }
    if ((e = load_kernels(h)) != cudaSuccess) {
        return bail(e, "kernels");
    }
    // One device allocation, one pinned one: an allocation takes some 0.3 ms, whatever
    // its size. What has to start from zero comes first, cleared by one call.
    size_t bytes = 0, cleared = 0;
    h->lm_ld = ((uint64_t)vocab + 3u) & ~uint64_t(3);
    h->lm_tokens = lily_head::padded_tokens(max_rows < lily_head::TOK ? max_rows : lily_head::TOK);
    for (int pass = 0; pass < 2; ++pass) {  // sizes, then addresses
        if (pass == 1) {
            if ((e = cudaMalloc(&h->arena, bytes)) != cudaSuccess || (e = cudaMemset(h->arena, 0, cleared)) != cudaSuccess) {
                return bail(e, "device workspaces");
            }
        }
        size_t at = 0;
        auto place = [&](auto *&p, size_t n) {
            if (pass == 1) {
                p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(h->arena + at);
            }
            at += (n + 255u) & ~size_t(255);
        };
        place(h->status_word, 4);
        place(h->tickets, (size_t)max_rows * 4);
        if (max_history > 0u) {
            // A row with a frequency penalty over a history LIST counts the list's ids
            // into this table and clears it again before the launch ends: all zero
            // between launches. Made here, never inside a draw.
            place(h->counts_scratch, (size_t)max_rows * vocab * sizeof(uint32_t));
        }
        if (flags & LILY_FLAG_COUNTS_TABLE) {
            place(h->counts_table, (size_t)max_rows * vocab * 4);
            place(h->seen_table, (size_t)max_rows * h->seen_words * 4);
        }
        if (flags & LILY_FLAG_PHASE_CLOCKS) {
            place(h->phase_clocks, (size_t)max_rows * LILY_MAX_SLICES * LILY_PHASES * sizeof(long long));
        }
        cleared = at;
        place(h->part, (size_t)max_rows * lily::CAP * sizeof(uint2));
        place(h->part_n, (size_t)max_rows * lily::MAX_SLICES * 4);
        // (Here, and not by the first head call: an allocation took that 1.2 to 2.3 ms.)
        place(h->lm_prepared, lily_head::prepared_bytes(h->lm_tokens));
        place(h->lm_flags, lily_head::flag_bytes((uint32_t)h->sm_count));
        if (flags & LILY_FLAG_LMHEAD) {
            place(h->lm_logits, (size_t)lily_head::TOK * h->lm_ld * sizeof(float));
        }
        for (int i = 0; i < RING; ++i) {
            place(h->d_stage[i], h->layout.total);
        }
        bytes = at;
    }
    if ((e = cudaMallocHost(&h->h_status, 256 + RING * h->layout.total)) != cudaSuccess) {
        return bail(e, "pinned workspaces");
    }
    for (int i = 0; i < RING; ++i) {
        h->h_stage[i] = reinterpret_cast<char *>(h->h_status) + 256 + i * h->layout.total;
        if ((e = cudaEventCreateWithFlags(&h->ev[i], cudaEventDisableTiming)) != cudaSuccess) {
            return bail(e, "staging ring");
        }
    }
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) {
        return bail(e, "create");
    }
    *out = h;
    return LILY_OK;
}

void lily_sampler_destroy(lily_sampler_t *h) {
    if (h == nullptr) {
        return;
    }
    DeviceGuard guard(h->device);
    cudaDeviceSynchronize();
    cudaFree(h->arena);
    cudaFree(h->lm_more);
    if (h->h_status) {
        cudaFreeHost(h->h_status);
    }
    for (int i = 0; i < RING; ++i) {
        if (h->ev[i]) {
            cudaEventDestroy(h->ev[i]);
        }
    }
    delete h;
}

uint32_t lily_sampler_vocab(const lily_sampler_t *h) { return h ? h->vocab : 0u; }

const char *lily_sampler_last_error(const lily_sampler_t *h) {
    return h ? h->last_error.c_str() : "null sampler";
}

void lily_sampler_inject_fault(lily_sampler_t *h, int32_t code) {
    if (h) {
        h->fault = code;
    }
}

void lily_sampler_clear_fault(lily_sampler_t *h) {
    if (h) {
        h->fault = 0;
    }
}

int32_t lily_sampler_set_wait_limit(lily_sampler_t *h, uint64_t nanoseconds) {
    if (h == nullptr) {
        return LILY_ERR_ARG;
    }
    h->wait_ns = nanoseconds == 0 ? 1000000000ull : nanoseconds;
    return LILY_OK;
}

void lily_sampler_inject_lost_copy(lily_sampler_t *h, uint32_t stage) {
    if (h) {
        h->lost_stage = stage;
    }
}

void lily_sampler_inject_lost_arrival(lily_sampler_t *h, uint32_t barrier, uint32_t block) {
    if (h) {
        h->lost_arrival = barrier ? (block << 8) | (barrier & 255u) : 0u;
    }
}

int32_t lily_sampler_status(lily_sampler_t *h, void *stream_) {
    if (h == nullptr) {
        return LILY_ERR_ARG;
    }
    if (h->fault != 0) {
        return fail(h, LILY_ERR_FAULT, "a fault is latched on this sampler");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    CU(h, cudaMemcpyAsync(h->h_status, h->status_word, 4, cudaMemcpyDeviceToHost, stream));
    CU(h, cudaMemsetAsync(h->status_word, 0, 4, stream));
    CU(h, cudaStreamSynchronize(stream));
    if (*h->h_status & (1u << lily_head::STATUS_TIMEOUT_BIT)) {
        return fail(h, LILY_ERR_TIMEOUT,
                    "a bounded wait ran out (inside a kernel, or for a peer's records): the results are not valid");
    }
    if (*h->h_status != 0u) {
        char buf[96];
        std::snprintf(buf, sizeof buf, "rows reported error bits 0x%x", *h->h_status);
        return fail(h, LILY_ERR_DEVICE_ROW, buf);
    }
    return LILY_OK;
}

// ------------------------------------------------------------- histogram --

int32_t lily_sampler_reset_counts(lily_sampler_t *h, void *stream_, uint32_t slot) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (h->counts_table == nullptr || slot >= h->max_rows) {
        return fail(h, LILY_ERR_ARG, "no such histogram slot");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    CU(h, cudaMemsetAsync(h->counts_table + (size_t)slot * h->vocab, 0, (size_t)h->vocab * 4,
                          stream));
    CU(h, cudaMemsetAsync(h->seen_table + (size_t)slot * h->seen_words, 0,
                          (size_t)h->seen_words * 4, stream));
    return LILY_OK;
}

int32_t lily_sampler_uncount(lily_sampler_t *h, void *stream_, uint32_t slot, uint32_t token) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (h->counts_table == nullptr || slot >= h->max_rows) {
        return fail(h, LILY_ERR_ARG, "no such histogram slot");
    }
    if (token >= h->vocab) {
        return LILY_OK;  // src/kernels/sample.rs:148-151: out of range is ignored
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    lily::uncount_kernel<<<1, 1, 0, stream>>>(h->counts_table + (size_t)slot * h->vocab,
                                              h->seen_table + (size_t)slot * h->seen_words,
                                              h->vocab, token);
    CU(h, cudaGetLastError());
    return LILY_OK;
}

int32_t lily_sampler_copy_counts(lily_sampler_t *dst, uint32_t dst_slot, const lily_sampler_t *src,
                                 uint32_t src_slot, void *stream_) {
    int32_t st = check_handle(dst);
    if (st != LILY_OK) {
        return st;
    }
    if (src == nullptr || dst->counts_table == nullptr || src->counts_table == nullptr ||
        dst_slot >= dst->max_rows || src_slot >= src->max_rows) {
        return fail(dst, LILY_ERR_ARG, "no such histogram slot");
    }
    if (src->vocab != dst->vocab) {
        return fail(dst, LILY_ERR_VOCAB, "sampler scratches for different vocabularies");
    }
    DeviceGuard guard(dst->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    CU(dst, cudaMemcpyAsync(dst->counts_table + (size_t)dst_slot * dst->vocab,
                            src->counts_table + (size_t)src_slot * src->vocab,
                            (size_t)dst->vocab * 4, cudaMemcpyDefault, stream));
    CU(dst, cudaMemcpyAsync(dst->seen_table + (size_t)dst_slot * dst->seen_words,
                            src->seen_table + (size_t)src_slot * src->seen_words,
                            (size_t)dst->seen_words * 4, cudaMemcpyDefault, stream));
    return LILY_OK;
}

// include/lily_batch.h: CountsSlot::Engine is the engine handle's slot 0,
// CountsSlot::Batch(i) slot i of the batch handle.
int32_t lily_move_counts(lily_sampler_t *engine, lily_sampler_t *batch, void *stream_,
                         uint32_t from, uint32_t to) {
    if (from == to) {
        return LILY_OK;
    }
    int32_t st = check_handle(engine);
    if (st != LILY_OK) {
        return st;
    }
    st = check_handle(batch);
    if (st != LILY_OK) {
        return st;
    }
    for (uint32_t slot : {from, to}) {
        if (slot != LILY_COUNTS_ENGINE && slot >= batch->max_rows) {
            std::string msg = "batch slot " + std::to_string(slot) + " of " +
                              std::to_string(batch->max_rows);
            fail(engine, LILY_ERR_ARG, msg.c_str());
            return fail(batch, LILY_ERR_ARG, msg.c_str());
        }
    }
    lily_sampler_t *src = from == LILY_COUNTS_ENGINE ? engine : batch;
    lily_sampler_t *dst = to == LILY_COUNTS_ENGINE ? engine : batch;
    return lily_sampler_copy_counts(dst, to == LILY_COUNTS_ENGINE ? 0u : to, src,
                                    from == LILY_COUNTS_ENGINE ? 0u : from, stream_);
}

int32_t lily_sampler_read_counts(lily_sampler_t *h, void *stream_, uint32_t slot,
                                 uint32_t *host_out) {
    if (h == nullptr || host_out == nullptr || h->counts_table == nullptr ||
        slot >= h->max_rows) {
        return fail(h, LILY_ERR_ARG, "no such histogram slot");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    CU(h, cudaMemcpyAsync(host_out, h->counts_table + (size_t)slot * h->vocab,
                          (size_t)h->vocab * 4, cudaMemcpyDeviceToHost, stream));
    CU(h, cudaStreamSynchronize(stream));
    return LILY_OK;
}

int32_t lily_sampler_write_counts(lily_sampler_t *h, void *stream_, uint32_t slot,
                                  const uint32_t *host_in) {
    if (h == nullptr || host_in == nullptr || h->counts_table == nullptr ||
        slot >= h->max_rows) {
        return fail(h, LILY_ERR_ARG, "no such histogram slot");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    uint32_t *counts = h->counts_table + (size_t)slot * h->vocab;
    CU(h, cudaMemcpyAsync(counts, host_in, (size_t)h->vocab * 4, cudaMemcpyHostToDevice, stream));
    const uint32_t threads = 256, blocks = (h->seen_words + threads - 1u) / threads;
    lily::rebuild_seen_kernel<<<blocks, threads, 0, stream>>>(
        counts, h->seen_table + (size_t)slot * h->seen_words, h->vocab);
    CU(h, cudaGetLastError());
    CU(h, cudaStreamSynchronize(stream));
    return LILY_OK;
}

int32_t lily_sampler_read_phase_clocks(lily_sampler_t *h, void *stream_, int64_t *host_out) {
    if (h == nullptr || host_out == nullptr || h->phase_clocks == nullptr) {
        return fail(h, LILY_ERR_ARG, "the sampler was not created with LILY_FLAG_PHASE_CLOCKS");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    const size_t pb = (size_t)h->max_rows * LILY_MAX_SLICES * LILY_PHASES * sizeof(long long);
    CU(h, cudaMemcpyAsync(host_out, h->phase_clocks, pb, cudaMemcpyDeviceToHost, stream));
    CU(h, cudaMemsetAsync(h->phase_clocks, 0, pb, stream));
    CU(h, cudaStreamSynchronize(stream));
    return LILY_OK;
}

// ------------------------------------------------------------------ draw --

int32_t lily_sample_batch(lily_sampler_t *h, void *stream_, const lily_sample_args_t *args) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (args == nullptr || args->struct_size != sizeof(lily_sample_args_t)) {
        return fail(h, LILY_ERR_ARG, "args is null or of another ABI version");
    }
    const lily_sample_args_t &g = *args;
    if (g.rows == 0u || g.rows > h->max_rows) {
        return fail(h, LILY_ERR_CAPACITY, "rows outside 1..max_rows");
    }
    if (g.logits == nullptr || g.out_ids == nullptr || g.params == nullptr ||
        g.logits_ld < h->vocab || g.logits_dtype > LILY_BF16) {
        return fail(h, LILY_ERR_ARG, "logits must be F32 or BF16 [rows, ld >= vocab]; out and params set");
    }
    if (g.uniforms == nullptr && g.steps == nullptr) {
        return fail(h, LILY_ERR_ARG, "either uniforms or steps must be given");
    }
    if ((g.history_ids != nullptr) != (g.history_len != nullptr) ||
        (g.bias_ids != nullptr) != (g.bias_len != nullptr) ||
        (g.bias_ids != nullptr) != (g.bias_vals != nullptr) ||
        (g.ban_ids != nullptr) != (g.ban_len != nullptr)) {
        return fail(h, LILY_ERR_ARG, "a list needs both its ids and its lengths");
    }
    if (g.kept_n != nullptr &&
        (g.kept_ids == nullptr || g.kept_probs == nullptr || g.kept_ld < LILY_K_CAP)) {
        return fail(h, LILY_ERR_ARG, "kept_n needs kept_ids, kept_probs and kept_ld >= 1024");
    }
    if (g.count_slots != nullptr && h->counts_table == nullptr) {
        return fail(h, LILY_ERR_ARG, "count_slots needs LILY_FLAG_COUNTS_TABLE");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);

    lily::KArgs a;
    base_args(h, &a);
    const lily_sampling_params_t *d_params = g.params;
    const uint32_t *d_steps = g.steps;
    const uint32_t *d_slots = nullptr;
    int slot = -1;
    a.logits = g.logits;
    a.logits_ld = g.logits_ld;
    a.rows = g.rows;
    // Host parameters (and slots) of up to INLINE_ROWS_MAX rows travel in the
    // kernel's own arguments: nothing is staged, no copy sits in front of the launch.
    SplitPlan plan;
    if (!g.params_on_device && g.rows <= INLINE_ROWS_MAX) {
        const bool history = g.history_ids != nullptr && g.count_slots == nullptr;
        bool counts = false;
        for (uint32_t r = 0; r < g.rows; ++r) {
            counts = counts || g.params[r].frequency_penalty != 0.0f;
        }
        plan = split_plan(h, a, g.rows, g.logits_dtype, history || g.bias_ids != nullptr || g.ban_ids != nullptr,
                          history && counts);
    }
    const StageLayout layout = stage_layout(g.rows);
    const bool in_args = plan.take;
    if (!in_args && (!g.params_on_device || g.count_slots != nullptr)) {
        st = next_stage(h, &slot);
        if (st != LILY_OK) {
            return st;
        }
    }
    if (!g.params_on_device) {
        for (uint32_t r = 0; r < g.rows; ++r) {
            if (!params_ok(g.params[r])) {
                char buf[64];
                std::snprintf(buf, sizeof buf, "row %u: invalid sampling parameters", r);
                return fail(h, LILY_ERR_PARAMS, buf);
            }
        }
    }
    if (g.count_slots != nullptr) {
        for (uint32_t r = 0; r < g.rows; ++r) {
            if (g.count_slots[r] >= h->max_rows) {
                return fail(h, LILY_ERR_ARG, "no such histogram slot");
            }
        }
    }
    if (!g.params_on_device && !in_args) {
        char *hs = h->h_stage[slot];
        std::memcpy(hs + layout.params, g.params, sizeof(lily_sampling_params_t) * g.rows);
        d_params = reinterpret_cast<const lily_sampling_params_t *>(h->d_stage[slot] +
                                                                    layout.params);
        if (g.steps != nullptr) {
            std::memcpy(hs + layout.steps, g.steps, sizeof(uint32_t) * g.rows);
            d_steps = reinterpret_cast<const uint32_t *>(h->d_stage[slot] + layout.steps);
        }
    }
    if (g.count_slots != nullptr && !in_args) {
        std::memcpy(h->h_stage[slot] + layout.slots, g.count_slots, sizeof(uint32_t) * g.rows);
        d_slots = reinterpret_cast<const uint32_t *>(h->d_stage[slot] + layout.slots);
    }
    if (slot >= 0) {
        if ((st = upload(h, slot, layout.total, stream)) != LILY_OK) {
            return st;
        }
    }
    a.params = d_params;
    a.uniforms = g.uniforms;
    a.steps = d_steps;
    a.history_ids = g.history_ids;
    a.history_len = g.history_len;
    a.history_ld = g.history_ld;
    a.bias_ids = g.bias_ids;
    a.bias_vals = g.bias_vals;
    a.bias_len = g.bias_len;
    a.bias_ld = g.bias_ld;
    a.ban_ids = g.ban_ids;
    a.ban_len = g.ban_len;
    a.ban_ld = g.ban_ld;
    a.forced_ids = g.forced_ids;
    a.count_slots = d_slots;
    a.out_ids = g.out_ids;
    a.out_status = g.out_status;
    a.kept_n = g.kept_n;
    a.kept_ids = g.kept_ids;
    a.kept_probs = g.kept_probs;
    a.kept_ld = g.kept_ld;
    a.n_slices = choose_slices(h, g.rows);
    if (in_args) {
        return launch_rows_inline(h, stream, a, plan, g.rows, g.logits_dtype, g.params, g.steps, g.count_slots);
    }
    st = launch(h, stream, a, g.rows, g.logits_dtype);
    if (slot >= 0) {
        CU(h, cudaEventRecord(h->ev[slot], stream));
    }
    return st;
}

int32_t lily_sample_one(lily_sampler_t *h, void *stream_, const void *logits, uint32_t logits_dtype,
                        uint64_t logits_len, const lily_sampling_params_t *params, uint32_t step,
                        const uint32_t *history_ids, uint32_t history_len, uint32_t *out_id) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (logits == nullptr || out_id == nullptr || params == nullptr || logits_len < h->vocab ||
        logits_dtype > LILY_BF16) {
        return fail(h, LILY_ERR_ARG, "logits must be F32 or BF16 [ld >= vocab]; out and params set");
    }
    if (history_len > 0u && history_ids == nullptr) {
        return fail(h, LILY_ERR_ARG, "history_len without history_ids");
    }
    if (!params_ok(*params)) {
        return fail(h, LILY_ERR_PARAMS, "row 0: invalid sampling parameters");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    lily::KArgs a;
    base_args(h, &a);
    a.logits = logits;
    a.logits_ld = logits_len;
    a.rows = 1;
    a.history_ids = history_ids;
    a.history_ld = history_len;
    a.out_ids = out_id;
    a.n_slices = choose_slices(h, 1u);
    const SplitPlan plan = split_plan(h, a, 1u, logits_dtype, history_ids != nullptr, params->frequency_penalty != 0.0f);
    if (plan.take) {
        return launch_split_inline<INLINE_ROWS>(h, stream, a, plan, 1u, logits_dtype, params, &step, nullptr,
                                                1u + history_len);
    }
    int slot = -1;
    st = next_stage(h, &slot);
    if (st != LILY_OK) {
        return st;
    }
    char *hs = h->h_stage[slot], *ds = h->d_stage[slot];
    const StageLayout layout = stage_layout(1u);
    std::memcpy(hs + layout.params, params, sizeof(*params));
    std::memcpy(hs + layout.steps, &step, 4);
    std::memcpy(hs + layout.hist_len, &history_len, 4);
    if ((st = upload(h, slot, layout.total, stream)) != LILY_OK) {
        return st;
    }
    a.params = reinterpret_cast<const lily_sampling_params_t *>(ds + layout.params);
    a.steps = reinterpret_cast<const uint32_t *>(ds + layout.steps);
    a.history_len = history_ids ? reinterpret_cast<const uint32_t *>(ds + layout.hist_len) : nullptr;
    st = launch(h, stream, a, 1u, logits_dtype);
    CU(h, cudaEventRecord(h->ev[slot], stream));
    return st;
}

int32_t lily_argmax_batch(lily_sampler_t *h, void *stream_, const void *logits,
                          uint32_t logits_dtype, uint64_t logits_ld, uint32_t rows,
                          uint32_t *out_ids) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (rows == 0u || rows > h->max_rows) {
        return fail(h, LILY_ERR_CAPACITY, "rows outside 1..max_rows");
    }
    if (logits == nullptr || out_ids == nullptr || logits_ld < h->vocab ||
        logits_dtype > LILY_BF16) {
        return fail(h, LILY_ERR_ARG, "logits must be F32 or BF16 [rows, ld >= vocab]");
    }
    DeviceGuard guard(h->device);
    lily::KArgs a;
    base_args(h, &a);
    a.logits = logits;
    a.logits_ld = logits_ld;
    a.rows = rows;
    a.force_greedy = 1;
    a.out_ids = out_ids;
    a.n_slices = choose_slices(h, rows);
    return launch(h, static_cast<cudaStream_t>(stream_), a, rows, logits_dtype);
}

// ------------------------------------------------ LM head, vocab shards --

namespace {

// cuTensorMapEncodeTiled through the runtime's entry-point query: the library
// does not link against the driver.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn tensor_map_encoder() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &res) == cudaSuccess &&
            res == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
        }
    }
    return fn;
}

int32_t lmhead_launch(lily_sampler *h, cudaStream_t stream, const lily_lmhead_t *head,
                      const void *hidden, uint64_t hidden_ld, uint32_t tokens, float *out,
                      uint64_t out_ld) {
    if (head == nullptr || head->struct_size != sizeof(lily_lmhead_t)) {
        return fail(h, LILY_ERR_ARG, "head is null or of another ABI version");
    }
    if (head->weights == nullptr || head->scales_bf16 == nullptr || hidden == nullptr || out == nullptr) {
        return fail(h, LILY_ERR_ARG, "weights, scales, hidden and out must be set");
    }
    if (head->group != (uint32_t)lily_head::GROUP_K || head->hidden == 0u || head->hidden % 512u != 0u) {
        return fail(h, LILY_ERR_ARG, "group must be 64 and hidden a multiple of 512");
    }
    if (tokens == 0u || tokens > (uint32_t)lily_head::TOK) {
        return fail(h, LILY_ERR_CAPACITY, "tokens outside 1..64");
    }
    if (head->rows == 0u || out_ld < head->rows || hidden_ld < head->hidden) {
        return fail(h, LILY_ERR_ARG, "out_ld < rows or hidden_ld < hidden");
    }
    if (reinterpret_cast<uintptr_t>(head->weights) % 16u || reinterpret_cast<uintptr_t>(head->scales_bf16) % 16u ||
        reinterpret_cast<uintptr_t>(head->biases_bf16) % 16u || reinterpret_cast<uintptr_t>(hidden) % 16u ||
        (hidden_ld * 2u) % 16u) {
        return fail(h, LILY_ERR_ARG, "weights, scales, biases and hidden rows must be 16-byte aligned");
    }
    const bool affine = head->biases_bf16 != nullptr;
    if (affine && head->hidden > lily_head::CHUNK_K) {
        return fail(h, LILY_ERR_CAPACITY, "an affine head takes a hidden size of at most 8192");
    }
    if (head->code_bits != 0u && head->code_bits != 8u && head->code_bits != 4u) {
        return fail(h, LILY_ERR_ARG, "code_bits must be 0, 8 or 4");
    }
    const bool q4 = head->code_bits == 4u;
    if (q4 && !affine) {
        return fail(h, LILY_ERR_ARG, "4-bit codes are the affine storage: biases must be set");
    }
    EncodeTiledFn encode = tensor_map_encoder();
    if (encode == nullptr) {
        return fail(h, LILY_ERR_CUDA, "the driver does not offer cuTensorMapEncodeTiled");
    }
    lily_head::Args a;
    {
        // Weights: uint8 [rows, hidden] (4-bit codes: [rows, hidden / 2]), boxes of 256 rows x
        // 128 bytes, fetched 256 bytes at a time: the next box along the row finds its half in
        // L2 (262144 x 4096, 16 tokens: 214 us with promotion to 128 bytes, 190 with this).
        const cuuint64_t row_bytes = q4 ? head->hidden / 2u : head->hidden;
        const cuuint64_t dims[2] = {row_bytes, head->rows};
        const cuuint64_t strides[1] = {row_bytes};
        const cuuint32_t box[2] = {128, (cuuint32_t)lily_head::TILE_ROWS};
        const cuuint32_t estr[2] = {1, 1};
        if (encode(&a.w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(head->weights), dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
            return fail(h, LILY_ERR_CUDA, "cuTensorMapEncodeTiled refused the weights");
        }
    }
    const lily_head::Format format = q4 ? lily_head::FMT_U4 : affine ? lily_head::FMT_U8 : lily_head::FMT_S8;
    a.scale_ld = head->hidden / lily_head::GROUP_K;
    a.tokens = tokens;
    a.rows = head->rows;
    a.out = out;
    a.ldo = out_ld;
    const uint32_t padded = lily_head::padded_tokens(tokens);
    const size_t prepared = (lily_head::prepared_bytes(lily_head::TOK) + 255u) & ~size_t(255);
    if ((padded > h->lm_tokens || head->hidden > lily_head::CHUNK_K) && h->lm_more == nullptr) {
        // (The stream may be under capture: the allocation is no part of the graph.)
        char *at = nullptr;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CU(h, cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t e = cudaMalloc(&at, prepared + lily_head::part_bytes((uint32_t)h->sm_count));
        CU(h, cudaThreadExchangeStreamCaptureMode(&mode));
        CU(h, e);
        h->lm_more = at;
    }
    a.prep = lily_head::prepared_at(padded > h->lm_tokens ? h->lm_more : h->lm_prepared, padded);
    a.flags = h->lm_flags;
    a.status_word = h->status_word;
    a.wait_ns = h->wait_ns;
    a.lost_stage = h->lost_stage;
    h->lost_stage = 0xFFFFFFFFu;  // one launch only
    for (uint32_t k0 = 0; k0 < head->hidden; k0 += lily_head::CHUNK_K) {
        const uint32_t columns = head->hidden - k0 < lily_head::CHUNK_K ? head->hidden - k0 : lily_head::CHUNK_K;
        a.groups = columns / lily_head::GROUP_K;
        a.byte0 = q4 ? k0 / 2u : k0;
        a.scales = static_cast<const __nv_bfloat16 *>(head->scales_bf16) + k0 / lily_head::GROUP_K;
        a.biases = affine ? static_cast<const __nv_bfloat16 *>(head->biases_bf16) + k0 / lily_head::GROUP_K : nullptr;
        a.accumulate = k0 != 0u ? 1u : 0u;
        a.part = k0 != 0u ? reinterpret_cast<float *>(h->lm_more + prepared) : nullptr;
        CU(h, lily_head::launch_prepare(a.prep, static_cast<const __nv_bfloat16 *>(hidden) + k0, hidden_ld, tokens,
                                        a.groups, format, a.flags, (uint32_t)h->sm_count, stream));
        CU(h, lily_head::launch_head(a, format, (uint32_t)h->sm_count, stream));
        a.lost_stage = 0xFFFFFFFFu;
    }
    return LILY_OK;
}

// The host parameters of a sharded call, checked.
int32_t check_shard_params(lily_sampler *h, const lily_sample_args_t &g) {
    if (g.rows == 0u || g.rows > h->max_rows) {
        return fail(h, LILY_ERR_CAPACITY, "rows outside 1..max_rows");
    }
    if (g.params == nullptr || g.params_on_device) {
        return fail(h, LILY_ERR_ARG, "sharded calls take host params");
    }
    if (g.history_ids || g.history_len || g.bias_ids || g.bias_vals || g.bias_len || g.ban_ids ||
        g.ban_len || g.forced_ids || g.count_slots) {
        return fail(h, LILY_ERR_ARG, "no penalties state, lists or forced ids in sharded calls");
    }
    for (uint32_t r = 0; r < g.rows; ++r) {
        const lily_sampling_params_t &p = g.params[r];
        if (!params_ok(p)) {
            return fail(h, LILY_ERR_PARAMS, "invalid sampling parameters");
        }
        if (uses_penalties(p)) {
            return fail(h, LILY_ERR_ARG, "no penalties in sharded calls");
        }
        if (!is_greedy(p) && (p.top_k == 0u || p.top_k > LILY_SHARD_CANDIDATES)) {
            return fail(h, LILY_ERR_ARG, "sharded sampling needs 1 <= top_k <= 64");
        }
    }
    return LILY_OK;
}

// Stages them to the device, for a call of more rows than a launch's own arguments take.
int32_t stage_shard_params(lily_sampler *h, cudaStream_t stream, const lily_sample_args_t &g,
                           const lily_sampling_params_t **d_params, const uint32_t **d_steps,
                           int *slot_out) {
    const StageLayout layout = stage_layout(g.rows);
    // What would be staged: [rows][has steps][params][steps].
    const size_t pb = sizeof(lily_sampling_params_t) * g.rows, sb = g.steps ? sizeof(uint32_t) * g.rows : 0;
    std::vector<char> want(8 + pb + sb);
    const uint32_t head[2] = {g.rows, g.steps != nullptr ? 1u : 0u};
    std::memcpy(want.data(), head, 8);
    std::memcpy(want.data() + 8, g.params, pb);
    if (sb) {
        std::memcpy(want.data() + 8 + pb, g.steps, sb);
    }
    int slot = h->shard_slot;
    const bool reuse = slot >= 0 && h->slot_serial[slot] == h->shard_serial && want == h->shard_bytes;
    if (!reuse) {
        int32_t st = next_stage(h, &slot);
        if (st != LILY_OK) {
            return st;
        }
        char *hs = h->h_stage[slot];
        std::memcpy(hs + layout.params, g.params, pb);
        if (sb) {
            std::memcpy(hs + layout.steps, g.steps, sb);
        }
        if ((st = upload(h, slot, layout.total, stream)) != LILY_OK) {
            return st;
        }
        h->shard_slot = slot;
        h->shard_serial = h->slot_serial[slot];
        h->shard_bytes.swap(want);
    }
    // (A reused slot is read by one more launch: the caller records the slot's
    // event after it, so the ring does not overwrite the slot under that launch.)
    *d_params = reinterpret_cast<const lily_sampling_params_t *>(h->d_stage[slot] + layout.params);
    *d_steps = g.steps != nullptr ? reinterpret_cast<const uint32_t *>(h->d_stage[slot] + layout.steps) : nullptr;
    *slot_out = slot;
    return LILY_OK;
}

int32_t shard_candidates(lily_sampler *h, cudaStream_t stream, const lily_sample_args_t &g,
                         uint32_t first_id, int32_t want_sums, void *records) {
    if (g.logits == nullptr || records == nullptr || g.logits_ld < h->vocab || g.logits_dtype > LILY_BF16) {
        return fail(h, LILY_ERR_ARG, "logits must be F32 or BF16 [rows, ld >= vocab]; records set");
    }
    if ((uint64_t)first_id + h->vocab > 0xFFFFFFFFull) {
        return fail(h, LILY_ERR_ARG, "first_id + vocab overflows an id");
    }
    int32_t st = check_shard_params(h, g);
    if (st != LILY_OK) {
        return st;
    }
    lily::KArgs a;
    base_args(h, &a);
    a.logits = g.logits;
    a.logits_ld = g.logits_ld;
    a.rows = g.rows;
    a.out_ids = nullptr;
    a.shard_k = LILY_SHARD_CANDIDATES;
    a.id_offset = first_id;
    a.cand_out = static_cast<lily::ShardRecord *>(records);
    const SplitPlan plan = split_plan(h, a, g.rows, g.logits_dtype, false, false);
    if (plan.take) {  // (the row kernel sums the exponentials in the same launch)
        a.shard_sums = want_sums ? 1u : 0u;
    }
    if (plan.take && g.rows <= INLINE_ROWS_MAX) {
        return launch_rows_inline(h, stream, a, plan, g.rows, g.logits_dtype, g.params, nullptr, nullptr);
    }
    const uint32_t *d_steps = nullptr;
    int slot = -1;
    st = stage_shard_params(h, stream, g, &a.params, &d_steps, &slot);
    if (st != LILY_OK) {
        return st;
    }
    const lily_sampling_params_t *d_params = a.params;
    a.n_slices = choose_slices(h, g.rows);
    // (The kernel of one block per row sums the exponentials in the same pass.)
    a.shard_sums = want_sums && (plan.take || stream_route(a, g.rows, g.logits_dtype)) ? 1u : 0u;
    st = launch(h, stream, a, g.rows, g.logits_dtype);
    if (st == LILY_OK && want_sums && a.shard_sums == 0u) {
        // The candidate launch has left the slice counters and the tickets (all
        // zero again) free: the sums use them for their pieces.
        uint32_t pieces = (2u * (uint32_t)h->sm_count + g.rows - 1u) / g.rows;
        const uint32_t by_len = (h->vocab + 8191u) / 8192u;
        pieces = pieces > by_len ? by_len : pieces;
        pieces = pieces < 1u ? 1u : (pieces > lily::MAX_SLICES ? lily::MAX_SLICES : pieces);
        const dim3 grid(pieces, g.rows, 1);
        float *scratch = reinterpret_cast<float *>(h->part_n);
        if (g.logits_dtype == LILY_F32) {
            lily::shard_sums_kernel<float><<<grid, 1024, 0, stream>>>(
                static_cast<const float *>(g.logits), g.logits_ld, h->vocab, d_params, a.cand_out, scratch,
                h->tickets);
        } else {
            lily::shard_sums_kernel<__nv_bfloat16><<<grid, 1024, 0, stream>>>(
                static_cast<const __nv_bfloat16 *>(g.logits), g.logits_ld, h->vocab, d_params, a.cand_out,
                scratch, h->tickets);
        }
        CU(h, cudaGetLastError());
    }
    CU(h, cudaEventRecord(h->ev[slot], stream));
    return st;
}

}  // namespace

int32_t lily_lmhead_logits(lily_sampler_t *h, void *stream_, const lily_lmhead_t *head,
                           const void *hidden_bf16, uint64_t hidden_ld, uint32_t tokens,
                           float *out_logits, uint64_t out_ld) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    DeviceGuard guard(h->device);
    return lmhead_launch(h, static_cast<cudaStream_t>(stream_), head, hidden_bf16, hidden_ld, tokens,
                         out_logits, out_ld);
}

int32_t lily_shard_candidates(lily_sampler_t *h, void *stream_, const lily_sample_args_t *args,
                              uint32_t first_id, int32_t want_sums, void *records) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (args == nullptr || args->struct_size != sizeof(lily_sample_args_t)) {
        return fail(h, LILY_ERR_ARG, "args is null or of another ABI version");
    }
    DeviceGuard guard(h->device);
    return shard_candidates(h, static_cast<cudaStream_t>(stream_), *args, first_id, want_sums, records);
}

int32_t lily_lmhead_shard_candidates(lily_sampler_t *h, void *stream_, const lily_lmhead_t *head,
                                     const void *hidden_bf16, uint64_t hidden_ld,
                                     const lily_sample_args_t *args, uint32_t first_id,
                                     int32_t want_sums, void *records) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (args == nullptr || args->struct_size != sizeof(lily_sample_args_t)) {
        return fail(h, LILY_ERR_ARG, "args is null or of another ABI version");
    }
    if (h->lm_logits == nullptr) {
        return fail(h, LILY_ERR_ARG, "the sampler was not created with LILY_FLAG_LMHEAD");
    }
    if (head == nullptr || head->rows != h->vocab) {
        return fail(h, LILY_ERR_VOCAB, "the head's rows must equal the sampler's vocabulary");
    }
    if (args->logits != nullptr) {
        return fail(h, LILY_ERR_ARG, "the logits come from the head: args->logits must be NULL");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    st = lmhead_launch(h, stream, head, hidden_bf16, hidden_ld, args->rows, h->lm_logits, h->lm_ld);
    if (st != LILY_OK) {
        return st;
    }
    lily_sample_args_t g = *args;
    g.logits = h->lm_logits;
    g.logits_dtype = LILY_F32;
    g.logits_ld = h->lm_ld;
    return shard_candidates(h, stream, g, first_id, want_sums, records);
}

namespace {
int32_t merge_draw(lily_sampler_t *h, void *stream_, const void *gathered, uint32_t n_shards,
                   uint64_t shard_stride, const lily_sample_args_t *args, float *out_lse,
                   const lily::KArgs::PeerLink *peer);

}  // namespace

int32_t lily_merge_draw(lily_sampler_t *h, void *stream_, const void *gathered, uint32_t n_shards,
                        uint64_t shard_stride, const lily_sample_args_t *args, float *out_lse) {
    return merge_draw(h, stream_, gathered, n_shards, shard_stride, args, out_lse, nullptr);
}

namespace {

int32_t merge_draw(lily_sampler_t *h, void *stream_, const void *gathered, uint32_t n_shards,
                   uint64_t shard_stride, const lily_sample_args_t *args, float *out_lse,
                   const lily::KArgs::PeerLink *peer) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (args == nullptr || args->struct_size != sizeof(lily_sample_args_t)) {
        return fail(h, LILY_ERR_ARG, "args is null or of another ABI version");
    }
    const lily_sample_args_t &g = *args;
    if (gathered == nullptr || n_shards == 0u || n_shards > 64u || shard_stride < g.rows ||
        g.out_ids == nullptr || g.logits != nullptr) {
        return fail(h, LILY_ERR_ARG, "records and out_ids set, 1..64 shards, stride >= rows, no logits");
    }
    if (g.uniforms == nullptr && g.steps == nullptr) {
        return fail(h, LILY_ERR_ARG, "either uniforms or steps must be given");
    }
    if (g.kept_n != nullptr &&
        (g.kept_ids == nullptr || g.kept_probs == nullptr || g.kept_ld < LILY_SHARD_CANDIDATES)) {
        return fail(h, LILY_ERR_ARG, "kept_n needs kept_ids, kept_probs and kept_ld >= 64");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    st = check_shard_params(h, g);
    if (st != LILY_OK) {
        return st;
    }
    lily::MergeArgs ma;
    const bool in_args = g.rows <= lily::INLINE_ROWS_MID;
    int slot = -1;
    const lily_sampling_params_t *d_params = nullptr;
    const uint32_t *d_steps = nullptr;
    if (in_args) {
        for (uint32_t r = 0; r < g.rows; ++r) {
            ma.in[r] = lily::row_in(g.params[r], g.steps != nullptr ? g.steps[r] : 0u);
        }
    } else if ((st = stage_shard_params(h, stream, g, &d_params, &d_steps, &slot)) != LILY_OK) {
        return st;
    }
    lily::KArgs &a = ma.a;
    base_args(h, &a);
    a.vocab = 0xFFFFFFFFu;  // ids are global here
    a.rows = g.rows;
    a.params = d_params;
    a.uniforms = g.uniforms;
    a.steps = d_steps;
    a.out_ids = g.out_ids;
    a.out_status = g.out_status;
    a.kept_n = g.kept_n;
    a.kept_ids = g.kept_ids;
    a.kept_probs = g.kept_probs;
    a.kept_ld = g.kept_ld;
    a.merge_in = static_cast<const lily::ShardRecord *>(gathered);
    a.merge_shards = n_shards;
    a.merge_stride = shard_stride;
    a.out_lse = out_lse;
    if (peer != nullptr) {
        a.peer = *peer;
    }
    CU(h, lily::merge_launch(ma, g.rows, stream));
    if (!in_args) {
        CU(h, cudaEventRecord(h->ev[slot], stream));
    }
    return LILY_OK;
}

}  // namespace

// ------------------------------------------------- records over peer memory --

namespace {

int32_t peer_check(lily_sampler *h, const lily_peer_exchange_t *x) {
    if (x == nullptr || x->struct_size != sizeof(lily_peer_exchange_t)) {
        return fail(h, LILY_ERR_ARG, "exchange is null or of another ABI version");
    }
    if (x->n_shards == 0u || x->n_shards > LILY_PEER_MAX || x->rank >= x->n_shards || x->max_rows == 0u) {
        return fail(h, LILY_ERR_ARG, "1..16 shards, rank below them, max_rows set");
    }
    for (uint32_t r = 0; r < x->n_shards; ++r) {
        if (x->buffers[r] == nullptr) {
            return fail(h, LILY_ERR_ARG, "every rank's buffer must be set");
        }
    }
    return LILY_OK;
}

}  // namespace

uint64_t lily_peer_buffer_bytes(uint32_t n_shards, uint32_t max_rows) {
    return (uint64_t)lily::peer_flag_bytes(n_shards, max_rows) +
           2ull * n_shards * max_rows * sizeof(lily::ShardRecord);
}

int32_t lily_peer_buffer_create(int32_t device, uint32_t n_shards, uint32_t max_rows, void **buffer,
                                void *ipc_handle) {
    if (buffer == nullptr || ipc_handle == nullptr || n_shards == 0u || n_shards > LILY_PEER_MAX ||
        max_rows == 0u) {
        return LILY_ERR_ARG;
    }
    static_assert(sizeof(cudaIpcMemHandle_t) == LILY_IPC_HANDLE_BYTES, "the handle travels as 64 bytes");
    DeviceGuard guard(device);
    const size_t bytes = lily_peer_buffer_bytes(n_shards, max_rows);
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        return LILY_ERR_CUDA;
    }
    cudaIpcMemHandle_t handle;
    if (cudaMemset(p, 0, bytes) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaIpcGetMemHandle(&handle, p) != cudaSuccess) {
        cudaFree(p);
        return LILY_ERR_CUDA;
    }
    std::memcpy(ipc_handle, &handle, sizeof handle);
    *buffer = p;
    return LILY_OK;
}

int32_t lily_peer_buffer_open(int32_t device, const void *ipc_handle, void **buffer) {
    if (buffer == nullptr || ipc_handle == nullptr) {
        return LILY_ERR_ARG;
    }
    DeviceGuard guard(device);
    cudaIpcMemHandle_t handle;
    std::memcpy(&handle, ipc_handle, sizeof handle);
    return cudaIpcOpenMemHandle(buffer, handle, cudaIpcMemLazyEnablePeerAccess) == cudaSuccess ? LILY_OK
                                                                                                : LILY_ERR_CUDA;
}

int32_t lily_peer_buffer_close(int32_t device, void *buffer) {
    DeviceGuard guard(device);
    return buffer != nullptr && cudaIpcCloseMemHandle(buffer) == cudaSuccess ? LILY_OK : LILY_ERR_CUDA;
}

int32_t lily_peer_buffer_destroy(int32_t device, void *buffer) {
    DeviceGuard guard(device);
    return cudaFree(buffer) == cudaSuccess ? LILY_OK : LILY_ERR_CUDA;
}

int32_t lily_shard_publish(lily_sampler_t *h, void *stream_, const lily_peer_exchange_t *x,
                           const void *records, uint32_t rows, uint32_t step) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if ((st = peer_check(h, x)) != LILY_OK) {
        return st;
    }
    if (records == nullptr || rows == 0u || rows > x->max_rows || reinterpret_cast<uintptr_t>(records) % 8u) {
        return fail(h, LILY_ERR_ARG, "records set and 8-byte aligned, 1 <= rows <= max_rows");
    }
    DeviceGuard guard(h->device);
    lily::PeerArgs p;
    std::memset(&p, 0, sizeof p);
    for (uint32_t r = 0; r < x->n_shards; ++r) {
        p.buffers[r] = x->buffers[r];
    }
    p.n_shards = x->n_shards;
    p.rank = x->rank;
    p.max_rows = x->max_rows;
    p.records = static_cast<const lily::ShardRecord *>(records);
    p.rows = rows;
    p.step = step;
    lily::shard_publish_kernel<<<x->n_shards, 256, 0, static_cast<cudaStream_t>(stream_)>>>(p);
    CU(h, cudaGetLastError());
    return LILY_OK;
}

int32_t lily_merge_draw_peer(lily_sampler_t *h, void *stream_, const lily_peer_exchange_t *x,
                             const void *records, uint32_t step, const lily_sample_args_t *args,
                             float *out_lse) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if ((st = peer_check(h, x)) != LILY_OK) {
        return st;
    }
    if (args == nullptr || args->struct_size != sizeof(lily_sample_args_t) || args->rows > x->max_rows) {
        return fail(h, LILY_ERR_ARG, "args is null, of another ABI version, or has more rows than max_rows");
    }
    if (reinterpret_cast<uintptr_t>(records) % 8u) {
        return fail(h, LILY_ERR_ARG, "records must be 8-byte aligned");
    }
    lily::KArgs::PeerLink peer;
    std::memset(&peer, 0, sizeof peer);
    for (uint32_t r = 0; r < x->n_shards; ++r) {
        peer.buffers[r] = x->buffers[r];
    }
    peer.own = records;
    peer.wait_ns = h->wait_ns;
    peer.n = x->n_shards;
    peer.rank = x->rank;
    peer.max_rows = x->max_rows;
    peer.step = step;
    const char *slot = static_cast<const char *>(x->buffers[x->rank]) +
                       lily::peer_flag_bytes(x->n_shards, x->max_rows) +
                       (size_t)(step & 1u) * x->n_shards * x->max_rows * sizeof(lily::ShardRecord);
    return merge_draw(h, stream_, slot, x->n_shards, x->max_rows, args, out_lse, &peer);
}

// ----------------------------------------------------------- speculation --

int32_t lily_spec_verify(lily_sampler_t *h, void *stream_, const lily_spec_args_t *args) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (args == nullptr || args->struct_size != sizeof(lily_spec_args_t)) {
        return fail(h, LILY_ERR_ARG, "args is null or of another ABI version");
    }
    const lily_spec_args_t &g = *args;
    if (g.m == 0u || g.m > 8u || g.m > h->max_rows) {
        return fail(h, LILY_ERR_CAPACITY, "m outside 1..min(8, max_rows)");
    }
    if (g.target_logits == nullptr || g.params == nullptr || g.out_ids == nullptr ||
        g.out_accepted == nullptr || g.logits_ld < h->vocab || g.logits_dtype > LILY_BF16 ||
        g.mode > LILY_SPEC_GREEDY_MATCH) {
        return fail(h, LILY_ERR_ARG, "target logits, params and outputs must be set");
    }
    if (g.m > 1u && g.draft_ids == nullptr) {
        return fail(h, LILY_ERR_ARG, "draft_ids missing");
    }
    if (!params_ok(*g.params)) {
        return fail(h, LILY_ERR_PARAMS, "invalid sampling parameters");
    }
    lily_sampling_params_t p = *g.params;
    if (g.mode == LILY_SPEC_GREEDY_MATCH) {
        p.temperature = 0.0f;
    }
    const bool pen = uses_penalties(p);
    const bool argmax_rows = is_greedy(p) && !pen;
    const bool spec_rows = g.mode == LILY_SPEC_REJECTION && !argmax_rows && g.m > 1u;
    if (spec_rows) {
        const bool dense = g.q_dense != nullptr;
        const bool sparse = g.q_ids != nullptr && g.q_probs != nullptr && g.q_n != nullptr;
        if (dense == sparse) {
            return fail(h, LILY_ERR_ARG, "give the draft distribution dense or sparse, not both");
        }
        if (dense && g.q_ld < h->vocab) {
            return fail(h, LILY_ERR_ARG, "q_ld < vocab");
        }
    }
    if (g.history_len > 0u && g.history_ids == nullptr) {
        return fail(h, LILY_ERR_ARG, "history_len without history_ids");
    }
    if (g.count_slot != nullptr && (h->counts_table == nullptr || *g.count_slot >= h->max_rows)) {
        return fail(h, LILY_ERR_ARG, "no such histogram slot");
    }
    DeviceGuard guard(h->device);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    lily::KArgs a;
    base_args(h, &a);
    a.logits = g.target_logits;
    a.logits_ld = g.logits_ld;
    a.rows = g.m;
    a.uniforms = g.u_accept;
    a.history_ids = g.history_ids;
    a.history_ld = 0;  // every row of the step reads the same list
    a.out_ids = g.out_ids;
    a.out_status = g.out_status;
    if (spec_rows) {
        a.spec.draft_ids = g.draft_ids;
        a.spec.q_dense = g.q_dense;
        a.spec.q_ld = g.q_ld;
        a.spec.q_ids = g.q_ids;
        a.spec.q_probs = g.q_probs;
        a.spec.q_n = g.q_n;
        a.spec.u_resid = g.u_resid;
        a.spec.n_spec = g.m - 1u;
    }
    // Without penalties the rows do not depend on one another. With them row j's see
    // the draws of rows < j (the reference's rows share one histogram,
    // src/qwen4exp/model.rs:3008-3012): one launch per row, in stream order.
    const uint32_t launches = pen ? g.m : 1u, rows = pen ? 1u : g.m;
    a.n_slices = choose_slices(h, rows);
    const bool listed = g.count_slot == nullptr && pen;
    const SplitPlan plan = split_plan(h, a, rows, g.logits_dtype, listed, p.frequency_penalty != 0.0f);
    const bool in_args = plan.take;
    lily_sampling_params_t params[8];
    uint32_t steps[8], slots[8];
    for (uint32_t j = 0; j < g.m; ++j) {
        params[j] = p;
        steps[j] = g.step0 + j;
        slots[j] = g.count_slot ? *g.count_slot : 0u;
    }
    int slot = -1;
    if (!in_args) {
        st = next_stage(h, &slot);
        if (st != LILY_OK) {
            return st;
        }
        char *hs = h->h_stage[slot], *ds = h->d_stage[slot];
        const StageLayout layout = stage_layout(g.m);
        auto *sh = reinterpret_cast<uint32_t *>(hs + layout.hist_len);
        std::memcpy(hs + layout.params, params, sizeof(params[0]) * g.m);
        std::memcpy(hs + layout.steps, steps, 4u * g.m);
        std::memcpy(hs + layout.slots, slots, 4u * g.m);
        for (uint32_t j = 0; j < g.m; ++j) {
            sh[j] = g.history_len;
        }
        if ((st = upload(h, slot, layout.total, stream)) != LILY_OK) {
            return st;
        }
        a.params = reinterpret_cast<const lily_sampling_params_t *>(ds + layout.params);
        a.steps = reinterpret_cast<const uint32_t *>(ds + layout.steps);
        a.history_len = g.history_ids ? reinterpret_cast<const uint32_t *>(ds + layout.hist_len) : nullptr;
        a.count_slots = g.count_slot ? reinterpret_cast<const uint32_t *>(ds + layout.slots) : nullptr;
    }
    for (uint32_t j = 0; j < launches && st == LILY_OK; ++j) {
        a.row0 = j;
        if (listed) {
            a.extra_ids = g.out_ids;
            a.extra_len = j;
        }
        st = in_args ? launch_split_inline<INLINE_ROWS>(h, stream, a, plan, pen ? j + 1u : g.m, g.logits_dtype, params,
                                                        steps, g.count_slot ? slots : nullptr, 1u + g.history_len, rows)
                     : launch(h, stream, a, rows, g.logits_dtype);
    }
    if (st == LILY_OK) {
        if (g.m > 1u) {
            st = launch_accept(h, stream, g.out_ids, g.draft_ids, 0u, g.m, g.out_accepted, 0u, 1u, 0u, 0u);
        } else {
            CU(h, cudaMemsetAsync(g.out_accepted, 0, 4, stream));
        }
        CU(h, cudaGetLastError());
    }
    if (slot >= 0) {
        CU(h, cudaEventRecord(h->ev[slot], stream));
    }
    return st;
}

int32_t lily_spec_accept(lily_sampler_t *h, void *stream_, const uint32_t *draws,
                         const uint32_t *ids, uint32_t m, uint32_t *ctrl, uint32_t pos0,
                         uint32_t ratio, uint32_t chain, uint32_t stride) {
    int32_t st = check_handle(h);
    if (st != LILY_OK) {
        return st;
    }
    if (draws == nullptr || ids == nullptr || ctrl == nullptr || m == 0u) {
        return fail(h, LILY_ERR_ARG, "draws and ids must both hold the verified rows");
    }
    if (ratio == 0u) {
        return fail(h, LILY_ERR_ARG, "indexer block ratio must be nonzero");
    }
    if (stride == 0u) {
        return fail(h, LILY_ERR_ARG, "stride must be nonzero");
    }
    DeviceGuard guard(h->device);
    return launch_accept(h, static_cast<cudaStream_t>(stream_), draws, ids, 1u, m, ctrl, pos0, ratio, chain, stride);
}

// ------------------------------------------------ allocation-free draw --

}  // extern "C"

namespace {

// Everything the kernel needs beyond its inputs and outputs, for up to
// LILY_NOALLOC_MAX_ROWS rows. The layout is what the kernel indexes:
// part[row][CAP], part_n[row][MAX_SLICES], tickets[row].
struct NoAllocScratch {
    uint2 part[LILY_NOALLOC_MAX_ROWS][lily::CAP];
    uint32_t part_n[LILY_NOALLOC_MAX_ROWS][lily::MAX_SLICES];
    uint32_t tickets[LILY_NOALLOC_MAX_ROWS];
    uint32_t status_word;
    uint32_t steps[LILY_NOALLOC_MAX_ROWS];
    lily_sampling_params_t params[LILY_NOALLOC_MAX_ROWS];
};
static_assert(sizeof(NoAllocScratch) <= LILY_NOALLOC_SCRATCH_BYTES, "stated size too small");

// Static device storage: no allocation call ever makes or frees it. In host
// code this name is only a stand-in for the array, not a device address: the
// address comes from cudaGetSymbolAddress, once per device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[LILY_NOALLOC_SCRATCH_BYTES];

struct NoAllocDevice {
    bool ready = false;
    NoAllocScratch *scratch = nullptr;  // device address on this device
    int sm_count = 0;
    int max_smem = 0;
    uint32_t attr_mask = 0;
};
NoAllocDevice g_noalloc_devices[64];
std::mutex g_noalloc_mutex;  // guards the per-device set-up above (host threads may race to the first call)

int32_t noalloc_fail(int32_t code, const char *msg, char *err, uint32_t err_cap) {
    if (err != nullptr && err_cap > 0u) {
        std::snprintf(err, err_cap, "%s", msg);
    }
    return code;
}

template <typename T, bool VEC>
cudaError_t noalloc_launch_one(NoAllocDevice *d, cudaStream_t stream, const lily::KArgs &a,
                               uint32_t rows, size_t smem) {
    auto kernel = lily::sample_rows_kernel<T, VEC>;
    const uint32_t bit = 1u << ((sizeof(T) == 4 ? 0 : 2) + (VEC ? 1 : 0));
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!(d->attr_mask & bit)) {
            const cudaError_t e = cudaFuncSetAttribute(
                kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, d->max_smem);
            if (e != cudaSuccess) {
                return e;
            }
            d->attr_mask |= bit;
        }
    }
    dim3 grid(a.n_slices, rows, 1);
    kernel<<<grid, lily::NT, smem, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace

extern "C" {

int32_t lily_sample_batch_noalloc(void *stream_, uint32_t vocab, const lily_sample_args_t *args,
                                  char *err, uint32_t err_cap) {
    if (args == nullptr || args->struct_size != sizeof(lily_sample_args_t)) {
        return noalloc_fail(LILY_ERR_ARG, "args is null or of another ABI version", err, err_cap);
    }
    const lily_sample_args_t &g = *args;
    if (g.rows == 0u || g.rows > LILY_NOALLOC_MAX_ROWS) {
        return noalloc_fail(LILY_ERR_CAPACITY, "rows outside 1..LILY_NOALLOC_MAX_ROWS", err, err_cap);
    }
    if (vocab == 0u || vocab > (1u << 24) || g.logits == nullptr || g.out_ids == nullptr ||
        g.params == nullptr || g.logits_ld < vocab || g.logits_dtype > LILY_BF16) {
        return noalloc_fail(LILY_ERR_ARG,
                            "logits must be F32 or BF16 [rows, ld >= vocab]; out and params set",
                            err, err_cap);
    }
    if (g.params_on_device != 0u || g.count_slots != nullptr) {
        return noalloc_fail(LILY_ERR_ARG,
                            "the allocation-free draw takes host params and no histogram slots",
                            err, err_cap);
    }
    if (g.uniforms == nullptr && g.steps == nullptr) {
        return noalloc_fail(LILY_ERR_ARG, "either uniforms or steps must be given", err, err_cap);
    }
    if ((g.history_ids != nullptr) != (g.history_len != nullptr) ||
        (g.bias_ids != nullptr) != (g.bias_len != nullptr) ||
        (g.bias_ids != nullptr) != (g.bias_vals != nullptr) ||
        (g.ban_ids != nullptr) != (g.ban_len != nullptr)) {
        return noalloc_fail(LILY_ERR_ARG, "a list needs both its ids and its lengths", err, err_cap);
    }
    if (g.kept_n != nullptr &&
        (g.kept_ids == nullptr || g.kept_probs == nullptr || g.kept_ld < LILY_K_CAP)) {
        return noalloc_fail(LILY_ERR_ARG, "kept_n needs kept_ids, kept_probs and kept_ld >= 1024",
                            err, err_cap);
    }
    for (uint32_t r = 0; r < g.rows; ++r) {
        if (!params_ok(g.params[r])) {
            return noalloc_fail(LILY_ERR_PARAMS, "invalid sampling parameters", err, err_cap);
        }
        if (g.history_ids != nullptr && uses_penalties(g.params[r]) &&
            g.params[r].frequency_penalty != 0.0f) {
            return noalloc_fail(LILY_ERR_CAPACITY,
                                "a frequency penalty over a history list needs a vocabulary-sized "
                                "count table, which the allocation-free draw does not carry",
                                err, err_cap);
        }
    }
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) {
        return noalloc_fail(LILY_ERR_CUDA, "no current CUDA device", err, err_cap);
    }
    NoAllocDevice *d = &g_noalloc_devices[device];
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!d->ready) {
            // Set-up, once per device, with that device current: the array's
            // address ON THIS DEVICE. (Passing the host-side name to the kernel
            // instead would hand it a host address.)
            void *p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || p == nullptr) {
                return noalloc_fail(LILY_ERR_CUDA, "cudaGetSymbolAddress failed for the static scratch",
                                    err, err_cap);
            }
            if (cudaDeviceGetAttribute(&d->sm_count, cudaDevAttrMultiProcessorCount, device) !=
                    cudaSuccess ||
                cudaDeviceGetAttribute(&d->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) !=
                    cudaSuccess) {
                return noalloc_fail(LILY_ERR_CUDA, "device attributes unavailable", err, err_cap);
            }
            d->scratch = static_cast<NoAllocScratch *>(p);
            d->ready = true;
        }
    }
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    NoAllocScratch *sc = d->scratch;
    // The array keeps the last call's contents: the tickets and the status
    // word must start at zero; the parameters are overwritten.
    if (cudaMemsetAsync(sc->tickets, 0, sizeof(sc->tickets) + sizeof(sc->status_word), stream) !=
            cudaSuccess ||
        cudaMemcpyAsync(sc->params, g.params, sizeof(lily_sampling_params_t) * g.rows,
                        cudaMemcpyHostToDevice, stream) != cudaSuccess ||
        (g.steps != nullptr &&
         cudaMemcpyAsync(sc->steps, g.steps, sizeof(uint32_t) * g.rows, cudaMemcpyHostToDevice,
                         stream) != cudaSuccess)) {
        return noalloc_fail(LILY_ERR_CUDA, "staging the parameters failed", err, err_cap);
    }
    lily::KArgs a;
    std::memset(&a, 0, sizeof(a));
    a.vocab = vocab;
    a.max_history = 1u << 16;
    a.max_list = 512u;
    a.part = &sc->part[0][0];
    a.part_n = &sc->part_n[0][0];
    a.tickets = sc->tickets;
    a.status_word = &sc->status_word;
    a.logits = g.logits;
    a.logits_ld = g.logits_ld;
    a.rows = g.rows;
    a.params = sc->params;
    a.uniforms = g.uniforms;
    a.steps = g.steps != nullptr ? sc->steps : nullptr;
    a.history_ids = g.history_ids;
    a.history_len = g.history_len;
    a.history_ld = g.history_ld;
    a.bias_ids = g.bias_ids;
    a.bias_vals = g.bias_vals;
    a.bias_len = g.bias_len;
    a.bias_ld = g.bias_ld;
    a.ban_ids = g.ban_ids;
    a.ban_len = g.ban_len;
    a.ban_ld = g.ban_ld;
    a.forced_ids = g.forced_ids;
    a.out_ids = g.out_ids;
    a.out_status = g.out_status;
    a.kept_n = g.kept_n;
    a.kept_ids = g.kept_ids;
    a.kept_probs = g.kept_probs;
    a.kept_ld = g.kept_ld;
    uint32_t slices = 2u * (uint32_t)d->sm_count / g.rows;
    const uint32_t by_len = (vocab + lily::MIN_SLICE - 1u) / lily::MIN_SLICE;
    slices = slices > lily::MAX_SLICES ? lily::MAX_SLICES : slices;
    slices = slices > by_len ? by_len : slices;
    a.n_slices = slices < 1u ? 1u : slices;
    const size_t smem = smem_bytes(vocab, a.n_slices);
    if (smem > (size_t)d->max_smem) {
        return noalloc_fail(LILY_ERR_CAPACITY, "vocabulary too large for the shared-memory bitmap",
                            err, err_cap);
    }
    const size_t esize = g.logits_dtype == LILY_F32 ? 4 : 2;
    const bool vec = (reinterpret_cast<uintptr_t>(a.logits) % 16u == 0u) &&
                     ((a.logits_ld * esize) % 16u == 0u);
    cudaError_t e;
    if (g.logits_dtype == LILY_F32) {
        e = vec ? noalloc_launch_one<float, true>(d, stream, a, g.rows, smem)
                : noalloc_launch_one<float, false>(d, stream, a, g.rows, smem);
    } else {
        e = vec ? noalloc_launch_one<__nv_bfloat16, true>(d, stream, a, g.rows, smem)
                : noalloc_launch_one<__nv_bfloat16, false>(d, stream, a, g.rows, smem);
    }
    if (e != cudaSuccess) {
        return noalloc_fail(LILY_ERR_CUDA, cudaGetErrorString(e), err, err_cap);
    }
    return LILY_OK;
}

int32_t lily_debug_exp(void *stream_, const float *in, float *out, uint64_t n) {
    if (in == nullptr || out == nullptr) {
        return LILY_ERR_ARG;
    }
    if (n == 0u) {
        return LILY_OK;
    }
    const uint32_t threads = 256;
    const uint64_t blocks = (n + threads - 1u) / threads;
    lily::exp_kernel<<<(uint32_t)(blocks > 65535u * 16u ? 65535u * 16u : blocks), threads, 0,
                       static_cast<cudaStream_t>(stream_)>>>(in, out, n);
    return cudaGetLastError() == cudaSuccess ? LILY_OK : LILY_ERR_CUDA;
}

}  // extern "C"
