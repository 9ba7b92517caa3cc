// The row kernel: a row's vocabulary is split over the blocks of a cluster (one,
// two, four or eight of them, as many as leave every SM something to do), which
// meet once.
//
//   1. every thread looks at its vectors of the row (16 bytes each) and keeps the
//      largest logit it saw; eight vectors (a bucket) share one maximum in shared
//      memory. History ids are marked on the way, one byte, bit or count per
//      vocabulary id of the block's share;
//   2. with penalties that only lower a logit, the adjusted value of any k
//      logits bounds the row's k-th largest from below: the block takes the k-th
//      largest among its threads' (adjusted) maxima as its bound. That is tight,
//      because the best logits hardly ever share a thread;
//   3. the buckets that reach the bound are read again (L2), and what reaches it
//      is adjusted, divided by the temperature and stored, as (key, id), in the
//      shared memory of the cluster's first block;
//   4. the first block ranks the candidates ((key descending, id ascending), as
//      the reference's CPU sampler orders them), runs the softmax weights, the
//      prefix sums in rank order, the cut and the draw.
//
// A row that keeps more than 64 candidates takes its bound from the maxima of all
// threads of the cluster (one more meeting). Rows this kernel does not take
// (penalties that can raise a logit, a NaN, more ties than the buffers hold, ...)
// are drawn by the first block alone with the general row code: the results do
// not depend on the way.
//
// Every warp reads 512 consecutive bytes at a time, and the pieces go round the
// blocks and warps in turn: neighbouring ids, which often have similar logits, end
// up in different threads. A row need not be aligned: the pieces lie on 16-byte
// boundaries, and the vectors that stick out at its two ends are put together
// element by element.
#pragma once

#include <type_traits>

#include "split_args.cuh"

namespace lily {

__device__ __forceinline__ void spl_sync() { asm volatile("bar.sync 1, %0;" ::"n"(SPL_NT) : "memory"); }

// The address of a shared-memory word in block `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_smem(const void *p, uint32_t rank) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return at;
}

// Stores into another block's shared memory that complete bytes of a barrier
// there: no fence on this side, no meeting of all threads.
__device__ __forceinline__ void put_u32(uint32_t at, uint32_t v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(at), "r"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void put_2u32(uint32_t at, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.u32 [%0], {%1, %2}, [%3];" ::"r"(at), "r"(x),
                 "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void put_4u32(uint32_t at, uint32_t x, uint32_t y, uint32_t z, uint32_t w, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.u32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(at),
                 "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void arrive_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

// Waits for the first phase of a barrier in this block, some milliseconds at most
// (the other blocks of the cluster are running: they only have to get there).
__device__ __forceinline__ bool wait_first_phase(const unsigned long long *bar) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(bar);
    for (uint32_t i = 0; i < (1u << 18); ++i) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(at)
            : "memory");
        if (done) {
            return true;
        }
    }
    return false;
}

// The largest of a vector's logits; NaN if one is.
template <typename T>
__device__ __forceinline__ float vec_max(const uint4 &q) {
    if (sizeof(T) == 4) {
        return max_nan_f32(max_nan_f32(__uint_as_float(q.x), __uint_as_float(q.y)),
                           max_nan_f32(__uint_as_float(q.z), __uint_as_float(q.w)));
    }
    const uint32_t m = max_nan_bf16x2(max_nan_bf16x2(q.x, q.y), max_nan_bf16x2(q.z, q.w));
    return max_nan_f32(bf16_lo(m), bf16_hi(m));
}

template <typename T>
__device__ __forceinline__ float vec_get(const uint4 &q, uint32_t e) {
    const uint32_t w = sizeof(T) == 4 ? e : e >> 1;
    const uint32_t x = w == 0u ? q.x : w == 1u ? q.y : w == 2u ? q.z : q.w;
    return sizeof(T) == 4 ? __uint_as_float(x) : (e & 1u) ? bf16_hi(x) : bf16_lo(x);
}

// A vector that sticks out of the row: element by element, -inf outside.
template <typename T>
static __device__ __noinline__ uint4 edge_vec(const T *row_ptr, uint32_t vocab, uint32_t skip, uint32_t v) {
    constexpr uint32_t PER = Piece<T>::PER;
    uint32_t w[4];
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
        w[i] = sizeof(T) == 4 ? 0xFF800000u : 0xFF80FF80u;
    }
#pragma unroll
    for (uint32_t e = 0; e < PER; ++e) {
        const uint32_t id = v * PER + e - skip;  // (wraps past the vocabulary in front of the row)
        if (id < vocab) {
            const uint32_t x = __float_as_uint(widen(row_ptr[id]));
            if (sizeof(T) == 4) {
                w[e & 3u] = x;
            } else {
                w[(e >> 1) & 3u] = (e & 1u) ? (w[(e >> 1) & 3u] & 0xFFFFu) | x
                                            : (w[(e >> 1) & 3u] & 0xFFFF0000u) | (x >> 16);
            }
        }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}


// The best k of the candidates in the blocks' regions, sorted into key[] / id[]
// [0, k): for rows that keep many. A histogram over the distance from the top puts
// each near its place, the few that share a bin are ranked by counting. Returns how
// many there are (at most k), 0 if they do not fit. Keys below `kmin` are not
// wanted. `room`: SPL_SORTED words of 8 bytes. All SPL_NT threads.
static __device__ __noinline__ uint32_t split_sort_bins(SmemFixed *sm, SplitSmem *ss, unsigned long long *room,
                                                 uint32_t log_blocks, uint32_t k, uint32_t kmin) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr uint32_t BPT = TH_BINS / SPL_NT;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint2 *cand = reinterpret_cast<const uint2 *>(sm->key);  // over key and id: CAP of them
    const uint32_t cap = CAP >> log_blocks, team = SPL_NT >> log_blocks;
    const uint32_t region = tid / team, n_region = ss->head[region].x;
    const uint2 *mine = cand + region * cap;
    uint32_t best = 0;
    for (uint32_t i = tid % team; i < n_region; i += team) {
        best = max(best, mine[i].x);
    }
    best = __reduce_max_sync(FULL, best);
    for (uint32_t b = tid; b < TH_BINS; b += SPL_NT) {
        sm->thist[b] = 0;
        sm->tkey[b] = 0;
    }
    if (lane == 0) {
        sm->warp_sums[warp] = best;
    }
    spl_sync();
    best = __reduce_max_sync(FULL, sm->warp_sums[lane & (SPL_WARPS - 1u)]);
    const float top = float_of_key(best), low = float_of_key(kmin);
    const float range = __fsub_rn(top, low);
    const float scale = range > 0.0f ? __fdiv_rn((float)(TH_BINS - 1u), range) : 0.0f;
    // (Falls with the key: every step is monotone. A NaN or an infinity lands in bin 0 or the last.)
    auto bin_of = [&](uint32_t x) -> uint32_t {
        const float d = __fmul_rn(__fsub_rn(top, float_of_key(x)), scale);
        return d > 0.0f ? min((uint32_t)d, TH_BINS - 1u) : 0u;
    };
    for (uint32_t i = tid % team; i < n_region; i += team) {
        const uint32_t x = mine[i].x;
        if (x >= kmin) {
            atomicAdd(&sm->thist[bin_of(x)], 1u);
        }
    }
    spl_sync();
    // Candidates in the bins before each.
    uint32_t c[BPT], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < BPT; ++j) {
        c[j] = sm->thist[tid * BPT + j];
        sum += c[j];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, incl, o);
        if (lane >= (uint32_t)o) {
            incl += t;
        }
    }
    if (lane == 31u) {
        sm->warp_sums[SPL_WARPS + warp] = incl;
    }
    if (tid == 0) {
        ss->bin = 0;  // the end of the last bin that is needed
    }
    spl_sync();
    uint32_t before = incl - sum, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < SPL_WARPS; ++w) {
        const uint32_t s = sm->warp_sums[SPL_WARPS + w];
        before += w < warp ? s : 0u;
        total += s;
    }
    uint32_t end = 0;
#pragma unroll
    for (uint32_t j = 0; j < BPT; ++j) {
        sm->tid[tid * BPT + j] = before;
        if (before < k) {
            end = before + c[j];
        }
        before += c[j];
    }
    end = __reduce_max_sync(FULL, end);
    if (lane == 0) {
        atomicMax(&ss->bin, end);
    }
    spl_sync();
    end = ss->bin;
    if (end > SPL_SORTED) {
        return 0u;
    }
    // To the bin's part of the array (bins that begin past rank k are not needed).
    for (uint32_t i = tid % team; i < n_region; i += team) {
        const uint2 e = mine[i];
        if (e.x >= kmin) {
            const uint32_t b = bin_of(e.x), first = sm->tid[b];
            if (first < k) {
                room[first + atomicAdd(&sm->tkey[b], 1u)] = ((unsigned long long)e.x << 32) | (uint32_t)~e.y;
            }
        }
    }
    spl_sync();
    for (uint32_t i = tid; i < end; i += SPL_NT) {
        const unsigned long long me = room[i];
        const uint32_t b = bin_of((uint32_t)(me >> 32)), first = sm->tid[b], last = first + sm->thist[b];
        uint32_t place = first;
        for (uint32_t j = first; j < last; ++j) {
            place += room[j] > me ? 1u : 0u;
        }
        if (place < k) {
            sm->key[place] = (uint32_t)(me >> 32);
            sm->id[place] = ~(uint32_t)me;
        }
    }
    spl_sync();
    return min(total, k);
}

// The draw of a row that keeps more than 64 candidates, sorted in key[] / id[]: the
// softmax weights, the prefix sums in rank order with one rounding per add
// (tests/unit/kernels/sample.rs:37-46), the cut, the draw. All SPL_NT threads.
static __device__ __noinline__ void split_finalize_wide(SmemFixed *sm, SplitSmem *ss, const KArgs &a, uint32_t row, uint32_t n,
                                                 float top_p, float min_p, float u, bool counts_draw, uint32_t slot) {
    const uint32_t tid = threadIdx.x;
    float *p = reinterpret_cast<float *>(sm->tkey), *cum = reinterpret_cast<float *>(sm->tid);
    const float top = float_of_key(sm->key[0]);
    if (top == neg_inf() || top == -neg_inf()) {
        if (tid == 0) {
            a.out_ids[row] = 0xFFFFFFFFu;
            if (a.out_status) {
                a.out_status[row] = LILY_ROW_NONFINITE;
            }
            if (a.kept_n) {
                a.kept_n[row] = 0;
            }
            atomicOr(a.status_word, 1u << LILY_ROW_NONFINITE);
        }
        return;
    }
    for (uint32_t i = tid; i < KCAP; i += SPL_NT) {
        p[i] = i < n ? exp_f32(__fsub_rn(float_of_key(sm->key[i]), top)) : 0.0f;
    }
    if (tid == 0) {
        ss->n_live = n;   // the first rank that is not kept
        ss->bin = n;      // the first rank whose prefix sum exceeds the target
    }
    spl_sync();
    if (tid == 0) {
        // A chain of n dependent adds; the loads run one step ahead of it. (Ranks past
        // n weigh 0, and s + 0 is s.)
        const float4 *p4 = reinterpret_cast<const float4 *>(p);
        float4 *c4 = reinterpret_cast<float4 *>(cum);
        const uint32_t steps = (n + 7u) / 8u;
        float s = 0.0f;
        float4 v0 = p4[0], v1 = p4[1];
        for (uint32_t i = 0; i < steps; ++i) {
            const uint32_t nx = min(i + 1u, KCAP / 8u - 1u);
            const float4 w0 = p4[2u * nx], w1 = p4[2u * nx + 1u];
            float4 o0, o1;
            o0.x = s = __fadd_rn(s, v0.x);
            o0.y = s = __fadd_rn(s, v0.y);
            o0.z = s = __fadd_rn(s, v0.z);
            o0.w = s = __fadd_rn(s, v0.w);
            o1.x = s = __fadd_rn(s, v1.x);
            o1.y = s = __fadd_rn(s, v1.y);
            o1.z = s = __fadd_rn(s, v1.z);
            o1.w = s = __fadd_rn(s, v1.w);
            c4[2u * i] = o0;
            c4[2u * i + 1u] = o1;
            v0 = w0;
            v1 = w1;
        }
    }
    spl_sync();
    const float limit = __fmul_rn(top_p, cum[n - 1u]);
    for (uint32_t i = tid + 1u; i < n; i += SPL_NT) {
        if (!(cum[i - 1u] < limit && p[i] >= min_p)) {
            atomicMin(&ss->n_live, i);
            break;  // (this thread's later ranks are larger)
        }
    }
    spl_sync();
    const uint32_t n_keep = ss->n_live;
    const float mass = cum[n_keep - 1u];
    // First kept rank whose prefix sum exceeds the target, else the last one.
    const float target = __fmul_rn(u, mass);
    for (uint32_t i = tid; i < n_keep; i += SPL_NT) {
        if (target < cum[i]) {
            atomicMin(&ss->bin, i);
            break;
        }
    }
    if (a.kept_n) {
        for (uint32_t i = tid; i < n_keep; i += SPL_NT) {
            a.kept_ids[(uint64_t)row * a.kept_ld + i] = sm->id[i];
            a.kept_probs[(uint64_t)row * a.kept_ld + i] = __fdiv_rn(p[i], mass);
        }
    }
    spl_sync();
    if (tid == 0) {
        const uint32_t id = sm->id[min(ss->bin, n_keep - 1u)];
        a.out_ids[row] = id;
        if (a.out_status) {
            a.out_status[row] = LILY_ROW_OK;
        }
        if (a.kept_n) {
            a.kept_n[row] = n_keep;
        }
        if (counts_draw && id < a.vocab) {
            // src/kernels/metal/sample.metal:509-511: the draw is counted.
            atomicAdd(a.counts_table + (uint64_t)slot * a.vocab + id, 1u);
            atomicOr(a.seen_table + (uint64_t)slot * a.seen_words + (id >> 5), 1u << (id & 31u));
        }
    }
}

// What a speculative row needs of its proposal, asked for while the row is still
// being read: warp 0 of the first block, lane i with entries i and i + 32 of a
// sparse draft distribution.
struct SpecAhead {
    uint32_t draft, n_q, id0, id1;
    float q_draft, p0, p1;
};

__device__ __forceinline__ void spec_ahead(const SpecArgs &s, uint32_t row, uint32_t vocab, SpecAhead &h) {
    const uint32_t lane = threadIdx.x & 31u;
    h.n_q = h.id0 = h.id1 = 0;
    h.q_draft = h.p0 = h.p1 = 0.0f;
    if (s.q_dense) {
        h.q_draft = h.draft < vocab ? __ldg(s.q_dense + (uint64_t)row * s.q_ld + h.draft) : 0.0f;
    } else {
        h.n_q = min(__ldg(s.q_n + row), KCAP);
        const uint32_t *qi = s.q_ids + (uint64_t)row * KCAP;
        const float *qp = s.q_probs + (uint64_t)row * KCAP;
        if (lane < h.n_q) {
            h.id0 = __ldg(qi + lane);
            h.p0 = __ldg(qp + lane);
        }
        if (lane + 32u < h.n_q) {
            h.id1 = __ldg(qi + lane + 32u);
            h.p1 = __ldg(qp + lane + 32u);
        }
    }
}

// Running sums in rank order, one rounding per add, of the weights w[0, 64) (ranks
// past the last weigh 0, and s + 0 is s): lane i gets those of ranks i and i + 32.
// Every lane runs its own chain up to its own rank; the weights come four at a time.
__device__ __forceinline__ void rank_sums(const float *w, uint32_t n, float &c0, float &c1) {
    const uint32_t lane = threadIdx.x & 31u;
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    c0 = 0.0f;
#pragma unroll 2
    for (uint32_t i = 0; i < 32u && i < n; i += 4u) {
        const float4 v = w4[i >> 2];
        c0 = lane >= i ? __fadd_rn(c0, v.x) : c0;
        c0 = lane >= i + 1u ? __fadd_rn(c0, v.y) : c0;
        c0 = lane >= i + 2u ? __fadd_rn(c0, v.z) : c0;
        c0 = lane >= i + 3u ? __fadd_rn(c0, v.w) : c0;
    }
    c1 = __shfl_sync(0xFFFFFFFFu, c0, 31);
#pragma unroll 2
    for (uint32_t i = 32u; i < n; i += 4u) {
        const float4 v = w4[i >> 2];
        c1 = lane + 32u >= i ? __fadd_rn(c1, v.x) : c1;
        c1 = lane + 32u >= i + 1u ? __fadd_rn(c1, v.y) : c1;
        c1 = lane + 32u >= i + 2u ? __fadd_rn(c1, v.z) : c1;
        c1 = lane + 32u >= i + 3u ? __fadd_rn(c1, v.w) : c1;
    }
}

// The draw from at most 64 candidates, sorted in key[] / id[], by one warp: the
// softmax weights, the prefix sums in rank order (tests/unit/kernels/sample.rs:37-46),
// the cut, the draw (speculative: tests/unit/kernels/sample.rs:264-283, src/kernels/
// metal/sample.metal:597-658), the outputs. lane i holds ranks i and i + 32.
static __device__ __noinline__ void split_finalize(SmemFixed *sm, const KArgs &a, uint32_t row, uint32_t n, float top_p, float min_p,
                                            float u, uint32_t step, uint64_t seed, bool counts_draw, uint32_t slot,
                                            const SpecAhead &ahead) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    float *w = reinterpret_cast<float *>(sm->tkey);
    const bool in0 = lane < n, in1 = lane + 32u < n;
    const uint32_t i0 = in0 ? sm->id[lane] : 0xFFFFFFFFu, i1 = in1 ? sm->id[lane + 32u] : 0xFFFFFFFFu;
    const float top = float_of_key(sm->key[0]);
    const bool spec = row < a.spec.n_spec;
    float q0 = 0.0f, q1 = 0.0f;
    if (spec && a.spec.q_dense) {  // (for the residual, if it comes to that: on their way meanwhile)
        const float *q = a.spec.q_dense + (uint64_t)row * a.spec.q_ld;
        q0 = in0 ? __ldg(q + i0) : 0.0f;
        q1 = in1 ? __ldg(q + i1) : 0.0f;
    }
    if (!(fabsf(top) < -neg_inf())) {
        if (lane == 0) {
            a.out_ids[row] = 0xFFFFFFFFu;
            if (a.out_status) {
                a.out_status[row] = LILY_ROW_NONFINITE;
            }
            if (a.kept_n) {
                a.kept_n[row] = 0;
            }
            atomicOr(a.status_word, 1u << LILY_ROW_NONFINITE);
        }
        return;
    }
    const float p0 = in0 ? exp_f32(__fsub_rn(float_of_key(sm->key[lane]), top)) : 0.0f;
    const float p1 = in1 ? exp_f32(__fsub_rn(float_of_key(sm->key[lane + 32u]), top)) : 0.0f;
    w[lane] = p0;
    w[lane + 32u] = p1;
    __syncwarp();
    float c0, c1;
    rank_sums(w, n, c0, c1);
    // Keep rank i >= 1 while the mass before it is below top_p of the total and
    // its weight reaches min_p; the first rank that fails ends the kept set.
    const float limit = __fmul_rn(top_p, __shfl_sync(FULL, c1, 31));
    const float before0 = __shfl_up_sync(FULL, c0, 1), last0 = __shfl_sync(FULL, c0, 31);
    const float up1 = __shfl_up_sync(FULL, c1, 1), before1 = lane == 0u ? last0 : up1;
    const unsigned stop0 = __ballot_sync(FULL, in0 && lane >= 1u && !(before0 < limit && p0 >= min_p));
    const unsigned stop1 = __ballot_sync(FULL, in1 && !(before1 < limit && p1 >= min_p));
    const uint32_t n_keep = stop0 ? (uint32_t)__ffs(stop0) - 1u : stop1 ? (uint32_t)__ffs(stop1) + 31u : n;
    const uint32_t last = n_keep - 1u;
    const float mass = __shfl_sync(FULL, last < 32u ? c0 : c1, (int)(last & 31u));
    const bool kept0 = lane < n_keep, kept1 = lane + 32u < n_keep;
    // First kept rank whose running sum exceeds the target, else the last one.
    auto pick = [&](float s0, float s1, float target) -> uint32_t {
        const unsigned h0 = __ballot_sync(FULL, kept0 && target < s0), h1 = __ballot_sync(FULL, kept1 && target < s1);
        const uint32_t at = h0 ? (uint32_t)__ffs(h0) - 1u : h1 ? (uint32_t)__ffs(h1) + 31u : last;
        return __shfl_sync(FULL, at < 32u ? i0 : i1, (int)(at & 31u));
    };
    float f0 = 0.0f, f1 = 0.0f;
    if (a.kept_n || spec) {
        f0 = __fdiv_rn(p0, mass);
        f1 = __fdiv_rn(p1, mass);
    }
    uint32_t chosen;
    if (!spec) {
        chosen = pick(c0, c1, __fmul_rn(u, mass));
    } else {
        const uint32_t d = ahead.draft;
        const unsigned m0 = __ballot_sync(FULL, kept0 && i0 == d), m1 = __ballot_sync(FULL, kept1 && i1 == d);
        const float p_d = m0 ? __shfl_sync(FULL, f0, __ffs(m0) - 1) : m1 ? __shfl_sync(FULL, f1, __ffs(m1) - 1) : 0.0f;
        float q_d = ahead.q_draft;
        const uint32_t *qi = a.spec.q_ids + (uint64_t)row * KCAP;
        const float *qp = a.spec.q_probs + (uint64_t)row * KCAP;
        if (!a.spec.q_dense) {
            const unsigned e0 = __ballot_sync(FULL, lane < ahead.n_q && ahead.id0 == d);
            const unsigned e1 = __ballot_sync(FULL, lane + 32u < ahead.n_q && ahead.id1 == d);
            q_d = e0 ? __shfl_sync(FULL, ahead.p0, __ffs(e0) - 1) : e1 ? __shfl_sync(FULL, ahead.p1, __ffs(e1) - 1) : 0.0f;
            for (uint32_t j = 64u; j < ahead.n_q && !e0 && !e1; j += 32u) {
                const unsigned e = __ballot_sync(FULL, j + lane < ahead.n_q && __ldg(qi + j + lane) == d);
                if (e) {
                    q_d = __ldg(qp + j + (uint32_t)__ffs(e) - 1u);
                    break;
                }
            }
        }
        if (__fmul_rn(u, q_d) < p_d) {
            chosen = d;
        } else {
            // Residual max(0, p - q) over the kept set, rank order.
            if (!a.spec.q_dense) {
                for (uint32_t j0 = 0; j0 < ahead.n_q; j0 += 32u) {
                    const bool have = j0 + lane < ahead.n_q;
                    const uint32_t e_id = j0 == 0u ? ahead.id0 : j0 == 32u ? ahead.id1 : have ? __ldg(qi + j0 + lane) : 0u;
                    const float e_p = j0 == 0u ? ahead.p0 : j0 == 32u ? ahead.p1 : have ? __ldg(qp + j0 + lane) : 0.0f;
                    const uint32_t m = min(32u, ahead.n_q - j0);
                    for (uint32_t j = 0; j < m; ++j) {
                        const uint32_t id = __shfl_sync(FULL, e_id, (int)j);
                        const float q = __shfl_sync(FULL, e_p, (int)j);
                        q0 = id == i0 ? q : q0;
                        q1 = id == i1 ? q : q1;
                    }
                }
            }
            const float x0 = kept0 ? __fsub_rn(f0, q0) : 0.0f, x1 = kept1 ? __fsub_rn(f1, q1) : 0.0f;
            __syncwarp();
            w[lane] = x0 > 0.0f ? x0 : 0.0f;
            w[lane + 32u] = x1 > 0.0f ? x1 : 0.0f;
            __syncwarp();
            float r0, r1;
            rank_sums(w, n_keep, r0, r1);
            const float r_total = __shfl_sync(FULL, last < 32u ? r0 : r1, (int)(last & 31u));
            const float u2 = a.spec.u_resid ? __ldg(a.spec.u_resid + row) : uniform_for(seed, step | 0x80000000u);
            chosen = r_total > 0.0f ? pick(r0, r1, __fmul_rn(u2, r_total)) : pick(c0, c1, __fmul_rn(u2, mass));
        }
    }
    if (lane == 0) {
        a.out_ids[row] = chosen;
        if (a.out_status) {
            a.out_status[row] = LILY_ROW_OK;
        }
        if (counts_draw && chosen < a.vocab) {
            // src/kernels/metal/sample.metal:509-511: the draw is counted.
            atomicAdd(a.counts_table + (uint64_t)slot * a.vocab + chosen, 1u);
            atomicOr(a.seen_table + (uint64_t)slot * a.seen_words + (chosen >> 5), 1u << (chosen & 31u));
        }
    }
    if (a.kept_n) {
        if (kept0) {
            a.kept_ids[(uint64_t)row * a.kept_ld + lane] = i0;
            a.kept_probs[(uint64_t)row * a.kept_ld + lane] = f0;
        }
        if (kept1) {
            a.kept_ids[(uint64_t)row * a.kept_ld + lane + 32u] = i1;
            a.kept_probs[(uint64_t)row * a.kept_ld + lane + 32u] = f1;
        }
        if (lane == 0) {
            a.kept_n[row] = n_keep;
        }
    }
}

// Grid (blocks per row, rows), clusters of (blocks per row), NT threads, of which
// SPL_NT do the work. BPS: blocks per SM the registers are cut for; with one, a
// block whose share fits one bucket keeps it in registers.
template <typename T, uint32_t MAXR, int BPS>
__global__ void __launch_bounds__(NT, BPS) split_rows_kernel(const __grid_constant__ SplitArgs<MAXR> ca) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr uint32_t NONE = 0xFFFFFFFFu;
    constexpr uint32_t PER = Piece<T>::PER, SHIFT = Piece<T>::SHIFT, SPL_U = split_u(BPS);
    const KArgs &a = ca.a;
    extern __shared__ uint4 smem_raw[];
    SmemFixed *sm = reinterpret_cast<SmemFixed *>(smem_raw);
    SplitSmem *ss = reinterpret_cast<SplitSmem *>(sm + 1);
    uint32_t *marks = reinterpret_cast<uint32_t *>(ss + 1);
    float *bmax = reinterpret_cast<float *>(marks + ca.mark_words);  // [buckets][SPL_NT]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t rank = blockIdx.x, log_blocks = ca.log_blocks, blocks = 1u << log_blocks;
    const uint32_t row = a.row0 + blockIdx.y;
    const uint32_t vocab = a.vocab;
    LILY_STAMP(PH_ENTRY);

    // What needs no input comes first (see sample_row on the launch attribute).
    if (tid == 0) {
        ss->n_flagged = 0;
        ss->n_hits = 0;
        ss->n_listed = 0;
        ss->n_sent = 0;
        ss->n_live = 0;
        ss->hard = 0;
        ss->bound_key = 0;
        if (blocks > 1u) {
            const uint32_t pool_bar = (uint32_t)__cvta_generic_to_shared(&ss->mbar_pool);
            const uint32_t cand_bar = (uint32_t)__cvta_generic_to_shared(&ss->mbar_cand);
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(pool_bar) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(cand_bar), "r"(blocks) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    for (uint32_t w = tid; w < ca.mark_words / 4u; w += NT) {
        reinterpret_cast<uint4 *>(marks)[w] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    if (blocks > 1u) {
        // (Waited for before the first store into another block.)
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const T *row_ptr = reinterpret_cast<const T *>(a.logits) + (uint64_t)row * a.logits_ld;
    const uint32_t skip = (uint32_t)(reinterpret_cast<uintptr_t>(row_ptr) & 15u) / (uint32_t)sizeof(T);
    // The first block draws the row alone with the general row code, all NT threads.
    auto draw_alone = [&]() {
        KArgs whole = a;
        whole.n_slices = 1;
        if (ca.inline_params) {
            if (tid == 0) {
                const RowIn &in = ca.in[row];
                lily_sampling_params_t P;
                P.temperature = (in.flags & ROW_GREEDY) ? 0.0f : in.temp;
                P.top_k = in.k;
                P.top_p = in.top_p;
                P.min_p = in.min_p;
                P.presence_penalty = in.presence;
                P.frequency_penalty = in.frequency;
                P.repetition_penalty = in.rep;
                P.reserved = 0;
                P.seed = in.seed;
                ca.spill_params[row] = P;
                ca.spill_steps[row] = in.step;
            }
            whole.params = ca.spill_params;
            whole.steps = ca.spill_steps;
        }
        if (ca.inline_slots) {
            if (tid == 0) {
                ca.spill_slots[row] = ca.slots[row];
            }
            whole.count_slots = ca.spill_slots;
        }
        if (ca.inline_history) {
            if (tid == 0) {
                ca.spill_history[row] = ca.inline_history - 1u;
            }
            whole.history_len = ca.spill_history;
        }
        __threadfence();
        __syncthreads();
        if (skip == 0u) {
            sample_whole_row<T, true>(whole, row);
        } else {
            sample_whole_row<T, false>(whole, row);
        }
    };
    // What the first block's waiting warps are told, at barrier 2: the row is done, it
    // is drawn alone, or (only to the warps that work) more hands are needed; in the
    // last case there is a second verdict. Threads that wait return only if they are
    // needed.
    enum { DONE = 0, ALONE = 1, HANDS = 2 };
    auto wait_verdict = [&](uint32_t at) -> bool {
        asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
        const uint32_t v = ss->verdict[at];
        if (v == ALONE) {
            draw_alone();
        }
        return v == HANDS;
    };
    auto verdict = [&](uint32_t at, uint32_t v) {
        if (tid == 0) {
            ss->verdict[at] = v;
        }
        if (v == ALONE) {
            asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
            draw_alone();
        } else {
            asm volatile("bar.arrive 2, %0;" ::"n"(NT) : "memory");
        }
    };
    if (tid >= SPL_NT) {
        if (rank == 0u) {
            if (ca.share && blocks > 1u) {
                // (Threads that stay have to come to the cluster's second meeting as well.)
                asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
                asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            }
            if (wait_verdict(0u)) {
                wait_verdict(1u);
            }
        }
        return;
    }
    // ---- the first bucket is asked for before anything is known about the row
    const uint4 *vec0 = reinterpret_cast<const uint4 *>(row_ptr - skip) + lane;
    const uint32_t pieces = split_pieces(vocab, skip, PER);
    const uint32_t pieces_here = (pieces - rank + blocks - 1u) >> log_blocks;
    const uint32_t buckets = split_buckets(pieces_here, SPL_U);
    const uint32_t whole_end = (vocab + skip) >> SHIFT;  // pieces from here on stick out of the row
    auto load_piece = [&](uint32_t j) -> uint4 {         // this lane's vector of the block's piece j
        const uint32_t t = (j << log_blocks) | rank;
        if (t < whole_end && (t != 0u || skip == 0u)) {
            return __ldg(vec0 + t * 32u);
        }
        return edge_vec<T>(row_ptr, vocab, skip, t * 32u + lane);
    };
    // The row's first history ids go first. (Their number is not known yet; the row
    // has room for history_ld of them.)
    constexpr uint32_t HU = BPS == 1 ? 4u : 2u;
    const uint32_t *hist = a.history_ids + (uint64_t)row * a.history_ld;
    const bool hist_vec = a.history_ids != nullptr && (reinterpret_cast<uintptr_t>(hist) & 15u) == 0u;
    const uint4 *h4 = reinterpret_cast<const uint4 *>(hist);
    const uint4 no_ids = make_uint4(NONE, NONE, NONE, NONE);
    // Either every block looks at the whole list for the ids of its share, or (a long
    // list, or one that is counted) a part of the list each, for all blocks.
    const uint32_t h_step = ca.share ? SPL_NT << log_blocks : SPL_NT, h_first = ca.share ? rank * SPL_NT + tid : tid;
    uint4 hx[HU];
    const uint32_t room4 = hist_vec ? (uint32_t)min(a.history_ld, (uint64_t)a.max_history) >> 2 : 0u;
#pragma unroll
    for (uint32_t i = 0; i < HU; ++i) {
        const uint32_t at = h_first + i * h_step;
        hx[i] = at < room4 ? __ldg(h4 + at) : no_ids;
    }
    uint4 q[SPL_U];
#pragma unroll
    for (uint32_t i = 0; i < SPL_U; ++i) {
        q[i] = load_piece(warp + SPL_WARPS * i);
    }

    // ---- the row's parameters
    RowIn in;
    uint32_t hist_len = 0, slot = 0;
    int32_t forced = -1;
    if (a.force_greedy) {
        in.temp = 1.0f;
        in.rep = in.top_p = 1.0f;
        in.presence = in.frequency = in.min_p = in.u = 0.0f;
        in.k = 1;
        in.flags = ROW_GREEDY;
        in.step = 0;
        in.seed = 0;
    } else if (ca.inline_params) {
        in = ca.in[row];
    } else {
        const uint2 *pp = reinterpret_cast<const uint2 *>(a.params + row);
        const uint2 w0 = __ldg(pp), w1 = __ldg(pp + 1), w2 = __ldg(pp + 2), w3 = __ldg(pp + 3), w4 = __ldg(pp + 4);
        lily_sampling_params_t P;
        P.temperature = __uint_as_float(w0.x);
        P.top_k = w0.y;
        P.top_p = __uint_as_float(w1.x);
        P.min_p = __uint_as_float(w1.y);
        P.presence_penalty = __uint_as_float(w2.x);
        P.frequency_penalty = __uint_as_float(w2.y);
        P.repetition_penalty = __uint_as_float(w3.x);
        P.reserved = w3.y;
        P.seed = (uint64_t)w4.x | ((uint64_t)w4.y << 32);
        in = row_in(P, (!a.uniforms && a.steps) ? __ldg(a.steps + row) : 0u);
    }
    if (a.history_ids) {
        hist_len = ca.inline_history ? ca.inline_history - 1u : a.history_len ? __ldg(a.history_len + row) : 0u;
    }
    const uint32_t n_bias = (a.bias_ids && a.bias_len) ? __ldg(a.bias_len + row) : 0u;
    const uint32_t n_ban = (a.ban_ids && a.ban_len) ? __ldg(a.ban_len + row) : 0u;
    if (a.forced_ids) {
        forced = __ldg(a.forced_ids + row);
    }
    const bool table_mode = ca.inline_slots != 0u || a.count_slots != nullptr;
    if (table_mode) {
        slot = ca.inline_slots ? ca.slots[row] : __ldg(a.count_slots + row);
    }
    const uint32_t n_sp = n_bias + n_ban;
    uint32_t status = LILY_ROW_OK;
    if (forced >= 0) {
        status = LILY_ROW_FORCED;
    } else if (in.flags & ROW_BAD) {
        status = LILY_ROW_PARAMS;
    } else if (hist_len > a.max_history || (a.history_ld != 0u && hist_len > a.history_ld) ||  // (a pitch of 0:
               n_bias > a.max_list || (a.bias_ld != 0u && n_bias > a.bias_ld) ||               // one list for all)
               n_ban > a.max_list || (a.ban_ld != 0u && n_ban > a.ban_ld)) {
        status = LILY_ROW_LIST;
    }
    const bool use_pen = (in.flags & ROW_PEN) != 0u, need_counts = (in.flags & ROW_COUNTS) != 0u;
    const bool list_mode = use_pen && !table_mode;
    if (!list_mode) {
        hist_len = 0;
    }
    const uint32_t extra_len = list_mode ? a.extra_len : 0u;
    const uint32_t k = in.k;
    const bool wide = k > SPL_SMALL_K;
    const uint32_t mark_mode = ca.mark_mode;
    // Decided alike by every block of the cluster: rows that end here.
    const bool general = (in.flags & ROW_RAISES) || n_sp > SP_SMEM ||
                         (n_sp != 0u && mark_mode == MARK_BITS) ||
                         (list_mode && need_counts && (mark_mode != MARK_COUNTS || hist_len + extra_len > SPL_COUNT_MAX)) ||
                         (wide && (row < a.spec.n_spec || blocks * SPL_NT < 2u * k));
    if (status != LILY_ROW_OK || general) {
        if (status != LILY_ROW_OK && rank == 0u && tid == 0) {
            a.out_ids[row] = status == LILY_ROW_FORCED ? (uint32_t)forced : 0xFFFFFFFFu;
            if (a.out_status) {
                a.out_status[row] = status;
            }
            if (a.kept_n) {
                a.kept_n[row] = 0;
            }
            if (status != LILY_ROW_FORCED) {
                atomicOr(a.status_word, 1u << (status & 31u));
            }
        }
        if (rank == 0u) {
            verdict(0u, status == LILY_ROW_OK ? ALONE : DONE);
        }
        return;
    }
    const bool argmax_mode = (in.flags & ROW_GREEDY) && !use_pen && n_sp == 0u;
    const bool draws = rank == 0u && warp == 0u;  // the warp that ends up with the row
    SpecAhead ahead;
    ahead.draft = draws && row < a.spec.n_spec ? __ldg(a.spec.draft_ids + row) : 0u;
    const float u_row = !draws ? 0.0f : a.uniforms ? __ldg(a.uniforms + row) : in.u;

    // ---- 1. the stream: maxima and marks
    // Which block an id belongs to, and its place in that block's marks.
    auto place_of = [&](uint32_t id, uint32_t &at) -> uint32_t {
        const uint32_t s = id + skip, t = s >> SHIFT;
        at = ((t >> log_blocks) << SHIFT) | (s & (Piece<T>::LOGITS - 1u));
        return id < vocab ? t & (blocks - 1u) : NONE;
    };
    uint8_t *mark8 = reinterpret_cast<uint8_t *>(marks);
    uint16_t *mark16 = reinterpret_cast<uint16_t *>(marks);
    const uint32_t marks_at = (uint32_t)__cvta_generic_to_shared(marks);
    // One id of the history; `WAY` says how (chosen once per row, not per id). Rows
    // that need no multiplicity: any thread may write the same.
    enum { OWN_BYTE, OWN_SHORT, OWN_BIT, OWN_COUNT, ANY_BYTE, ANY_SHORT, ANY_BIT, ANY_COUNT };
    auto mark_id = [&](auto way, uint32_t id) {
        constexpr int WAY = decltype(way)::value;
        uint32_t at, to;
        const uint32_t owner = place_of(id, at);
        if (WAY < ANY_BYTE) {
            if (owner == rank) {
                if (WAY == OWN_BYTE) {
                    mark8[at] = 1;
                } else if (WAY == OWN_SHORT) {
                    mark16[at] = 1;
                } else if (WAY == OWN_BIT) {
                    atomicOr(marks + (at >> 5), 1u << (at & 31u));
                } else {
                    atomicAdd(marks + (at >> 1), 1u << (16u * (at & 1u)));
                }
            }
        } else if (WAY != ANY_COUNT) {
            if (owner != NONE) {
                const uint32_t off = WAY == ANY_BYTE ? at : WAY == ANY_SHORT ? at * 2u : (at >> 5) * 4u;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(marks_at + off), "r"(owner));
                if (WAY == ANY_BYTE) {
                    asm volatile("st.shared::cluster.u8 [%0], %1;" ::"r"(to), "h"((unsigned short)1) : "memory");
                } else if (WAY == ANY_SHORT) {
                    asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(to), "h"((unsigned short)1) : "memory");
                } else {
                    asm volatile("red.shared::cluster.or.b32 [%0], %1;" ::"r"(to), "r"(1u << (at & 31u)) : "memory");
                }
            }
        } else {
            // Real histories repeat a few ids very often: the lanes that hold the same id as
            // the first of a warp add up to one atomic. Every lane of the warp is here.
            const uint32_t first = __shfl_sync(FULL, id, 0);
            const bool same = id == first;
            const uint32_t n = (uint32_t)__popc(__ballot_sync(FULL, same));
            if (owner != NONE && (!same || lane == 0u)) {
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(marks_at + (at >> 1) * 4u), "r"(owner));
                asm volatile("red.shared::cluster.add.u32 [%0], %1;" ::"r"(to), "r"((same ? n : 1u) << (16u * (at & 1u)))
                             : "memory");
            }
        }
    };
    // Calls f with the row's way of marking.
    auto with_way = [&](bool own, auto f) {
        if (own) {
            if (mark_mode == MARK_BYTES) {
                f(std::integral_constant<int, OWN_BYTE>());
            } else if (mark_mode == MARK_BITS) {
                f(std::integral_constant<int, OWN_BIT>());
            } else if (need_counts) {
                f(std::integral_constant<int, OWN_COUNT>());
            } else {
                f(std::integral_constant<int, OWN_SHORT>());
            }
        } else if (mark_mode == MARK_BYTES) {
            f(std::integral_constant<int, ANY_BYTE>());
        } else if (mark_mode == MARK_BITS) {
            f(std::integral_constant<int, ANY_BIT>());
        } else if (need_counts) {
            f(std::integral_constant<int, ANY_COUNT>());
        } else {
            f(std::integral_constant<int, ANY_SHORT>());
        }
    };
    const uint32_t n4 = hist_vec ? hist_len >> 2 : 0u;
    const uint32_t h_rounds = (n4 + h_step - 1u) / h_step;  // 16-byte loads of ids per thread
    const uint32_t h_per = buckets == 1u ? h_rounds : (h_rounds + buckets - 1u) / buckets;  // ... per bucket
    const bool shared_list = ca.share != 0u && n4 != 0u;
    if (shared_list) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // the other blocks' marks are cleared
    }
    for (uint32_t j = tid; j < n_sp; j += SPL_NT) {
        sm->sp_ids[j] = j < n_bias ? a.bias_ids[(uint64_t)row * a.bias_ld + j]
                                   : a.ban_ids[(uint64_t)row * a.ban_ld + (j - n_bias)];
        sm->sp_vals[j] = j < n_bias ? a.bias_vals[(uint64_t)row * a.bias_ld + j] : 0.0f;
    }
    float best = neg_inf(), bm = neg_inf();
    uint32_t best_j = NONE;
    bool bad = false;
    uint4 best_v = make_uint4(0, 0, 0, 0);
    for (uint32_t b = 0;;) {
        const uint32_t h_end = min(h_rounds, (b + 1u) * h_per);
        for (uint32_t h_at = min(h_rounds, b * h_per); h_at < h_end; h_at += HU) {
            if (h_at != 0u) {
#pragma unroll
                for (uint32_t i = 0; i < HU; ++i) {
                    const uint32_t at = (h_at + i) * h_step + h_first;
                    hx[i] = (at < n4 && h_at + i < h_end) ? __ldg(h4 + at) : no_ids;
                }
            } else {
#pragma unroll
                for (uint32_t i = 0; i < HU; ++i) {
                    const uint32_t at = i * h_step + h_first;
                    if (at >= n4 || i >= h_end) {
                        hx[i] = no_ids;
                    } else if (at >= room4) {
                        hx[i] = __ldg(h4 + at);
                    }
                }
            }
            with_way(ca.share == 0u, [&](auto way) {
#pragma unroll
                for (uint32_t i = 0; i < HU; ++i) {
                    mark_id(way, hx[i].x);
                    mark_id(way, hx[i].y);
                    mark_id(way, hx[i].z);
                    mark_id(way, hx[i].w);
                }
            });
        }
        if (shared_list && b + 1u == buckets) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        }
        bm = neg_inf();
#pragma unroll
        for (uint32_t i = 0; i < SPL_U; ++i) {
            const float m = vec_max<T>(q[i]);
            bm = max_nan_f32(bm, m);
            if (m > best) {
                best = m;
                best_j = b * SPL_U + i;
                best_v = q[i];
            }
            if (b + 1u < buckets) {  // (asked for as soon as its place is free)
                q[i] = load_piece(warp + SPL_WARPS * ((b + 1u) * SPL_U + i));
            }
        }
        bad = bad || bm != bm;
        if (buckets != 1u) {
            bmax[b * SPL_NT + tid] = bm;
        }
        if (++b == buckets) {
            break;
        }
    }
    bool joined = shared_list;  // the other blocks of the cluster are known to be running
    if (argmax_mode) {
        // Nothing adjusts a logit: every warp sends its best, equal values in favour of
        // the lowest id (within a thread the ids rise).
        uint32_t key = 0u, id = NONE;
        if (best_j != NONE) {
            uint32_t e = 0;
#pragma unroll
            for (int i = (int)PER - 1; i >= 0; --i) {
                e = vec_get<T>(best_v, (uint32_t)i) == best ? (uint32_t)i : e;
            }
            key = key_of(__fadd_rn(best, 0.0f));  // (the two zeros tie: src/kernels/metal/elementwise.metal:145-150)
            id = ((((warp + SPL_WARPS * best_j) << log_blocks | rank) * 32u + lane) * PER + e) - skip;
        }
        if (bad) {
            key = SPL_NAN_KEY;
            id = 0u;
        }
        const uint32_t m = __reduce_max_sync(FULL, key);
        const uint32_t mi = __reduce_min_sync(FULL, key == m ? id : NONE);
        if (blocks > 1u) {
            if (!joined) {
                asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            }
            if (lane == 0) {
                put_2u32(peer_smem(&ss->pool[2u * (rank * SPL_WARPS + warp)], 0), m, mi, peer_smem(&ss->mbar_pool, 0));
            }
        } else {
            if (lane == 0) {
                ss->pool[2u * warp] = m;
                ss->pool[2u * warp + 1u] = mi;
            }
        }
        if (rank != 0u) {
            return;
        }
        bool ok = true;
        if (blocks > 1u) {
            if (tid == 0) {
                arrive_expect(peer_smem(&ss->mbar_pool, 0), blocks * SPL_WARPS * 8u);
            }
            ok = warp != 0u || wait_first_phase(&ss->mbar_pool);
        } else {
            spl_sync();
        }
        if (warp != 0u) {
            wait_verdict(0u);
            return;
        }
        uint32_t top = 0u, at = NONE;
        for (uint32_t i = lane; i < blocks * SPL_WARPS; i += 32u) {
            const uint32_t x = ss->pool[2u * i], y = ss->pool[2u * i + 1u];
            if (x > top || (x == top && y < at)) {
                top = x;
                at = y;
            }
        }
        const uint32_t win = __reduce_max_sync(FULL, top);
        const uint32_t win_id = __reduce_min_sync(FULL, top == win ? at : NONE);
        // (Nothing but -inf, or a NaN somewhere: the general code's rules.)
        if (!__all_sync(FULL, ok) || win_id == NONE || win == SPL_NAN_KEY) {
            verdict(0u, ALONE);
            return;
        }
        if (lane == 0) {
            a.out_ids[row] = win_id;
            if (a.out_status) {
                a.out_status[row] = LILY_ROW_OK;
            }
            if (a.kept_n) {
                a.kept_n[row] = 1;
                a.kept_ids[(uint64_t)row * a.kept_ld] = win_id;
                a.kept_probs[(uint64_t)row * a.kept_ld] = 1.0f;
            }
        }
        verdict(0u, DONE);
        LILY_STAMP(PH_END);
        return;
    }
    const bool marked = hist_len + extra_len != 0u;
    if (marked) {
        // What the 16-byte loads left out, and ids drawn earlier in this step.
        const uint32_t rest = hist_len - n4 * 4u, more = rest + extra_len;
        for (uint32_t i = tid; i < more; i += SPL_NT) {
            const uint32_t id = i < rest ? __ldg(hist + n4 * 4u + i) : __ldcg(a.extra_ids + (i - rest));
            with_way(true, [&](auto way) { mark_id(way, id); });
        }
        if (shared_list) {
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every block's marks have arrived
        }
        spl_sync();
    }
    if (draws && row < a.spec.n_spec) {
        spec_ahead(a.spec, row, vocab, ahead);
    }
    LILY_STAMP(PH_PASS1);

    // The logit, as it was before the division by the temperature, with the
    // penalties for an id that was emitted `count` times.
    auto penalised = [&](float x, uint32_t count) -> float {
        if (count != 0u) {
            x = x > 0.0f ? __fdiv_rn(x, in.rep) : __fmul_rn(x, in.rep);
            x = __fsub_rn(x, __fadd_rn(in.presence, __fmul_rn(in.frequency, (float)count)));
        }
        return x;
    };
    // The mark of an id of this block's share: how often it was emitted (without a
    // frequency penalty any number but 0 will do), and LISTED if it is on a bias or
    // ban list.
    constexpr uint32_t LISTED = 0x80000000u;
    auto mark_of = [&](uint32_t id) -> uint32_t {
        uint32_t m = 0;
        if (marked || n_sp != 0u) {
            uint32_t at;
            place_of(id, at);
            if (mark_mode == MARK_BYTES) {
                const uint32_t x = mark8[at];
                m = (x & 0x7Fu) | (x >> 7 << 31);
            } else if (mark_mode == MARK_COUNTS) {
                const uint32_t x = mark16[at];
                m = (x & 0x7FFFu) | (x >> 15 << 31);
            } else {
                m = (marks[at >> 5] >> (at & 31u)) & 1u;
            }
        }
        if (use_pen && table_mode) {
            if (need_counts) {  // (a slot's bits say no more than its counts do)
                m |= __ldcg(a.counts_table + (uint64_t)slot * vocab + id);
            } else {
                m |= (__ldcg(a.seen_table + (uint64_t)slot * a.seen_words + (id >> 5)) >> (id & 31u)) & 1u;
            }
        }
        return m;
    };
    if (n_sp != 0u) {
        // The ids on the bias or ban list that are this block's, each by the thread of
        // its first entry: marked, so that the stream's candidates leave them out, and
        // a candidate of its own with its bias entries added in list order (a banned
        // id is none).
        if (!marked) {
            spl_sync();  // (the lists are in shared memory)
        }
        for (uint32_t j = tid; j < n_sp; j += SPL_NT) {
            const uint32_t id = sm->sp_ids[j];
            uint32_t at;
            if (place_of(id, at) != rank) {
                continue;
            }
            float x = widen(row_ptr[id]);
            bool first = true, banned = false;
#pragma unroll 4
            for (uint32_t e = 0; e < n_sp; ++e) {
                if (sm->sp_ids[e] == id) {
                    first = first && e >= j;
                    banned = banned || e >= n_bias;
                    if (e < n_bias) {
                        x = __fadd_rn(x, sm->sp_vals[e]);
                    }
                }
            }
            if (first) {
                if (mark_mode == MARK_BYTES) {
                    mark8[at] |= 0x80u;
                } else {
                    mark16[at] |= 0x8000u;
                }
                if (!banned) {
                    const uint32_t to = atomicAdd(&ss->n_listed, 1u);
                    sm->tkey[to] = __float_as_uint(x);
                    sm->tid[to] = id;
                }
            }
        }
        spl_sync();
    }

    // ---- 2. the bound
    auto id_at = [&](uint32_t j, uint32_t e) -> uint32_t {  // element e of this lane's vector of piece j of the block
        return ((((j << log_blocks) | rank) * 32u + lane) * PER + e) - skip;
    };
    // This thread's best logit, adjusted but for the temperature (which keeps the order).
    uint32_t key = 0u;
    if (best_j != NONE) {
        float x = best;
        if (use_pen || n_sp != 0u) {
            uint32_t e = 0;
#pragma unroll
            for (int i = (int)PER - 1; i >= 0; --i) {
                e = vec_get<T>(best_v, (uint32_t)i) == best ? (uint32_t)i : e;
            }
            const uint32_t m = mark_of(id_at(warp + SPL_WARPS * best_j, e));
            x = (m & LISTED) ? neg_inf() : penalised(x, m);
        }
        key = key_of(__fadd_rn(x, 0.0f));
    }
    if (bad) {
        ss->hard = 1;  // (read after the next barrier)
    }
    if (blocks > 1u && !joined) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    uint32_t bound_key = 0;
    float reach = 0.0f;  // the largest magnitude that went into the bound's arithmetic
    if (!wide) {
        // Every warp of the cluster gives its best keys: so many that a warp hardly ever
        // has more of the row's best k than it gives (k / warps of them on average).
        const uint32_t rounds = ca.rounds_of(k), n = (blocks * SPL_WARPS) * rounds;
        for (uint32_t r = 0; r < rounds; ++r) {
            const uint32_t m = __reduce_max_sync(FULL, key);
            const unsigned who = __ballot_sync(FULL, key == m);
            if (lane == (uint32_t)__ffs(who) - 1u) {
                key = 0u;
            }
            // (The place in the pool takes the key's last eight bits: no two keys are the same, and
            // a bound may be a little lower than it could be.)
            const uint32_t to = (rank * SPL_WARPS + warp) * rounds + r, placed = (m & ~255u) | to;
            if (blocks > 1u) {
                if (lane < blocks) {
                    put_u32(peer_smem(&ss->pool[to], lane), placed, peer_smem(&ss->mbar_pool, lane));
                }
            } else if (lane == 0) {
                ss->pool[to] = placed;
            }
        }
        if (blocks > 1u) {
            if (tid == 0) {
                arrive_expect(peer_smem(&ss->mbar_pool, rank), n * 4u);
            }
            if (!wait_first_phase(&ss->mbar_pool)) {
                ss->hard = 1;
            }
        } else {
            spl_sync();
        }
        // The k-th largest of them: up to four threads share the count of a key's betters.
        if (k == 1u) {
            uint32_t m = 0;
            for (uint32_t i = lane; i < n; i += 32u) {
                m = max(m, ss->pool[i]);
            }
            bound_key = __reduce_max_sync(FULL, m);
        } else {
            const uint32_t log_team = n <= SPL_NT / 4u ? 2u : n <= SPL_NT / 2u ? 1u : 0u;
            const uint32_t i = tid >> log_team, part = tid & ((1u << log_team) - 1u);
            const uint32_t mine = i < n ? ss->pool[i] : 0u;
            const uint4 *four = reinterpret_cast<const uint4 *>(ss->pool);
            uint32_t above = 0;
#pragma unroll 4
            for (uint32_t j = part; j < n / 4u; j += 1u << log_team) {
                const uint4 o = four[j];
                above += (o.x > mine ? 1u : 0u) + (o.y > mine ? 1u : 0u);
                above += (o.z > mine ? 1u : 0u) + (o.w > mine ? 1u : 0u);
            }
            if (log_team != 0u) {
                above += __shfl_xor_sync(FULL, above, 1);
                if (log_team == 2u) {
                    above += __shfl_xor_sync(FULL, above, 2);
                }
            }
            if (i < n && above == k - 1u) {
                ss->bound_key = mine;
            }
            spl_sync();
            bound_key = ss->bound_key;
        }
        bound_key &= ~255u;
    } else {
        // The maxima of the whole cluster, 32 bins per unit under the largest.
        if (blocks > 1u) {
            if (tid == 0) {
                arrive_expect(peer_smem(&ss->mbar_pool, rank), blocks * SPL_NT * 4u);
            }
            for (uint32_t r = 0; r < blocks; ++r) {
                put_u32(peer_smem(&ss->tmax[rank * SPL_NT + tid], r), key, peer_smem(&ss->mbar_pool, r));
            }
        } else {
            ss->tmax[tid] = key;
        }
        for (uint32_t b = tid; b < TH_BINS; b += SPL_NT) {
            sm->thist[b] = 0;
        }
        if (tid == 0) {
            ss->bin = NONE;
        }
        if (blocks > 1u && !wait_first_phase(&ss->mbar_pool)) {
            ss->hard = 1;
        }
        spl_sync();
        uint32_t keys[SPL_MAX_BLOCKS], m = 0;
#pragma unroll
        for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
            keys[r] = r < blocks ? ss->tmax[r * SPL_NT + tid] : 0u;
            m = max(m, keys[r]);
        }
        m = __reduce_max_sync(FULL, m);
        if (lane == 0) {
            sm->warp_sums[SPL_WARPS + warp] = m;
        }
        spl_sync();
        const float top = float_of_key(__reduce_max_sync(FULL, sm->warp_sums[SPL_WARPS + (lane & (SPL_WARPS - 1u))]));
        reach = fabsf(top);
        constexpr float BINS_PER_UNIT = 32.0f;
#pragma unroll
        for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
            const float d = __fmul_rn(__fsub_rn(top, float_of_key(keys[r])), BINS_PER_UNIT);
            if (keys[r] != 0u && d < (float)TH_BINS) {
                atomicAdd(&sm->thist[(uint32_t)d], 1u);
            }
        }
        spl_sync();
        constexpr uint32_t BPT = TH_BINS / SPL_NT;
        uint32_t c[BPT], sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < BPT; ++j) {
            c[j] = sm->thist[tid * BPT + j];
            sum += c[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) {
                incl += t;
            }
        }
        if (lane == 31u) {
            sm->warp_sums[warp] = incl;
        }
        spl_sync();
        uint32_t cum = incl - sum;
#pragma unroll
        for (uint32_t w = 0; w < SPL_WARPS; ++w) {
            cum += w < warp ? sm->warp_sums[w] : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < BPT; ++j) {
            if (cum < k && k <= cum + c[j]) {
                ss->bin = tid * BPT + j;
            }
            cum += c[j];
        }
        spl_sync();
        // The lower edge of the k-th maximum's bin (the rounding of d is covered below).
        const uint32_t bin = ss->bin;
        bound_key = bin == NONE ? 0u : key_of(__fsub_rn(top, __fdiv_rn((float)(bin + 1u), BINS_PER_UNIT)));
    }
    LILY_STAMP(PH_FIRST_THRESHOLD);
    // At least k logits of the row have a value (before the division) of `bound`
    // or more, so one of the best k divides to bound / T or more: it lies at most
    // two rounding steps under the bound (T * 2^-149 apart where quotients are
    // subnormal).
    const float bound = float_of_key(bound_key);
    const float slack = __fadd_rn(__fmul_rn(fmaxf(reach, fabsf(bound)), 4.76837158203125e-7f),
                                  __fmul_rn(in.temp, 2.8025969e-45f));
    const float least = __fsub_rn(bound, slack);
    // Fewer than k finite maxima, or quotients that overflow: the general code.
    const bool hopeless = bound_key == 0u || !(least > -3.0e38f) || !(__fdiv_rn(least, in.temp) > -3.0e38f);

    // ---- 3. the vectors that reach the bound ...
    uint4 *hits = reinterpret_cast<uint4 *>(sm->lkey);  // over lkey and lid
    static_assert(SPL_HITS * 16u <= 2u * LCAP * 4u, "");
    auto hit = [&](const uint4 &x, uint32_t first_id) {
        const uint32_t to = atomicAdd(&ss->n_hits, 1u);
        if (to < SPL_HITS) {
            hits[to] = x;
            ss->hit_at[to] = first_id;
        }
    };
    if (hopeless) {
        ss->hard = 1;
    } else if (BPS == 1 && buckets == 1u) {
        if (bm >= least) {
#pragma unroll
            for (uint32_t i = 0; i < SPL_U; ++i) {
                if (vec_max<T>(q[i]) >= least) {
                    hit(q[i], id_at(warp + SPL_WARPS * i, 0u));
                }
            }
        }
    } else {
        for (uint32_t b = 0; b < buckets; ++b) {
            const bool over = (buckets == 1u ? bm : bmax[b * SPL_NT + tid]) >= least;
            const unsigned who = __ballot_sync(FULL, over);
            if (who != 0u) {
                uint32_t at = 0;
                if (lane == 0) {
                    at = atomicAdd(&ss->n_flagged, (uint32_t)__popc(who));
                }
                at = __shfl_sync(FULL, at, 0) + __popc(who & ((1u << lane) - 1u));
                if (over && at < SPL_FLAGGED) {
                    ss->flagged[at] = (uint16_t)(b * SPL_NT + tid);
                }
            }
        }
        spl_sync();
        const uint32_t n_flagged = ss->n_flagged;
        if (n_flagged > SPL_FLAGGED) {
            ss->hard = 1;
        } else {
            // (Each of them again, from L2: a vector per thread.)
            for (uint32_t i = tid; i < n_flagged * SPL_U; i += SPL_NT) {
                const uint32_t f = ss->flagged[i / SPL_U], owner = f % SPL_NT;
                const uint32_t j = (owner >> 5) + SPL_WARPS * ((f / SPL_NT) * SPL_U + i % SPL_U);
                const uint32_t t = (j << log_blocks) | rank, v = t * 32u + (owner & 31u);
                const uint4 x = (t < whole_end && (t != 0u || skip == 0u)) ? __ldg(vec0 - lane + v)
                                                                           : edge_vec<T>(row_ptr, vocab, skip, v);
                if (vec_max<T>(x) >= least) {
                    hit(x, v * PER - skip);
                }
            }
        }
    }
    spl_sync();
    LILY_STAMP(PH_LISTS);
    // ... and their logits, a thread each: what reaches the bound is adjusted, divided
    // and sent to the first block, and so are the ids of the bias list.
    const uint32_t cap = CAP >> log_blocks;
    const uint32_t n_hits = ss->n_hits;
    uint2 *cand = reinterpret_cast<uint2 *>(sm->key);  // over key and id: CAP of them, a region per block
    const uint32_t bar = blocks > 1u ? peer_smem(&ss->mbar_cand, 0) : 0u;
    const uint32_t cand_at = blocks > 1u ? peer_smem(cand + rank * cap, 0) : 0u;
    if (n_hits <= SPL_HITS && ss->hard == 0u) {
        const uint32_t n_elem = n_hits * PER, n_all = n_elem + ss->n_listed;
        for (uint32_t i = tid; i < n_all; i += SPL_NT) {
            uint32_t id;
            float x;
            if (i < n_elem) {
                const T l = reinterpret_cast<const T *>(hits)[i];
                x = widen(l);
                id = ss->hit_at[i / PER] + i % PER;
                if (!(x >= least) || id >= vocab) {
                    continue;
                }
            } else {
                x = __uint_as_float(sm->tkey[i - n_elem]);
                id = sm->tid[i - n_elem];
            }
            if (use_pen || n_sp != 0u) {
                const uint32_t m = mark_of(id);
                if ((m & LISTED) && i < n_elem) {
                    continue;  // (its own entry stands for it)
                }
                x = penalised(x, m & ~LISTED);
            }
            const float quot = __fdiv_rn(x, in.temp);
            if (x >= least || quot != quot) {
                const uint32_t to = atomicAdd(&ss->n_sent, 1u);
                if (to < cap) {
                    const uint32_t key_q = quot != quot ? SPL_NAN_KEY : key_of(quot);
                    if (blocks > 1u) {
                        put_2u32(cand_at + to * 8u, key_q, id, bar);
                    } else {
                        cand[to] = make_uint2(key_q, id);
                    }
                }
            }
        }
    }
    spl_sync();
    if (tid == 0) {
        const uint32_t sent = min(ss->n_sent, cap);
        const uint32_t hard = (ss->hard != 0u || n_hits > SPL_HITS || ss->n_sent > cap) ? 1u : 0u;
        if (blocks > 1u) {
            put_4u32(peer_smem(&ss->head[rank], 0), sent, hard, __float_as_uint(least), 0u, bar);
            arrive_expect(bar, sent * 8u + 16u);
        } else {
            ss->head[0] = make_uint4(sent, hard, __float_as_uint(least), 0u);
        }
    }
    LILY_STAMP(PH_LOCAL_SELECT);
    if (rank != 0u) {
        return;
    }

    // ---- 4. ranks and the draw
    const bool counts_draw = use_pen && table_mode;
    auto draw = [&](uint32_t n) {  // (n candidates sorted in key[] / id[]; the warp that draws)
        split_finalize(sm, a, row, n, in.top_p, in.min_p, u_row, a.uniforms ? 0u : in.step, in.seed, counts_draw, slot,
                       ahead);
    };
    if (blocks == 1u) {
        spl_sync();  // (head[0] and the candidates are this block's own)
    }
    uint32_t second = 0;
    if (!wide) {
        // Hardly more candidates than the row keeps: one warp does the rest.
        if (warp != 0u) {
            if (!wait_verdict(0u)) {
                return;
            }
        } else {
            const bool late = blocks > 1u && !wait_first_phase(&ss->mbar_cand);
            LILY_STAMP(PH_MERGE);
            const uint4 head = lane < blocks ? ss->head[lane] : make_uint4(0, 0, 0, 0);
            const uint32_t n = __reduce_add_sync(FULL, head.x);
            if (__any_sync(FULL, head.y != 0u || late) || n == 0u) {
                verdict(0u, ALONE);
                return;
            }
            if (n <= SPL_SMALL_K) {
                // Candidates `lane` and `lane + 32`: the first ends of the regions add up to places.
                uint32_t end = head.x;
#pragma unroll
                for (int o = 1; o < (int)SPL_MAX_BLOCKS; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, end, o);
                    end += lane >= (uint32_t)o ? t : 0u;
                }
                uint32_t r0 = 0, r1 = 0, b0 = 0, b1 = 0;
                for (uint32_t r = 0; r + 1u < blocks; ++r) {
                    const uint32_t e = __shfl_sync(FULL, end, (int)r);
                    r0 = lane >= e ? r + 1u : r0;
                    b0 = lane >= e ? e : b0;
                    r1 = lane + 32u >= e ? r + 1u : r1;
                    b1 = lane + 32u >= e ? e : b1;
                }
                const uint2 c0 = lane < n ? cand[r0 * cap + (lane - b0)] : make_uint2(0u, 0u);
                const uint2 c1 = lane + 32u < n ? cand[r1 * cap + (lane + 32u - b1)] : make_uint2(0u, 0u);
                if (__any_sync(FULL, c0.x == SPL_NAN_KEY || c1.x == SPL_NAN_KEY)) {
                    verdict(0u, ALONE);
                    return;
                }
                const unsigned long long m0 = lane < n ? ((unsigned long long)c0.x << 32) | (uint32_t)~c0.y : 0ull;
                const unsigned long long m1 = lane + 32u < n ? ((unsigned long long)c1.x << 32) | (uint32_t)~c1.y : 0ull;
                unsigned long long *packed = reinterpret_cast<unsigned long long *>(sm->tkey);
                packed[lane] = m0;
                packed[lane + 32u] = m1;
                __syncwarp();
                uint32_t p0 = 0, p1 = 0;
                const ulonglong2 *pairs = reinterpret_cast<const ulonglong2 *>(packed);
#pragma unroll 4
                for (uint32_t j = 0; j < (n + 1u) / 2u; ++j) {
                    const ulonglong2 o = pairs[j];
                    p0 += (o.x > m0 ? 1u : 0u) + (o.y > m0 ? 1u : 0u);
                    p1 += (o.x > m1 ? 1u : 0u) + (o.y > m1 ? 1u : 0u);
                }
                if (lane < n) {
                    sm->key[p0] = c0.x;
                    sm->id[p0] = c0.y;
                }
                if (lane + 32u < n) {
                    sm->key[p1] = c1.x;
                    sm->id[p1] = c1.y;
                }
                __syncwarp();
                LILY_STAMP(PH_SORT);
                draw(min(n, k));
                LILY_STAMP(PH_END);
                verdict(0u, DONE);
                return;
            }
            verdict(0u, HANDS);
        }
        second = 1u;
    }
    if (blocks > 1u && !wait_first_phase(&ss->mbar_cand)) {
        ss->hard = 2;
    }
    LILY_STAMP(PH_MERGE);
    const uint4 head = lane < blocks ? ss->head[lane] : make_uint4(0, 0, 0, 0);
    // Every block's bound holds for the row: what does not reach the largest is out.
    const uint32_t least_key = __reduce_max_sync(FULL, lane < blocks ? key_of(__uint_as_float(head.z)) : 0u);
    const uint32_t kmin = key_of(__fdiv_rn(float_of_key(least_key), in.temp));
    unsigned long long *packed = reinterpret_cast<unsigned long long *>(sm->tkey);  // (key, ~id), over tkey and tid
    if (__any_sync(FULL, head.y != 0u)) {
        ss->hard = 2;
    } else {
        // A region to each of as many teams of warps: NaNs, and in narrow rows the live ones.
        const uint32_t team = SPL_NT >> log_blocks, first = tid & (team - 1u);
        const uint32_t region = tid / team, n_region = __shfl_sync(FULL, head.x, (int)region);
        const uint2 *mine = cand + region * cap;
        bool nan = false;
        for (uint32_t i = first; i - lane < n_region; i += team) {  // (a team is whole warps)
            const uint2 e = i < n_region ? mine[i] : make_uint2(0u, 0u);
            nan = nan || e.x == SPL_NAN_KEY;
            const bool live = e.x >= kmin && i < n_region;
            const unsigned who = __ballot_sync(FULL, live);
            if (who != 0u && !wide) {
                uint32_t at = 0;
                if (lane == 0) {
                    at = atomicAdd(&ss->n_live, (uint32_t)__popc(who));
                }
                at = __shfl_sync(FULL, at, 0) + __popc(who & ((1u << lane) - 1u));
                if (live && at < KCAP) {
                    packed[at] = ((unsigned long long)e.x << 32) | (uint32_t)~e.y;
                }
            }
        }
        if (nan) {
            ss->hard = 2;
        }
    }
    spl_sync();
    const uint32_t n_live = ss->n_live;
    if (ss->hard != 0u || (!wide && (n_live == 0u || n_live > KCAP))) {
        verdict(second, ALONE);
        return;
    }
    uint32_t n;
    if (!wide) {
        for (uint32_t c = tid; c < n_live; c += SPL_NT) {
            const unsigned long long mine = packed[c];
            uint32_t before = 0;
#pragma unroll 8
            for (uint32_t j = 0; j < n_live; ++j) {
                before += packed[j] > mine ? 1u : 0u;
            }
            if (before < k) {
                sm->key[before] = (uint32_t)(mine >> 32);
                sm->id[before] = ~(uint32_t)mine;
            }
        }
        spl_sync();
        n = min(n_live, k);
    } else {
        n = split_sort_bins(sm, ss, reinterpret_cast<unsigned long long *>(ss + 1), log_blocks, k, kmin);
        if (n == 0u) {
            verdict(second, ALONE);
            return;
        }
    }
    verdict(second, DONE);
    LILY_STAMP(PH_SORT);
    if (n <= SPL_SMALL_K) {
        if (draws) {
            draw(n);
        }
    } else {
        split_finalize_wide(sm, ss, a, row, n, in.top_p, in.min_p, a.uniforms ? __ldg(a.uniforms + row) : in.u, counts_draw,
                            slot);
    }
    LILY_STAMP(PH_END);
}

}  // namespace lily
