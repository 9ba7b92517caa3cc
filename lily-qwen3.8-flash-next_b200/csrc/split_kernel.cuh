// The row kernel: a row's vocabulary is split over the blocks of a cluster (one,
// two, four or eight of them, as many as leave every SM something to do), which
// meet once (an argmax), twice, or (a row that keeps many) at the pool, at the exchange of their
// lists and at the first block's candidates and every block's receipt.
//
//   1. 256 threads of a block look at its vectors of the row (16 bytes each) and keep the
//      largest logit they saw; ten vectors (a bucket) share one maximum in shared
//      memory. The block's other 256 threads meanwhile mark the row's history, one
//      byte, bit or half word (a count) per vocabulary id of the block's share, and work off the
//      bias and ban lists (or, for a vocabulary shard, add up the exponentials);
//   2. with penalties that only lower a logit, the adjusted value of any k logits bounds
//      the row's k-th largest from below: every warp gives its best few adjusted maxima
//      to a pool that all blocks of the cluster hold, and the k-th largest of the pool
//      (less what a warp may have kept back) is the row's bound;
//   3. the buckets that reach the bound are read again (L2; a share of one bucket is
//      still in registers), and what reaches it is adjusted, divided by the temperature
//      and stored, as (key, id), in the shared memory of the cluster's first block;
//   4. there one warp ranks the candidates ((key descending, id ascending), as the
//      reference's CPU sampler orders them), runs the softmax weights, the prefix sums
//      in rank order, the cut and the draw (or writes a shard's record).
//
// What bounds it is latency, not memory: a call of a few rows is a chain of some ten
// dependent steps: from the share read to the bound known, with the pool's meeting in between, 1.05 to
// 1.45 us, from the candidates sent to all of them there 0.1 to 0.25. So blocks meet by stores
// that complete a barrier in the receiver, no warp waits for one that it does not need, and the
// draw's adds run in two chains of 32 lanes. Measured back to back: 1 row x 151936 f32 with a history of 4096 ids 50 -> 7.7 us, 64 rows x
// 151936 bf16 with histories 32 -> 12.8, argmax of 1 x 32768 9.2 -> 2.55 to 2.7 (before: cut in
// slices through global memory, or a cluster that kept the row in shared memory). Code that the
// warps run once is slow code: of the 18 and 15.5 clocks between two instructions of a warp (the first two of
// these) 5.7 and 3.2 wait for the instruction itself and 5.4 and 4.2 at barriers. So what stands on the way counts: functions
// that take the launch's arguments by address load each of them from memory (1 us), an
// arrival that releases waits for the thread's stores (0.3 us each), and code that a call never
// runs still slows it where it stands between what it does run: the kernel is compiled for what a
// launch's rows bring (split_args.cuh).
//
// A row that keeps more than 64 candidates takes its bound from the maxima of all
// threads of the cluster, and all blocks rank its candidates. Where penalties can raise a
// logit, an emitted id may be among the best whatever its logit: once the bound is known
// the block's other half looks at these ids, and what may reach it is a candidate of its
// own, as the ids on the bias list are. Rows this kernel does not take (a NaN, more ties
// than the buffers hold, ...) are drawn by the first block alone with the general row
// code: the results do not depend on the way.
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
__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void arrive_expect(uint32_t bar, uint32_t bytes) {
    // (Relaxed: what it counts on comes by stores that order themselves with the barrier, and the
    // receiver writes nothing into this block that it was not free to write before. A release
    // waits for every store of the thread before it.)
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// The same where the receiver goes on to write over memory that this block has read: its reads
// (in order with this arrival by a barrier of the block) come before those writes.
__device__ __forceinline__ void arrive_expect_release(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

// Waits for the first phase of a barrier in this block, for at most `limit_ns` since `t0`; true
// if it is complete. (The other blocks of the cluster are running and only have to get
// there: the limit is met only where something is wrong. The clock is looked at after
// 16 polls; t0 = 0: since then.)
// The row's last meeting has the launch's limit, the one before it half of that, the pool of a wide
// row a quarter: a block whose wait for the keys ran out still comes to the later meetings, in time to
// say so there. (It does not send on what it has not got: of a wide row that lost its lists the
// others wait for candidates and receipt in vain.)
__device__ __forceinline__ bool wait_first_phase(const unsigned long long *bar, uint64_t limit_ns, uint64_t &t0) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(bar);
    for (uint32_t i = 0;; ++i) {
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
        if ((i & 15u) == 15u) {
            const uint64_t now = (uint64_t)global_ns();
            if (t0 == 0u) {
                t0 = now;
            } else if (now - t0 > limit_ns) {
                return false;
            }
        }
    }
}

__device__ __forceinline__ bool wait_first_phase(const unsigned long long *bar, uint64_t limit_ns) {
    uint64_t t0 = 0;
    return wait_first_phase(bar, limit_ns, t0);
}

// All threads of the cluster that have not returned yet meet here, for a thread that has
// met the others at most once before (`met`: at the start). A block whose wait ran out goes
// through it before it returns or uses its shared memory for anything else: the others'
// waits are bounded too, so each of them comes here or returns, and until then it may
// store into this block.
__device__ __forceinline__ void meet_cluster(bool met) {
    if (!met) {
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}

// Every thread of the block's working half learns whether one of them says so.
__device__ __forceinline__ bool spl_any(bool mine) {
    uint32_t any;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}"
        : "=r"(any)
        : "r"(mine ? 1u : 0u), "n"(SPL_NT)
        : "memory");
    return any != 0u;
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


// The sum of p[0, 4 * tid), added up in rank order with one rounding per add
// (tests/unit/kernels/sample.rs:37-46), for each of the SPL_NT threads; the sum of all n of them goes to
// ss->least. p: KCAP weights, those past n are 0. Here by one thread, a chain of n dependent adds.
__device__ __forceinline__ float chain_of_sums(SplitSmem *ss, const float *p, uint32_t n) {
    const uint32_t tid = threadIdx.x;
    float *ends = reinterpret_cast<float *>(ss->tmax);  // sums up to every fourth rank (the maxima have served)
    static_assert(KCAP / 4u == SPL_NT, "four ranks a thread");
    if (tid == 0) {
        // All that stands beside the adds is a load of four weights and the
        // store of every fourth sum. (Ranks past n weigh 0, and s + 0 is s. With every sum stored,
        // and the weights loaded ahead moved from register to register, an add took 8 clocks
        // instead of 4.5: 1024 kept, 8100 -> 4560 clocks.)
        const float4 *p4 = reinterpret_cast<const float4 *>(p);
        float4 *e4 = reinterpret_cast<float4 *>(ends);
        constexpr uint32_t A = 8;
        float s = 0.0f;
        float4 v[2][A];
#pragma unroll
        for (uint32_t h = 0; h < A; ++h) {
            v[0][h] = p4[h];
        }
        for (uint32_t i = 0; i < n; i += 8u * A) {
#pragma unroll
            for (uint32_t side = 0; side < 2u; ++side) {
                const uint32_t at = i / 4u + side * A, next = min(at + A, KCAP / 4u - A);
#pragma unroll
                for (uint32_t h = 0; h < A; ++h) {
                    v[side ^ 1u][h] = p4[next + h];
                }
                float o[4];
#pragma unroll
                for (uint32_t h = 0; h < A; ++h) {
                    const float4 x = v[side][h];
                    s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, x.x), x.y), x.z), x.w);
                    o[h & 3u] = s;
                    if ((h & 3u) == 3u) {
                        e4[(at + h) >> 2] = make_float4(o[0], o[1], o[2], o[3]);
                    }
                }
            }
        }
        ss->least = s;  // (what it held has served)
    }
    spl_sync();
    return tid != 0u ? ends[tid - 1u] : 0.0f;
}

// The same sums without the chain. While the sum stays between two powers of two it is a multiple
// of its last place u, and adding x adds x rounded to a multiple of u, whatever the sum is (but
// for a tie, which goes by the sum's last bit). So every thread finds from approximate sums, with a
// margin above what n roundings can do, which power of two its four adds lie at; where that is one and no
// add ties, it rounds its weights by itself, and these add up exactly, in any order, as integers in
// units of 2^-23. Some eleven threads are left, those in which the sum passes a power of two: one thread
// makes their adds one after the other, with what lies between two of them as one more, exact,
// add. 1024 kept: 4560 clocks of a chain become some 1700. Up to CHAIN_MAX the chain is the shorter
// (3 x 151936 f32, by the chain and so: 320 kept 12.60 and 12.66 us, 384 12.86 and 12.76, 512 13.58 and
// 13.16, 1024 16.94 and 15.49).
constexpr uint32_t CHAIN_MAX = 384;
__device__ __forceinline__ float sums_in_rank_order(SmemFixed *sm, SplitSmem *ss, const float *p, uint32_t n) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr uint32_t LIST = 32;       // threads whose adds are made one after the other, at most
    constexpr float UNIT = 8388608.0f;  // 2^23
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    static_assert(KCAP / 4u == SPL_NT && SPL_WARPS == 8u, "four ranks a thread");
    // (Over the maxima, which have served.)
    float *totals = reinterpret_cast<float *>(ss->tmax), *after = totals + 8;
    uint32_t *whole = ss->tmax + 64, *count = whole + 8, *list_at = whole + 16;
    float4 *list_x = reinterpret_cast<float4 *>(ss->tmax + 128);
    const float4 x = reinterpret_cast<const float4 *>(p)[tid];
    float incl = __fadd_rn(__fadd_rn(x.x, x.y), __fadd_rn(x.z, x.w));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(FULL, incl, o);
        incl = lane >= (uint32_t)o ? __fadd_rn(incl, t) : incl;
    }
    if (lane == 31u) {
        totals[warp] = incl;
    }
    const float up = __shfl_up_sync(FULL, incl, 1);
    spl_sync();
    float before = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < SPL_WARPS; ++w) {
        before = w < warp ? __fadd_rn(before, totals[w]) : before;
    }
    // (1024 adds are off by less than 2^-14 of the sum, these sums by less than 2^-19.)
    constexpr float MARGIN = 1.220703125e-4f;  // 2^-13
    const uint32_t lo = __float_as_uint(__fmul_rn(lane != 0u ? __fadd_rn(before, up) : before, 1.0f - MARGIN));
    const uint32_t hi = __float_as_uint(__fmul_rn(__fadd_rn(before, incl), 1.0f + MARGIN));
    const float power = __uint_as_float(lo & 0x7F800000u);
    auto rounded = [&](float v) -> float { return __fsub_rn(__fadd_rn(v, power), power); };  // (v at most `power`)
    const float rx = rounded(x.x), ry = rounded(x.y), rz = rounded(x.z), rw = rounded(x.w);
    const float tie = __fmul_rn(power, 5.9604644775390625e-8f);  // half of the last place
    const bool ties = fabsf(__fsub_rn(x.x, rx)) == tie || fabsf(__fsub_rn(x.y, ry)) == tie ||
                      fabsf(__fsub_rn(x.z, rz)) == tie || fabsf(__fsub_rn(x.w, rw)) == tie;
    // (A thread past the last rank adds nothing. Below 512 a run between two powers fits 32 bits.)
    const bool dead = 4u * tid >= n;
    const bool one_by_one = !dead && (((lo ^ hi) >> 23) != 0u || ties || power < 1.0f || power > 512.0f ||
                                      fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)) > power);
    uint32_t units = 0;
    if (!dead && !one_by_one) {
        units = __float2uint_rn(__fmul_rn(__fadd_rn(__fadd_rn(rx, ry), __fadd_rn(rz, rw)), UNIT));
    }
    uint32_t sum = units;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, sum, o);
        sum += lane >= (uint32_t)o ? t : 0u;
    }
    const unsigned who = __ballot_sync(FULL, one_by_one);
    if (lane == 31u) {
        whole[warp] = sum;
        count[warp] = __popc(who);
    }
    spl_sync();
    uint32_t at = sum - units, j = __popc(who & ((1u << lane) - 1u)), n_list = 0;
#pragma unroll
    for (uint32_t w = 0; w < SPL_WARPS; ++w) {
        at += w < warp ? whole[w] : 0u;
        j += w < warp ? count[w] : 0u;
        n_list += count[w];
    }
    if (n_list > LIST) {  // (a tail of hardly anything beside a power of two)
        spl_sync();
        return chain_of_sums(ss, p, n);
    }
    if (one_by_one) {
        list_at[j] = at;
        list_x[j] = x;
    }
    if (tid == SPL_NT - 1u) {
        list_at[n_list] = at + units;
    }
    spl_sync();
    auto exact = [&](uint32_t u) -> float { return __fmul_rn(__uint2float_rn(u), 1.0f / UNIT); };
    if (tid == 0) {
        float s = 0.0f;
        float4 v = list_x[0];  // (rank 0 is always one of them)
        uint32_t here = list_at[0];
        for (uint32_t i = 0; i < n_list; ++i) {
            const float4 next_v = list_x[min(i + 1u, LIST - 1u)];
            const uint32_t next = list_at[i + 1u];
            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
            after[i] = s;
            s = __fadd_rn(s, exact(next - here));
            v = next_v;
            here = next;
        }
        ss->least = s;  // (what it held has served)
    }
    spl_sync();
    return j != 0u ? __fadd_rn(after[j - 1u], exact(at - list_at[j - 1u])) : 0.0f;
}

// The draw of a row that keeps more than 64 candidates, sorted in `best`: the
// softmax weights, the prefix sums in rank order with one rounding per add
// (tests/unit/kernels/sample.rs:37-46), the cut, the draw. All SPL_NT threads.
__device__ __forceinline__ void split_finalize_wide(SmemFixed *sm, SplitSmem *ss, const unsigned long long *best,
                                                    const KArgs &a, uint32_t row, uint32_t n, float top_p, float min_p,
                                                    float u, bool counts_draw, uint32_t slot) {
    const uint32_t tid = threadIdx.x;
    float *p = reinterpret_cast<float *>(sm->tkey), *cum = reinterpret_cast<float *>(sm->tid);
    const float top = float_of_key((uint32_t)(best[0] >> 32));
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
        p[i] = i < n ? exp_f32(__fsub_rn(float_of_key((uint32_t)(best[i] >> 32)), top)) : 0.0f;
    }
    if (tid == 0) {
        ss->n_live = n;   // the first rank that is not kept
        ss->bin = n;      // the first rank whose prefix sum exceeds the target
    }
    spl_sync();
    const float before_mine = n > CHAIN_MAX ? sums_in_rank_order(sm, ss, p, n) : chain_of_sums(ss, p, n);
    // Every thread its four ranks' sums, the same adds once more, and the cut.
    const float limit = __fmul_rn(top_p, ss->least);
    if (4u * tid < n) {
        float before = before_mine;
        const float4 x = reinterpret_cast<const float4 *>(p)[tid];
        const float w[4] = {x.x, x.y, x.z, x.w};
        float c[4];
        uint32_t stop = n;
#pragma unroll
        for (uint32_t e = 0; e < 4u; ++e) {
            const uint32_t i = 4u * tid + e;
            if (stop == n && i != 0u && i < n && !(before < limit && w[e] >= min_p)) {
                stop = i;
            }
            c[e] = before = __fadd_rn(before, w[e]);
        }
        reinterpret_cast<float4 *>(cum)[tid] = make_float4(c[0], c[1], c[2], c[3]);
        if (stop < n) {
            atomicMin(&ss->n_live, stop);
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
            a.kept_ids[(uint64_t)row * a.kept_ld + i] = ~(uint32_t)best[i];
            a.kept_probs[(uint64_t)row * a.kept_ld + i] = __fdiv_rn(p[i], mass);
        }
    }
    spl_sync();
    if (tid == 0) {
        const uint32_t id = ~(uint32_t)best[min(ss->bin, n_keep - 1u)];
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

// A block's candidates of a wide row: over the pool, which has served, or over key and id.
constexpr uint32_t WIDE_OWN = SPL_MAX_BLOCKS * SPL_NT / 2u;
__device__ __forceinline__ unsigned long long *wide_own(SmemFixed *sm, SplitSmem *ss, uint32_t blocks) {
    static_assert(2u * SPL_SORTED <= CAP, "one block's candidates, and their runs in order");
    return reinterpret_cast<unsigned long long *>(blocks > 1u ? ss->tmax : sm->key);
}

// Every block sorts its list and sends it to all blocks; then each knows its
// entries' ranks in the row (their places in the eight lists, by bisection) and
// sends them to the first block, to where they belong. (Merged by the first block
// alone, 1300 entries took 6 to 9 us: gathers from one SM's shared memory.)
// All SPL_NT threads. The number of candidates, merged behind *ss in the first block; 0: there
// is no such list (the first block draws the row alone), and in the other blocks.
static __device__ __noinline__ uint32_t merge_lists(SmemFixed *sm, SplitSmem *ss, uint32_t log_blocks, uint32_t sent,
                                                   uint32_t hard, uint64_t wait_ns) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, rank = blockIdx.x, blocks = 1u << log_blocks;
    const uint32_t cap = CAP >> log_blocks, cand_bar = blocks > 1u ? peer_smem(&ss->mbar[MEET_CANDIDATES], 0) : 0u;
    unsigned long long *own = wide_own(sm, ss, blocks);
    unsigned long long *lists = reinterpret_cast<unsigned long long *>(sm->key);  // over key and id: CAP
    unsigned long long *best_of = reinterpret_cast<unsigned long long *>(ss + 1);  // SPL_SORTED (the marks have served)
    // Every warp puts its runs of 32 in order; then an entry's place is the number of larger ones in
    // each run, by bisection, eight runs at a time. (Counted over the whole list, 150 entries a
    // block took 6900 clocks, so 2200.)
    const uint32_t runs = (sent + 31u) / 32u;
    // (Over the vectors that reach the bound, which have served.)
    static_assert(WIDE_OWN * 8u <= 2u * LCAP * 4u, "");
    unsigned long long *run_of = blocks > 1u ? reinterpret_cast<unsigned long long *>(sm->lkey) : own + SPL_SORTED;
    // Behind the lists' meeting the others store into the first block's best_of, where its threads have
    // read their marks: the arrival releases those reads, which lie before the caller's last barrier.
    // It counts on a list that is still to be sent, from here and by a warp that mostly has no run to
    // put in order. (3 x 151936 f32, 1024 kept: 16.8 us without a release, 16.9 so, 17.25 with it where the
    // list is sent.)
    auto bytes_for = [&](uint32_t to) -> uint32_t { return to != rank ? (sent * 8u + 15u) & ~15u : 0u; };
    if (blocks > 1u && tid - (SPL_NT - 32u) < blocks) {
        arrive_expect_release(peer_smem(&ss->mbar[MEET_LISTS], lane), bytes_for(lane) + 16u);
    }
    for (uint32_t c = tid >> 5; c < runs; c += SPL_WARPS) {
        unsigned long long x = c * 32u + lane < sent ? own[c * 32u + lane] : 0ull;
#pragma unroll
        for (uint32_t size = 2u; size <= 32u; size <<= 1) {
#pragma unroll
            for (uint32_t stride = size >> 1; stride > 0u; stride >>= 1) {
                const unsigned long long other = __shfl_xor_sync(FULL, x, stride);
                const bool larger = ((lane & size) == 0u) == ((lane & stride) == 0u);
                x = (other > x) == larger ? other : x;
            }
        }
        run_of[c * 32u + lane] = x;
    }
    spl_sync();
    for (uint32_t i = tid; i < sent; i += SPL_NT) {
        const unsigned long long mine = run_of[i];
        uint32_t place = 0;
        for (uint32_t c0 = 0; c0 < runs; c0 += SPL_WARPS) {
            uint32_t low[SPL_WARPS];
#pragma unroll
            for (uint32_t c = 0; c < SPL_WARPS; ++c) {
                low[c] = 0;
            }
#pragma unroll
            for (uint32_t step = 32u; step != 0u; step >>= 1) {
#pragma unroll
                for (uint32_t c = 0; c < SPL_WARPS; ++c) {
                    const uint32_t to = low[c] + step;
                    const unsigned long long at = run_of[min(c0 + c, runs - 1u) * 32u + min(to, 32u) - 1u];
                    low[c] = to <= 32u && at > mine ? to : low[c];
                }
            }
#pragma unroll
            for (uint32_t c = 0; c < SPL_WARPS; ++c) {
                place += c0 + c < runs ? low[c] : 0u;
            }
        }
        (blocks > 1u ? lists + rank * cap : best_of)[place] = mine;
    }
    uint32_t total = sent;
    bool lost = hard != 0u, gave_up = false;
    if (blocks > 1u) {
        // (One copy per block: stores of a thread each cost the SM some 4 clocks a piece.)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        spl_sync();
        if (tid < blocks) {
            const uint32_t list_bar = peer_smem(&ss->mbar[MEET_LISTS], tid);
            const uint32_t bytes = bytes_for(tid);
            put_4u32(peer_smem(&ss->head[rank], tid), sent, hard, 0u, 0u, list_bar);
            if (bytes != 0u) {
                asm volatile(
                    "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        peer_smem(lists + rank * cap, tid)),
                    "r"((uint32_t)__cvta_generic_to_shared(lists + rank * cap)), "r"(bytes), "r"(list_bar)
                    : "memory");
            }
        }
        gave_up = spl_any(!wait_first_phase(&ss->mbar[MEET_LISTS], wait_ns >> 1));
        if (gave_up) {
            ss->late = 1;
        }
        // A copy completes in its receiver, but its source is the sender's shared memory: no
        // block leaves or draws alone in that memory before every receiver has said so.
        if (tid < blocks && !gave_up) {
            arrive(peer_smem(&ss->mbar[MEET_GONE], tid));
        }
        const uint4 head = lane < blocks ? ss->head[lane] : make_uint4(0, 0, 0, 0);
        total = __reduce_add_sync(FULL, head.x);
        lost = __any_sync(FULL, gave_up || head.y != 0u);
    }
    if (lost || total == 0u || total > SPL_SORTED) {  // (every block decides alike)
        // (Whoever gave up meets all of the cluster before it leaves; its own receipt will not come.)
        if (blocks > 1u && !gave_up && !wait_first_phase(&ss->mbar[MEET_GONE], wait_ns)) {
            ss->late = 1;
        }
        return 0u;
    }
    if (blocks > 1u) {
        uint32_t n_of[SPL_MAX_BLOCKS], longest = 1;  // (its own list counts for nothing)
#pragma unroll
        for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
            n_of[r] = r < blocks && r != rank ? ss->head[r].x : 0u;
            longest = max(longest, n_of[r]);
        }
        for (uint32_t i = tid; i < sent; i += SPL_NT) {
            const unsigned long long x = lists[rank * cap + i];
            uint32_t low[SPL_MAX_BLOCKS], place = i;
#pragma unroll
            for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
                low[r] = 0;
            }
            // (Steps of falling powers of two: low counts the entries known to be larger.
            // Eight independent chains of loads, no branches: that is what makes it fast.)
            for (uint32_t step = 1u << (31 - __clz(longest)); step != 0u; step >>= 1) {
#pragma unroll
                for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
                    const uint32_t to = low[r] + step;
                    const unsigned long long at = lists[(r * cap + min(to, cap) - 1u) & (CAP - 1u)];
                    low[r] = (uint32_t)(to <= n_of[r]) & (uint32_t)(at > x) ? to : low[r];
                }
            }
#pragma unroll
            for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
                place += low[r];
            }
            put_2u32(peer_smem(best_of + place, 0), (uint32_t)x, (uint32_t)(x >> 32), cand_bar);
        }
        if (tid == 0) {
            arrive_expect(cand_bar, sent * 8u);
        }
        if (rank != 0u) {
            if (!wait_first_phase(&ss->mbar[MEET_GONE], wait_ns)) {
                ss->late = 1;
            }
            return 0u;
        }
        uint64_t t0 = 0;  // (the two share the limit)
        if (!wait_first_phase(&ss->mbar[MEET_CANDIDATES], wait_ns, t0) || !wait_first_phase(&ss->mbar[MEET_GONE], wait_ns, t0)) {
            ss->hard = 2;
            ss->late = 1;
        }
    }
    spl_sync();
    return ss->hard != 0u ? 0u : total;
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
    // (Eight loads at a time: one in front of its four adds cost each add 20 clocks instead of 5.)
    auto half = [&](uint32_t first, float &c) {
        float4 v[8];
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i) {
            v[i] = w4[first / 4u + i];
        }
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i) {
            const uint32_t at = first + 4u * i, mine = lane + first;
            if (at < n) {
                c = mine >= at ? __fadd_rn(c, v[i].x) : c;
                c = mine >= at + 1u ? __fadd_rn(c, v[i].y) : c;
                c = mine >= at + 2u ? __fadd_rn(c, v[i].z) : c;
                c = mine >= at + 3u ? __fadd_rn(c, v[i].w) : c;
            }
        }
    };
    c0 = 0.0f;
    half(0u, c0);
    c1 = __shfl_sync(0xFFFFFFFFu, c0, 31);
    if (n > 32u) {
        half(32u, c1);
    }
}

// The draw from at most 64 candidates, sorted in key[] / id[], by one warp: the
// softmax weights, the prefix sums in rank order (tests/unit/kernels/sample.rs:37-46),
// the cut, the draw (speculative: tests/unit/kernels/sample.rs:264-283, src/kernels/
// metal/sample.metal:597-658), the outputs. lane i holds ranks i and i + 32.
template <bool SPEC>
__device__ __forceinline__ void split_finalize(SmemFixed *sm, const KArgs &a, uint32_t row, uint32_t n, float top_p, float min_p,
                                               float u, uint32_t step, uint64_t seed, bool counts_draw, uint32_t slot,
                                               const SpecAhead &ahead) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    float *w = reinterpret_cast<float *>(sm->tkey);
    const bool in0 = lane < n, in1 = lane + 32u < n;
    const uint32_t i0 = in0 ? sm->id[lane] : 0xFFFFFFFFu, i1 = in1 ? sm->id[lane + 32u] : 0xFFFFFFFFu;
    const float top = float_of_key(sm->key[0]);
    const bool spec = SPEC && row < a.spec.n_spec;
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

// The logit, as it was before the division by the temperature, with the penalties for an
// id that was emitted `count` times.
__device__ __forceinline__ float penalise(float x, uint32_t count, float rep, float presence, float frequency) {
    if (count != 0u) {
        x = x > 0.0f ? __fdiv_rn(x, rep) : __fmul_rn(x, rep);
        x = __fsub_rn(x, __fadd_rn(presence, __fmul_rn(frequency, (float)count)));
    }
    return x;
}

// Penalties that can raise a logit: the block's emitted ids whose adjusted logits may reach
// ss->least (a NaN does) join the ids of the bias list in tkey[] / tid[]; those on the bias
// or ban list themselves are left out. The marking half of the block, while the other half
// reads again what reaches the bound. A look costs no division: the logit is adjusted
// exactly where all candidates are. Measured, presence penalty -0.3, 4096 ids: 4 rows x
// 151936 bf16 17.5 us (the row left to one block: 95; in slices: 34), 148 x 50257 f32 21 (82).
// A step of eight ids a thread costs 1.6 us (32000 ids, 4 rows: 41 us), latency all. No loop over an id's bits: lanes that went round one a
// different number of times took 0.5 us a round (148 rows x 50257: 50 of 98 us).
struct Emitted {
    const uint32_t *hist;  // the row's list ...
    uint32_t hist_len, extra_len, slot;
    float rep, presence, frequency;
    bool table, need_counts, has_lists;  // table: ... or histogram slot `slot`
};

__device__ __forceinline__ void take_emitted(SmemFixed *sm, SplitSmem *ss, const Emitted &in, float inv, float least,
                                             uint32_t id, float l, uint32_t count) {
    const float y = l > 0.0f ? l * inv : l * in.rep, pen = in.presence + in.frequency * (float)count;
    // (Away from the adjusted logit by a few roundings of 2^-24 of these three at most.)
    if (!(y - pen < least - (1e-6f * (fabsf(y) + fabsf(pen) + fabsf(least)) + 1e-37f))) {
        const uint32_t to = atomicAdd(&ss->n_listed, 1u);
        if (to < KCAP) {
            sm->tkey[to] = __float_as_uint(l);
            sm->tid[to] = id;
        } else {
            ss->hard = 1;
        }
    }
}

template <typename T>
static __device__ __noinline__ void emitted_candidates(SmemFixed *sm, SplitSmem *ss, const KArgs &a, const T *row_ptr,
                                                      uint32_t log_blocks, uint32_t *marks, uint32_t mark_mode,
                                                      const Emitted &in) {
    constexpr uint32_t PER = Piece<T>::PER, SHIFT = Piece<T>::SHIFT, NONE = 0xFFFFFFFFu;
    const uint32_t t = threadIdx.x - SPL_NT, rank = blockIdx.x, blocks = 1u << log_blocks, vocab = a.vocab;
    const uint32_t skip = (uint32_t)(reinterpret_cast<uintptr_t>(row_ptr) & 15u) / (uint32_t)sizeof(T);
    const float inv = __fdiv_rn(1.0f, in.rep), least = ss->least;
    const bool bytes = mark_mode == MARK_BYTES;
    if (!in.table) {
        // The list once more: the first of an id's entries to get there claims its mark.
        constexpr uint32_t U = 8u;  // ids of a thread on their way
        const uint32_t total = in.hist_len + in.extra_len, listed_or_claimed = bytes ? BYTE_LISTED | BYTE_CLAIMED
                                                                                     : HALF_LISTED | HALF_CLAIMED;
        for (uint32_t i0 = 0; i0 < total; i0 += U * SPL_NT) {
            uint32_t id[U], was[U], shift[U];
            T l[U];  // (nothing is done with what is asked for before all of it has been)
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t i = i0 + u * SPL_NT + t;
                id[u] = i < in.hist_len ? __ldg(in.hist + i) : i < total ? __ldcg(a.extra_ids + (i - in.hist_len)) : NONE;
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t place = id[u] + skip, piece = place >> SHIFT;
                const uint32_t at = ((piece >> log_blocks) << SHIFT) | (place & (Piece<T>::LOGITS - 1u));
                shift[u] = bytes ? (at & 3u) * 8u : (at & 1u) * 16u;
                was[u] = 0u;
                l[u] = T(0.0f);
                if (id[u] < vocab && (piece & (blocks - 1u)) == rank) {
                    l[u] = row_ptr[id[u]];
                    was[u] = atomicOr(marks + (at >> (bytes ? 2u : 1u)), (bytes ? BYTE_CLAIMED : HALF_CLAIMED) << shift[u]);
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t mark = was[u] >> shift[u], count = mark & (bytes ? BYTE_MAX : MARK_MAX);
                if (count != 0u && (mark & listed_or_claimed) == 0u) {
                    take_emitted(sm, ss, in, inv, least, id[u], widen(l[u]), count);
                }
            }
        }
        return;
    }
    // The slot's bits over the block's pieces: a warp per piece, a lane per vector.
    constexpr uint32_t U = 2u;
    const uint32_t lane = t & 31u, pieces = split_pieces(vocab, skip, PER);
    const uint32_t *seen = a.seen_table + (uint64_t)in.slot * a.seen_words;
    const uint32_t *counts = a.counts_table + (uint64_t)in.slot * vocab;
    for (uint32_t j0 = t >> 5; (j0 << log_blocks) < pieces; j0 += U * SPL_WARPS) {
        uint32_t bits[U];
        float l[U][PER];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t j = j0 + u * SPL_WARPS, first_id = (((j << log_blocks) | rank) * 32u + lane) * PER - skip;
            bits[u] = 0u;
#pragma unroll
            for (uint32_t e = 0; e < PER; ++e) {
                const uint32_t id = first_id + e;
                bits[u] |= id < vocab && ((__ldcg(seen + (id >> 5)) >> (id & 31u)) & 1u) ? 1u << e : 0u;
            }
#pragma unroll
            for (uint32_t e = 0; e < PER; ++e) {
                l[u][e] = (bits[u] >> e) & 1u ? widen(row_ptr[first_id + e]) : 0.0f;
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t j = j0 + u * SPL_WARPS, first_id = (((j << log_blocks) | rank) * 32u + lane) * PER - skip;
#pragma unroll
            for (uint32_t e = 0; e < PER; ++e) {
                // (first_id may lie in front of the row, mod 2^32: ids are added up in 32 bits, then used.)
                const uint32_t at = (j << SHIFT) | (lane * PER + e), id = first_id + e;
                if ((bits[u] >> e) & 1u) {
                    const bool listed = in.has_lists && (bytes ? reinterpret_cast<const uint8_t *>(marks)[at] & BYTE_LISTED
                                                               : reinterpret_cast<const uint16_t *>(marks)[at] & HALF_LISTED);
                    if (!listed) {
                        take_emitted(sm, ss, in, inv, least, id, l[u][e], in.need_counts ? __ldcg(counts + id) : 1u);
                    }
                }
            }
        }
    }
}

// The first block draws the row alone with the general row code, all NT threads; or, where a wait
// for the row ran out, the row has no result, and the status word says so. (A function of its
// own: it stands at a dozen places of the kernel, none of them on its way. It finds the row by
// itself, so that those places pass on one address, and the general code is part of it: behind another
// call such a row took 2 us longer. 100 x 9001 bf16, 512 kept, 43.8 -> 41.6 us; 60 x 30000
// f32, 1024 kept, 53.8 -> 51.6.)
template <typename T, uint32_t MAXR>
static __device__ __noinline__ void draw_alone_row(const SplitArgs<MAXR> &ca) {
    extern __shared__ uint4 smem_raw[];
    SplitSmem *ss = reinterpret_cast<SplitSmem *>(reinterpret_cast<SmemFixed *>(smem_raw) + 1);
    const KArgs &a = ca.a;
    const uint32_t tid = threadIdx.x, row = a.row0 + blockIdx.y;
    const T *row_ptr = reinterpret_cast<const T *>(a.logits) + (uint64_t)row * a.logits_ld;
    const bool aligned = (reinterpret_cast<uintptr_t>(row_ptr) & 15u) == 0u;
    if (ss->late != 0u) {
        if (tid == 0) {
            if (a.cand_out) {
                a.cand_out[row].max_adj = neg_inf();
                a.cand_out[row].sum_exp = 0.0f;
            } else {
                a.out_ids[row] = 0xFFFFFFFFu;
                if (a.out_status) {
                    a.out_status[row] = ROW_INTERNAL;
                }
                if (a.kept_n) {
                    a.kept_n[row] = 0;
                }
            }
            atomicOr(a.status_word, 1u << STATUS_TIMEOUT_BIT);
        }
        if (a.cand_out && tid < LILY_SHARD_CANDIDATES) {
            a.cand_out[row].cand[tid] = make_uint2(0u, 0xFFFFFFFFu);
        }
        meet_cluster(tid < SPL_NT || a.shard_sums != 0u);
        return;
    }
    RowGiven given;
    if (ca.inline_params) {
        const RowIn &in = ca.in[row];
        given.params.temperature = (in.flags & ROW_GREEDY) ? 0.0f : in.temp;
        given.params.top_k = in.k;
        given.params.top_p = in.top_p;
        given.params.min_p = in.min_p;
        given.params.presence_penalty = in.presence;
        given.params.frequency_penalty = in.frequency;
        given.params.repetition_penalty = in.rep;
        given.params.reserved = 0;
        given.params.seed = in.seed;
        given.step = in.step;
        given.has_slot = ca.inline_slots != 0u;
        given.slot = ca.inline_slots ? ca.slots[row] : 0u;
        given.has_history = ca.inline_history != 0u;
        given.history_len = ca.inline_history ? ca.inline_history - 1u : 0u;
    }
    const RowGiven *in_args = ca.inline_params ? &given : nullptr;
    __syncthreads();
    if (aligned) {
        sample_row<T, true>(a, row, 0u, 1u, in_args);
    } else {
        sample_row<T, false>(a, row, 0u, 1u, in_args);
    }
    if (a.cand_out) {
        __syncthreads();
        if (tid == SPL_NT) {
            ss->record_key = key_of(__ldcg(&a.cand_out[row].max_adj));
            ss->late = 0;  // (the general code's memory, meanwhile)
        }
        __syncthreads();
    }
}

// What the first block's waiting threads are told: the row is done, it is drawn alone, or more hands
// are needed.
enum { DONE = 0, ALONE = 1, HANDS = 2 };

// The end of an argmax row for the first block's threads that look at its logits and then only wait. (A
// function: as part of the kernel's body it stood on the way of the warp they wait for. 1 x 32768
// f32 3.5 - 3.8 -> 3.25 us.)
template <typename T, uint32_t MAXR>
static __device__ __noinline__ void wait_for_the_end(const SplitArgs<MAXR> &ca) {
    extern __shared__ uint4 smem_raw[];
    const SplitSmem *ss = reinterpret_cast<const SplitSmem *>(reinterpret_cast<SmemFixed *>(smem_raw) + 1);
    asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
    if (ss->verdict[0] == ALONE) {
        draw_alone_row<T, MAXR>(ca);
    }
}

// Grid (blocks per row, rows), clusters of (blocks per row), NT threads, of which
// SPL_NT do the work. BPS: blocks per SM the registers are cut for; with one, a
// block whose share fits one bucket keeps it in registers. HAS: what the launch's rows may bring (split_args.cuh);
// what they do not is not in the code.
template <typename T, uint32_t MAXR, int BPS, uint32_t HAS>
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
    const bool many = variant_many(HAS, MAXR) || blocks > 1u;
    const uint32_t row = a.row0 + blockIdx.y;
    const uint32_t vocab = a.vocab;
    LILY_STAMP(PH_ENTRY);

    // What needs no input comes first (see sample_row on the launch attribute).
    if (tid == 32u) {  // (two warps share the stores: they stand before the block's first barrier)
        ss->n_flagged = 0;
        ss->n_hits = 0;
        ss->n_listed = 0;
        ss->n_sent = 0;
        ss->n_live = 0;
        ss->hard = 0;
        ss->bound_key = 0;
        ss->late = 0;
    }
    if (many && tid < MEETS) {
        const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&ss->mbar[tid]);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar),
                     "r"((tid == MEET_POOL || tid == MEET_SUMS ? 1u : blocks) + (ca.lost == (rank << 8 | (tid + 1u)) ? 1u : 0u))
                     : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (uint32_t w = tid; w < ca.mark_words / 4u; w += NT) {
        reinterpret_cast<uint4 *>(marks)[w] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    if (many) {
        // (Waited for before the first store into another block.)
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const T *row_ptr = reinterpret_cast<const T *>(a.logits) + (uint64_t)row * a.logits_ld;
    const uint32_t skip = (uint32_t)(reinterpret_cast<uintptr_t>(row_ptr) & 15u) / (uint32_t)sizeof(T);
    auto draw_alone = [&]() { draw_alone_row<T, MAXR>(ca); };
    // What the first block's waiting warps are told, at barrier 2: the row is done, it
    // is drawn alone, or (only to the warps that work) more hands are needed; in the
    // last case there is a second verdict. Threads that wait return only if they are
    // needed.
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
    // A shard's record of n candidates in key[] / id[], by one warp.
    auto write_record = [&](uint32_t n) {
        ShardRecord *rec = a.cand_out + row;
#pragma unroll
        for (uint32_t i = lane; i < LILY_SHARD_CANDIDATES; i += 32u) {
            rec->cand[i] = i < n ? make_uint2(sm->key[i], sm->id[i] + a.id_offset) : make_uint2(0u, 0xFFFFFFFFu);
        }
        if (lane == 0) {
            rec->max_adj = float_of_key(sm->key[0]);
            if (!a.shard_sums) {
                rec->sum_exp = 0.0f;
            }
            ss->record_key = sm->key[0];
        }
    };
    // The upper half of the block marks the row's history while the lower half reads
    // its logits; then it waits (in the first block) for the verdict.
    const bool marker = tid >= SPL_NT;
    auto marker_ends = [&]() {
        if (rank == 0u && wait_verdict(0u)) {
            wait_verdict(1u);
        }
    };
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
        if (t >= pieces) {  // (most of a short share's: not worth a call)
            constexpr uint32_t NO = sizeof(T) == 4 ? 0xFF800000u : 0xFF80FF80u;  // -inf
            return make_uint4(NO, NO, NO, NO);
        }
        return edge_vec<T>(row_ptr, vocab, skip, t * 32u + lane);
    };
    // The row's first history ids go first. (Their number is not known yet; the row
    // has room for history_ld of them.)
    constexpr uint32_t HU = SPL_U < 8u ? SPL_U : 8u;  // (16-byte words of ids in flight a thread: they lie in q)
    static_assert(HU <= SPL_U, "the history's words in flight");
    const uint32_t *hist = a.history_ids + (uint64_t)row * a.history_ld;
    const uint32_t lead = (4u - ((uint32_t)(reinterpret_cast<uintptr_t>(hist) >> 2) & 3u)) & 3u;  // ids before the first 16-byte boundary
    const uint4 *h4 = reinterpret_cast<const uint4 *>(hist + lead);
    const uint32_t room = a.history_ids ? (uint32_t)min(a.history_ld, (uint64_t)a.max_history) : 0u;
    const uint32_t room4 = room > lead ? (room - lead) >> 2 : 0u;
    uint4 q[SPL_U];
    if (marker) {
        const uint4 no_ids = make_uint4(NONE, NONE, NONE, NONE);
#pragma unroll
        for (uint32_t i = 0; i < HU; ++i) {
            const uint32_t at = tid - SPL_NT + i * SPL_NT;
            q[i] = at < room4 ? __ldg(h4 + at) : no_ids;
        }
    } else {
#pragma unroll
        for (uint32_t i = 0; i < SPL_U; ++i) {
            q[i] = load_piece(warp + SPL_WARPS * i);
        }
    }

    // ---- the row's parameters
    RowIn in;
    uint32_t hist_len = 0, slot = 0;
    int32_t forced = -1;
    if (HAS == HAS_ARGMAX || a.force_greedy) {
        in.temp = 1.0f;
        in.rep = in.top_p = 1.0f;
        in.presence = in.frequency = in.min_p = in.u = 0.0f;
        in.k = 1;
        in.flags = ROW_GREEDY;
        in.step = 0;
        in.seed = 0;
    } else if (variant_inline(HAS) || ca.inline_params) {
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
    if (HAS != HAS_ARGMAX && a.history_ids) {
        hist_len = ca.inline_history ? ca.inline_history - 1u : a.history_len ? __ldg(a.history_len + row) : 0u;
    }
    constexpr bool LISTS = (HAS & HAS_LISTS) != 0u;
    const uint32_t n_bias = (LISTS && a.bias_ids && a.bias_len) ? __ldg(a.bias_len + row) : 0u;
    const uint32_t n_ban = (LISTS && a.ban_ids && a.ban_len) ? __ldg(a.ban_len + row) : 0u;
    if (HAS != HAS_ARGMAX && a.forced_ids) {
        forced = __ldg(a.forced_ids + row);
    }
    const bool table_mode = HAS != HAS_ARGMAX && (ca.inline_slots != 0u || a.count_slots != nullptr);
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
    const bool use_pen = HAS != HAS_ARGMAX && (in.flags & ROW_PEN) != 0u, need_counts = (in.flags & ROW_COUNTS) != 0u;
    const bool list_mode = use_pen && !table_mode;
    if (!list_mode) {
        hist_len = 0;
    }
    const uint32_t extra_len = list_mode ? a.extra_len : 0u;
    // A vocabulary shard's launch ends in the row's record, not in a draw: the best shard_k
    // logits (a greedy row's best one) and, if asked for, the sum of exponentials.
    const bool shard = (HAS & HAS_SHARD) != 0u && a.cand_out != nullptr;
    const uint32_t k = shard && !(in.flags & ROW_GREEDY) ? a.shard_k : in.k;
    const bool wide = (HAS & HAS_WIDE) != 0u && k > SPL_SMALL_K;
    const uint32_t mark_mode = ca.mark_mode;
    const bool marked = hist_len + extra_len != 0u;
    const bool counted = marked && need_counts;  // (a list whose multiplicities matter)
    const bool raises = (HAS & HAS_RAISES) != 0u && (in.flags & ROW_RAISES) != 0u;
    const bool emitted = raises && (table_mode || marked);
    // A row that keeps many takes its bound from at most SPL_MAX_BLOCKS * SPL_NT maxima: one of
    // every thread, or, of a short row over four or eight blocks, those of `groups` parts of a
    // thread's logits. (One maximum a thread, 3 x 8192 bf16, 1024 kept: not enough of them, the
    // general code's 42 us. With fewer blocks their ranking takes longer than that code: 55.)
    const uint32_t most_pieces = (pieces + blocks - 1u) >> log_blocks;
    uint32_t log_live = SPL_LOG_NT, groups = 1u;
    bool wide_fits = true;
    if (wide) {
        // (Of the threads that take part: half of them where the other half has nothing, or, of
        // eight blocks, one warp of it a piece: without its logits the bound is somewhat lower.)
        log_live = most_pieces <= (log_blocks == 3u ? 5u : SPL_MIN_TILES) ? SPL_LOG_NT - 1u : SPL_LOG_NT;
        if (BPS == 1 && log_blocks >= 2u && most_pieces <= SPL_WARPS * SPL_U) {
            groups = SPL_MAX_BLOCKS * SPL_NT >> (log_live + log_blocks);
        }
        wide_fits = min(vocab / PER, blocks << log_live) * min(groups, PER) * 8u >= 9u * k &&
                    (groups == 1u || most_pieces * 32u <= SPL_HITS || k * 5u <= blocks * SPL_HITS * 3u);
    }
    // Decided alike by every block of the cluster: rows that end here.
    const bool general = n_sp > SP_SMEM || (raises && marked && mark_mode == MARK_BITS) ||
                         (n_sp != 0u && mark_mode == MARK_BITS) ||
                         (list_mode && need_counts && mark_mode != MARK_COUNTS) ||
                         (wide && (((HAS & HAS_SPEC) != 0u && row < a.spec.n_spec) || !wide_fits));
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
        if (marker) {
            marker_ends();
        } else if (rank == 0u) {
            verdict(0u, status == LILY_ROW_OK ? ALONE : DONE);
        }
        return;
    }
    const bool argmax_mode = HAS == HAS_ARGMAX || ((in.flags & ROW_GREEDY) && !use_pen && n_sp == 0u);
    const bool draws = rank == 0u && warp == 0u;  // the warp that ends up with the row
    SpecAhead ahead;
    ahead.draft = (HAS & HAS_SPEC) != 0u && draws && row < a.spec.n_spec ? __ldg(a.spec.draft_ids + row) : 0u;
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
    if (marker && shard && a.shard_sums) {
        // A shard has no history: this half reads the share a second time (it comes from L2,
        // just behind the other half) and adds up the exponentials, in the base-2 domain and
        // relative to each thread's running maximum.
        const float scale = 1.4426950408889634f / in.temp;
        float ref = -1e30f, part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        constexpr uint32_t SU = 4u;
        static_assert(SU <= SPL_U, "the vectors in flight");
        for (uint32_t j = warp - SPL_WARPS; j < pieces_here; j += SPL_WARPS * SU) {
            float m = neg_inf();
#pragma unroll
            for (uint32_t i = 0; i < SU; ++i) {
                q[i] = load_piece(j + SPL_WARPS * i);
            }
#pragma unroll
            for (uint32_t i = 0; i < SU; ++i) {
                m = fmaxf(m, vec_max<T>(q[i]));
            }
            const float y = m * scale;
            if (y > ref) {
                const float f = exp2f(ref - y);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    part[c] *= f;
                }
                ref = y;
            }
#pragma unroll
            for (uint32_t i = 0; i < SU; ++i) {
#pragma unroll
                for (uint32_t e = 0; e < PER; ++e) {
                    part[e & 3u] += exp2f(fmaf(vec_get<T>(q[i], e), scale, -ref));  // (a masked -inf adds 0)
                }
            }
        }
        float sum = (part[0] + part[1]) + (part[2] + part[3]);
        float top = ref;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            top = fmaxf(top, __shfl_xor_sync(FULL, top, o));
        }
        sum *= exp2f(ref - top);
        sum = sum == sum ? sum : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum += __shfl_xor_sync(FULL, sum, o);
        }
        uint2 *place = &ss->sums[rank * SPL_WARPS + warp - SPL_WARPS];
        if (many) {
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (lane == 0) {
                put_2u32(peer_smem(place, 0), __float_as_uint(top), __float_as_uint(sum), peer_smem(&ss->mbar[MEET_SUMS], 0));
            }
        } else if (lane == 0) {
            *place = make_uint2(__float_as_uint(top), __float_as_uint(sum));
        }
        if (rank != 0u) {
            return;
        }
        if (!many) {
            asm volatile("bar.sync 6, %0;" ::"n"(SPL_NT) : "memory");
        }
        float total = 0.0f;
        top = neg_inf();
        bool late = false;
        if (warp == SPL_WARPS) {
            // (Collected before the verdict: the general code uses this memory for its own.)
            if (many) {
                if (lane == 0) {
                    arrive_expect(peer_smem(&ss->mbar[MEET_SUMS], 0), blocks * SPL_WARPS * 8u);
                }
                late = !__all_sync(FULL, wait_first_phase(&ss->mbar[MEET_SUMS], ca.wait_ns));
                if (late) {
                    ss->late = 1;  // (before the verdict)
                }
            }
            constexpr uint32_t EACH = SPL_MAX_BLOCKS * SPL_WARPS / 32u;
            uint2 v[EACH];
#pragma unroll
            for (uint32_t c = 0; c < EACH; ++c) {
                const uint32_t at = lane + 32u * c;
                v[c] = at < blocks * SPL_WARPS ? ss->sums[at] : make_uint2(0xFF800000u, 0u);
                top = fmaxf(top, __uint_as_float(v[c].x));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                top = fmaxf(top, __shfl_xor_sync(FULL, top, o));
            }
#pragma unroll
            for (uint32_t c = 0; c < EACH; ++c) {  // (in a fixed order: a lane's two, then the lanes' tree)
                total += __uint_as_float(v[c].y) * exp2f(__uint_as_float(v[c].x) - top);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                total += __shfl_xor_sync(FULL, total, o);
            }
        }
        marker_ends();
        if (tid == SPL_NT) {  // (the record's largest logit is there: written before the verdict)
            total *= exp2f(top - float_of_key(ss->record_key) * 1.4426950408889634f);
            a.cand_out[row].sum_exp = total == total ? total : 0.0f;
            if (ss->late != 0u) {
                a.cand_out[row].sum_exp = 0.0f;
                atomicOr(a.status_word, 1u << STATUS_TIMEOUT_BIT);
            }
        }
        if (late) {
            meet_cluster(true);
        }
        return;
    }
    if (marker) {
        // Every block looks at the whole list for the ids of its share. (Sharing the list
        // out and marking in the owner's memory was measured slower from 2000 ids on:
        // a remote store costs an SM some 4 clocks, looking at an id a fraction of one.)
        const uint32_t t = tid - SPL_NT;
        const uint32_t n4 = hist_len > lead ? (hist_len - lead) >> 2 : 0u;
        const uint32_t loose = hist_len - n4 * 4u, more = loose + extra_len;  // what the 16-byte loads leave out, and
                                                                              // ids drawn earlier in this step
        bool loaded = n4 <= room4;  // q holds the list's first part
        auto each_four = [&](auto f) {  // f(four ids) over the list (NONE where there are no four)
            for (uint32_t h_at = 0; h_at < n4; h_at += HU * SPL_NT) {
                if (!loaded) {
#pragma unroll
                    for (uint32_t i = 0; i < HU; ++i) {
                        const uint32_t at = h_at + i * SPL_NT + t;
                        q[i] = at < n4 ? __ldg(h4 + at) : make_uint4(NONE, NONE, NONE, NONE);
                    }
                }
                loaded = false;
#pragma unroll
                for (uint32_t i = 0; i < HU; ++i) {
                    if (h_at + i * SPL_NT < n4) {
                        f(h_at + i * SPL_NT + t < n4 ? q[i] : make_uint4(NONE, NONE, NONE, NONE));
                    }
                }
            }
            loaded = n4 <= HU * SPL_NT;
            const uint32_t first = min(lead, loose);
            for (uint32_t i0 = 0; i0 < more; i0 += SPL_NT) {
                const uint32_t i = i0 + t;
                const uint32_t id = i < loose ? __ldg(hist + (i < first ? i : n4 * 4u + i))
                                    : i < more ? __ldcg(a.extra_ids + (i - loose)) : NONE;
                f(make_uint4(id, NONE, NONE, NONE));
            }
        };
        for (uint32_t j = t; j < n_sp; j += SPL_NT) {
            sm->sp_ids[j] = j < n_bias ? a.bias_ids[(uint64_t)row * a.bias_ld + j]
                                       : a.ban_ids[(uint64_t)row * a.ban_ld + (j - n_bias)];
            sm->sp_vals[j] = j < n_bias ? a.bias_vals[(uint64_t)row * a.bias_ld + j] : 0.0f;
        }
        if (t < 4u) {
            sm->sp_ids[min(n_sp, SP_SMEM) + t] = NONE;
        }
        // Any thread may write the same mark; where a frequency penalty counts, every id is an add
        // of its own: 1 to 2.6 us for 16000 ids of a skewed history, whose most frequent id is a
        // fifth of it. (Marks first, and the candidates' ids counted in a second pass over the list:
        // 6 us, 4 x 151936 bf16 with 15953 ids 18.4 us against 13.9 here; and the bound had to leave out
        // what was not counted yet, so that rows which had emitted most of a short vocabulary went
        // to the general code: 6 x 8448 with as many ids, 1024 kept, 76 to 136 us against 26.)
        auto mark_all = [&](auto mark) {
            each_four([&](const uint4 &x) {
                uint32_t at;
                if (place_of(x.x, at) == rank) {
                    mark(at);
                }
                if (place_of(x.y, at) == rank) {
                    mark(at);
                }
                if (place_of(x.z, at) == rank) {
                    mark(at);
                }
                if (place_of(x.w, at) == rank) {
                    mark(at);
                }
            });
        };
        if (!marked) {
        } else if (mark_mode == MARK_BYTES) {
            mark_all([&](uint32_t at) { mark8[at] = 1; });
        } else if (mark_mode == MARK_COUNTS && counted) {
            auto add = [&](uint32_t at) { atomicAdd(marks + (at >> 1), 1u << ((at & 1u) * 16u)); };
            // No count may reach into the flags or its neighbour (one id so often: the general code).
            if (hist_len + extra_len <= 0xFFFFu) {
                mark_all(add);
                if (hist_len + extra_len > MARK_MAX) {
                    constexpr uint32_t FLAGS = (HALF_LISTED | HALF_CLAIMED) * 0x10001u;
                    asm volatile("bar.sync 6, %0;" ::"n"(SPL_NT) : "memory");
                    for (uint32_t w = t; w < ca.mark_words / 4u; w += SPL_NT) {
                        const uint4 m = reinterpret_cast<const uint4 *>(marks)[w];
                        if (((m.x | m.y | m.z | m.w) & FLAGS) != 0u) {
                            ss->hard = 1;
                        }
                    }
                }
            } else {
                // (A look first, with room for all threads that looked at the same time.)
                mark_all([&](uint32_t at) {
                    if (static_cast<volatile uint16_t *>(mark16)[at] < MARK_MAX - 4u * SPL_NT) {
                        add(at);
                    } else {
                        ss->hard = 1;
                    }
                });
            }
        } else if (mark_mode == MARK_COUNTS) {
            mark_all([&](uint32_t at) { mark16[at] = 1; });
        } else {
            mark_all([&](uint32_t at) { atomicOr(marks + (at >> 5), 1u << (at & 31u)); });
        }
        if (n_sp != 0u) {
            // The ids on the bias or ban list that are this block's, each by the thread of
            // its first entry: marked, so that the stream's candidates leave them out, and
            // a candidate of its own with its bias entries added in list order (a banned
            // id is none).
            asm volatile("bar.sync 6, %0;" ::"n"(SPL_NT) : "memory");  // the lists and the marks are there
            for (uint32_t j = t; j < n_sp; j += SPL_NT) {
                const uint32_t id = sm->sp_ids[j];
                uint32_t at;
                if (place_of(id, at) != rank) {
                    continue;
                }
                float x = widen(row_ptr[id]);
                // (Four entries per load; the padding never matches an id of the vocabulary.)
                uint32_t before = 0, bans = 0, same = 0;
                const uint4 *v4 = reinterpret_cast<const uint4 *>(sm->sp_ids);
#pragma unroll 4
                for (uint32_t e = 0; e < n_sp; e += 4u) {
                    const uint4 v = v4[e >> 2];
                    const uint32_t m = (v.x == id ? 1u : 0u) | (v.y == id ? 2u : 0u) | (v.z == id ? 4u : 0u) | (v.w == id ? 8u : 0u);
                    same += __popc(m);
                    before |= e >= j ? 0u : m & ((1u << min(j - e, 4u)) - 1u);
                    bans |= e + 4u <= n_bias ? 0u : m & ~((1u << (n_bias > e ? n_bias - e : 0u)) - 1u);
                }
                const bool first = before == 0u, banned = bans != 0u;
                if (same == 1u) {
                    x = j < n_bias ? __fadd_rn(x, sm->sp_vals[j]) : x;
                } else {
                    for (uint32_t e = 0; e < n_bias; ++e) {
                        x = sm->sp_ids[e] == id ? __fadd_rn(x, sm->sp_vals[e]) : x;
                    }
                }
                if (first) {
                    if (mark_mode == MARK_BYTES) {
                        mark8[at] |= BYTE_LISTED;
                    } else {
                        mark16[at] |= HALF_LISTED;
                    }
                    if (!banned) {
                        const uint32_t to = atomicAdd(&ss->n_listed, 1u);
                        sm->tkey[to] = __float_as_uint(x);
                        sm->tid[to] = id;
                    }
                }
            }
        }
        if (marked || n_sp != 0u) {
            asm volatile("bar.arrive 3, %0;" ::"n"(NT) : "memory");
        }
        if (emitted) {
            const Emitted r = {hist, hist_len, extra_len, slot, in.rep, in.presence, in.frequency, table_mode, need_counts,
                               n_sp != 0u};
            asm volatile("bar.sync 4, %0;" ::"n"(NT) : "memory");
            emitted_candidates<T>(sm, ss, a, row_ptr, log_blocks, marks, mark_mode, r);
            asm volatile("bar.arrive 5, %0;" ::"n"(NT) : "memory");
        }
        marker_ends();
        return;
    }
    float best = neg_inf(), bm = neg_inf();
    uint32_t best_j = NONE;
    bool bad = false;
    uint4 best_v = make_uint4(0, 0, 0, 0);
    for (uint32_t b = 0;;) {
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
        if (many) {
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (lane == 0) {
                put_2u32(peer_smem(&ss->pool[2u * (rank * SPL_WARPS + warp)], 0), m, mi, peer_smem(&ss->mbar[MEET_POOL], 0));
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
        if (many) {
            if (tid == 0) {
                arrive_expect(peer_smem(&ss->mbar[MEET_POOL], 0), blocks * SPL_WARPS * 8u);
            }
            ok = warp != 0u || wait_first_phase(&ss->mbar[MEET_POOL], ca.wait_ns);
            if (!ok) {
                ss->late = 1;
            }
        } else {
            spl_sync();
        }
        if (warp != 0u) {
            wait_for_the_end<T>(ca);
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
        if (shard) {
            if (lane == 0) {
                sm->key[0] = win;
                sm->id[0] = win_id;
            }
            __syncwarp();
            write_record(1u);
        } else if (lane == 0) {
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
    if (marked || n_sp != 0u) {
        asm volatile("bar.sync 3, %0;" ::"n"(NT) : "memory");
    }
    if ((HAS & HAS_SPEC) != 0u && draws && row < a.spec.n_spec) {
        spec_ahead(a.spec, row, vocab, ahead);
    }
    LILY_STAMP(PH_PASS1);

    auto penalised = [&](float x, uint32_t count) -> float {
        return penalise(x, count, in.rep, in.presence, in.frequency);
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
                m = (x & BYTE_MAX) | ((x & BYTE_LISTED) ? LISTED : 0u);
            } else if (mark_mode == MARK_COUNTS) {
                const uint32_t x = mark16[at];
                m = (x & MARK_MAX) | ((x & HALF_LISTED) ? LISTED : 0u);
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
    // ---- 2. the bound
    auto id_at = [&](uint32_t j, uint32_t e) -> uint32_t {  // element e of this lane's vector of piece j of the block
        return ((((j << log_blocks) | rank) * 32u + lane) * PER + e) - skip;
    };
    // This thread's best logit, adjusted but for the temperature (which keeps the order).
    auto adjusted = [&](float x, uint32_t j, uint32_t e) -> uint32_t {  // (of piece j of the block)
        if (use_pen || n_sp != 0u) {
            const uint32_t m = mark_of(id_at(j, e));
            x = (m & LISTED) ? neg_inf() : penalised(x, m);  // (a listed id: left out, which can only lower the bound)
        }
        return key_of(__fadd_rn(x, 0.0f));
    };
    uint32_t key = 0u;
    if (best_j != NONE) {
        uint32_t e = 0;
        if (use_pen || n_sp != 0u) {
#pragma unroll
            for (int i = (int)PER - 1; i >= 0; --i) {
                e = vec_get<T>(best_v, (uint32_t)i) == best ? (uint32_t)i : e;
            }
        }
        key = adjusted(best, warp + SPL_WARPS * best_j, e);
    }
    if (bad) {
        ss->hard = 1;  // (read after the next barrier)
    }
    if (many) {
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
            if (many) {
                if (lane < blocks) {
                    put_u32(peer_smem(&ss->pool[to], lane), placed, peer_smem(&ss->mbar[MEET_POOL], lane));
                }
            } else if (lane == 0) {
                ss->pool[to] = placed;
            }
        }
        if (many) {
            if (tid == 0) {
                arrive_expect(peer_smem(&ss->mbar[MEET_POOL], rank), n * 4u);
            }
            if (!wait_first_phase(&ss->mbar[MEET_POOL], ca.wait_ns >> 1)) {
                ss->hard = ss->late = 1;
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
        if (many) {
            if (tid == 0) {
                arrive_expect(peer_smem(&ss->mbar[MEET_POOL], rank), (blocks * groups << log_live) * 4u);
            }
        }
        for (uint32_t g = 0; g < groups && tid >> log_live == 0u; ++g) {
            if (BPS == 1 && groups > 1u) {  // (all of the thread's vectors are in q)
                float m = neg_inf();
                uint32_t m_at = NONE;
#pragma unroll
                for (uint32_t i = 0; i < SPL_U * PER; ++i) {
                    const float x = vec_get<T>(q[i / PER], i % PER);
                    if ((i & (groups - 1u)) == g && x > m) {
                        m = x;
                        m_at = i;
                    }
                }
                key = m_at == NONE ? 0u : adjusted(m, warp + SPL_WARPS * (m_at / PER), m_at % PER);
            }
            const uint32_t to = ((rank * groups + g) << log_live) + tid;
            if (many) {
                for (uint32_t r = 0; r < blocks; ++r) {
                    put_u32(peer_smem(&ss->tmax[to], r), key, peer_smem(&ss->mbar[MEET_POOL], r));
                }
            } else {
                ss->tmax[to] = key;
            }
        }
        for (uint32_t b = tid; b < TH_BINS; b += SPL_NT) {
            sm->thist[b] = 0;
        }
        if (tid == 0) {
            ss->bin = NONE;
        }
        if (many && !wait_first_phase(&ss->mbar[MEET_POOL], ca.wait_ns >> 2)) {
            ss->hard = ss->late = 1;
            // (Others may still put their maxima where the list of buckets would lie: it is full.)
            ss->n_flagged = SPL_FLAGGED + 1u;
        }
        spl_sync();
        uint32_t keys[SPL_MAX_BLOCKS], m = 0;
#pragma unroll
        for (uint32_t r = 0; r < SPL_MAX_BLOCKS; ++r) {
            keys[r] = r * SPL_NT + tid < blocks * groups << log_live ? ss->tmax[r * SPL_NT + tid] : 0u;
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
    if (emitted) {
        if (tid == 0) {
            ss->least = hopeless ? -neg_inf() : least;
        }
        asm volatile("bar.arrive 4, %0;" ::"n"(NT) : "memory");
    }
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
        uint32_t listed = buckets;
        if (HAS == HAS_WIDE && BPS == 1 && buckets == 2u && k > HELD_MIN) {
            // (A row of two buckets that keeps many looks at most of its vectors again: the second
            // bucket's are still in registers. It pays where the read again would take a thread more than a
            // round or two. From L2 and so, by the number kept: 3 x 151936 f32, eight blocks, 100 10.74 and 10.99 us,
            // 256 11.49 and 11.54, 320 11.80 and 11.87, 384 12.18 and 12.18, 512 12.40 and 12.29, 1024 14.71 and 13.88;
            // 3 x 248320 bf16 384 12.49 and 12.35, 1024 15.33 and 14.37; 24 x 100352 bf16, four blocks, 192 12.03 and 12.01,
            // 256 12.60 and 12.46, 384 14.23 and 13.58; 50 x 40000 f32, two, 128 12.77 and 12.81, 192 13.99 and 13.59. So the
            // line lies where neither side loses more than 0.15 us, but for two blocks. Of three buckets, two read
            // again: 1 x 200064 f32, 100 11.36 and 11.52, 512 12.89 and 12.83, 1024 15.24 and 14.83: left out. In
            // the variants for lists and for parameters on the device it gains as much (4 x 151936 f32, 1024 kept
            // 15.48 and 14.36), and their other rows lose 0.1: left out.)
            listed = 1u;
            if (bm >= least) {
#pragma unroll
                for (uint32_t i = 0; i < SPL_U; ++i) {
                    if (vec_max<T>(q[i]) >= least) {
                        hit(q[i], id_at(warp + SPL_WARPS * (SPL_U + i), 0u));
                    }
                }
            }
        }
        for (uint32_t b0 = 0; b0 < listed; b0 += 32u) {
            uint32_t over = buckets == 1u && bm >= least ? 1u : 0u;
            if (buckets != 1u) {
                const float *mine = bmax + b0 * SPL_NT + tid;
                const uint32_t end = min(listed - b0, 32u);
#pragma unroll 4
                for (uint32_t b = 0; b < end; ++b) {
                    over |= mine[b * SPL_NT] >= least ? 1u << b : 0u;
                }
            }
            if (over != 0u) {  // (few threads: an add each is sooner there than a vote and an add a bucket)
                uint32_t at = atomicAdd(&ss->n_flagged, (uint32_t)__popc(over));
                for (; over != 0u && at < SPL_FLAGGED; over &= over - 1u) {
                    ss->flagged[at++] = (uint16_t)((b0 + (uint32_t)__ffs(over) - 1u) * SPL_NT + tid);
                }
            }
        }
        spl_sync();
        const uint32_t n_flagged = ss->n_flagged;
        if (n_flagged > SPL_FLAGGED) {
            ss->hard = 1;
        } else {
            // (Each of them again, from L2: a narrow row has hardly more than one vector per thread. Four and two at
            // a time: 1 x 151936 f32 with 4096 ids 7.88 and 7.77 us, 8 x 248320 f32 from slots 13.32 and 13.54, 24 x 50257
            // f32 and 64 x 151936 bf16 the same.)
            constexpr uint32_t AGAIN = (HAS & HAS_WIDE) != 0u ? 4u : 2u;
            for (uint32_t i0 = tid; i0 < n_flagged * SPL_U; i0 += AGAIN * SPL_NT) {
                uint4 x[AGAIN];
                uint32_t v[AGAIN];
#pragma unroll
                for (uint32_t h = 0; h < AGAIN; ++h) {
                    const uint32_t i = i0 + h * SPL_NT;
                    v[h] = NONE;
                    if (i < n_flagged * SPL_U) {
                        const uint32_t f = ss->flagged[i / SPL_U], owner = f % SPL_NT;
                        const uint32_t j = (owner >> 5) + SPL_WARPS * ((f / SPL_NT) * SPL_U + i % SPL_U);
                        const uint32_t t = (j << log_blocks) | rank;
                        v[h] = t * 32u + (owner & 31u);
                        x[h] = (t < whole_end && (t != 0u || skip == 0u)) ? __ldg(vec0 - lane + v[h])
                                                                           : edge_vec<T>(row_ptr, vocab, skip, v[h]);
                    }
                }
#pragma unroll
                for (uint32_t h = 0; h < AGAIN; ++h) {
                    if (v[h] != NONE && vec_max<T>(x[h]) >= least) {
                        hit(x[h], v[h] * PER - skip);
                    }
                }
            }
        }
    }
    if (emitted) {
        asm volatile("bar.sync 5, %0;" ::"n"(NT) : "memory");
    } else {
        spl_sync();
    }
    LILY_STAMP(PH_LISTS);
    // ... and their logits, a thread each: what reaches the bound is adjusted, divided
    // and sent to the first block, and so are the ids of the bias list.
    const uint32_t cap = CAP >> log_blocks;
    const uint32_t n_hits = ss->n_hits;
    uint2 *cand = reinterpret_cast<uint2 *>(sm->key);  // over key and id: CAP of them, a region per block
    const uint32_t bar = many ? peer_smem(&ss->mbar[MEET_CANDIDATES], 0) : 0u;
    const uint32_t cand_at = many ? peer_smem(cand + rank * cap, 0) : 0u;
    // (Wide rows: first here, over the pool, which has served.)
    // (A block alone: where the others' lists would be.)
    unsigned long long *own = wide_own(sm, ss, blocks);
    const uint32_t most = wide ? (many ? min(cap, WIDE_OWN) : SPL_SORTED) : cap;
    // f(id, logit, whether it comes from the bias list) for every one that may be among
    // the best: a thread per vector, mostly with one such logit.
    const uint32_t n_vecs = n_hits <= SPL_HITS && ss->hard == 0u ? n_hits : 0u;
    const uint32_t n_all = n_vecs + (ss->hard == 0u ? ss->n_listed : 0u);  // (more of these than there is room for: hard)
    auto each_logit = [&](auto f) {
        for (uint32_t i = tid; i < n_all; i += SPL_NT) {
            if (i < n_vecs) {
                const uint4 x = hits[i];
                const uint32_t first_id = ss->hit_at[i];
                uint32_t pass = 0;
#pragma unroll
                for (uint32_t e = 0; e < PER; ++e) {
                    pass |= vec_get<T>(x, e) >= least ? 1u << e : 0u;
                }
                for (; pass != 0u; pass &= pass - 1u) {
                    const uint32_t e = (uint32_t)__ffs(pass) - 1u;
                    if (first_id + e < vocab) {
                        f(first_id + e, vec_get<T>(x, e), false);
                    }
                }
            } else {
                f(sm->tid[i - n_vecs], __uint_as_float(sm->tkey[i - n_vecs]), true);
            }
        }
    };
    each_logit([&](uint32_t id, float x, bool listed) {
        if (use_pen || n_sp != 0u) {
            uint32_t m = mark_of(id);
            if ((m & LISTED) && !listed) {
                return;  // (its own entry stands for it)
            }
            m &= ~LISTED;
            if (raises && m != 0u && !listed) {
                return;  // (likewise)
            }
            x = penalised(x, m);
        }
        const float quot = __fdiv_rn(x, in.temp);
        if (x >= least || quot != quot) {
            const uint32_t to = atomicAdd(&ss->n_sent, 1u);
            if (to < most) {
                if (quot != quot) {
                    ss->hard = 1;
                }
                const uint32_t key_q = key_of(quot);
                if (wide) {
                    own[to] = ((unsigned long long)key_q << 32) | (uint32_t)~id;
                } else if (many) {
                    put_2u32(cand_at + to * 8u, key_q, id, bar);
                } else {
                    cand[to] = make_uint2(key_q, id);
                }
            }
        }
    });
    spl_sync();
    const uint32_t sent = min(ss->n_sent, most);
    const uint32_t hard = (ss->hard != 0u || n_hits > SPL_HITS || ss->n_sent > most) ? 1u : 0u;
    const bool counts_draw = use_pen && table_mode;
    if (wide) {
        LILY_STAMP(PH_LOCAL_SELECT);
        const uint32_t total = merge_lists(sm, ss, log_blocks, sent, hard, ca.wait_ns);
        if (rank != 0u) {
            if (ss->late != 0u) {
                meet_cluster(true);
            }
            return;
        }
        LILY_STAMP(PH_MERGE);
        if (total == 0u) {
            verdict(0u, ALONE);
            return;
        }
        verdict(0u, DONE);
        LILY_STAMP(PH_SORT);
        split_finalize_wide(sm, ss, reinterpret_cast<const unsigned long long *>(ss + 1), a, row, min(total, k), in.top_p, in.min_p,
                            a.uniforms ? __ldg(a.uniforms + row) : in.u, counts_draw, slot);
        LILY_STAMP(PH_END);
        return;
    }
    if (tid == 0) {
        if (many) {
            put_4u32(peer_smem(&ss->head[rank], 0), sent, hard, __float_as_uint(least), 0u, bar);
            arrive_expect(bar, sent * 8u + 16u);
        } else {
            ss->head[0] = make_uint4(sent, hard, __float_as_uint(least), 0u);
        }
    }
    LILY_STAMP(PH_LOCAL_SELECT);
    if (rank != 0u) {
        if (ss->late != 0u) {
            meet_cluster(true);
        }
        return;
    }

    // ---- 4. ranks and the draw
    if (!many) {
        spl_sync();  // (head[0] and the candidates are this block's own)
    }
    // Hardly more candidates than the row keeps: one warp does the rest.
    uint32_t n_ranked = 0;  // candidates sorted in key[] / id[]
    if (warp != 0u) {
        if (!wait_verdict(0u)) {
            return;
        }
    } else {
        const bool late = many && !wait_first_phase(&ss->mbar[MEET_CANDIDATES], ca.wait_ns);
        if (late) {
            ss->late = 1;
        }
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
            n_ranked = min(n, k);
        } else {
            verdict(0u, HANDS);
        }
    }
    const bool alone = n_ranked != 0u;  // (the warp that has ranked them)
    if (!alone) {
        if (many && !wait_first_phase(&ss->mbar[MEET_CANDIDATES], ca.wait_ns)) {
            ss->hard = 2;
            ss->late = 1;
        }
        LILY_STAMP(PH_MERGE);
        const uint4 head = lane < blocks ? ss->head[lane] : make_uint4(0, 0, 0, 0);
        // Every block's bound holds for the row: what does not reach the largest is out.
        const uint32_t least_key = __reduce_max_sync(FULL, lane < blocks ? key_of(__uint_as_float(head.z)) : 0u);
        const uint32_t kmin = key_of(__fdiv_rn(float_of_key(least_key), in.temp));
        if (__any_sync(FULL, head.y != 0u)) {
            ss->hard = 2;
        }
        unsigned long long *packed = reinterpret_cast<unsigned long long *>(sm->tkey);  // (key, ~id), over tkey and tid
        {
            // A region to each of as many teams of whole warps: the live ones.
            const uint32_t team = SPL_NT >> log_blocks, first = tid & (team - 1u);
            const uint32_t region = tid / team, n_region = __shfl_sync(FULL, head.x, (int)region);
            const uint2 *mine = cand + region * cap;
            for (uint32_t i = first; i - lane < n_region; i += team) {
                const uint2 e = i < n_region ? mine[i] : make_uint2(0u, 0u);
                const bool live = e.x >= kmin && i < n_region;
                const unsigned who = __ballot_sync(FULL, live);
                if (who != 0u) {
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
        }
        spl_sync();
        const uint32_t n_live = ss->n_live;
        if (ss->hard != 0u || n_live == 0u || n_live > KCAP) {
            verdict(1u, ALONE);
            return;
        }
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
        n_ranked = min(n_live, k);
    }
    LILY_STAMP(PH_SORT);
    // (One place for the draw, part of the kernel's body: called as a function it took the launch's
    // arguments by their address, and every one of them was a load from memory.)
    if (draws) {
        if (shard) {
            write_record(n_ranked);
        } else {
            split_finalize<(HAS & HAS_SPEC) != 0u>(sm, a, row, n_ranked, in.top_p, in.min_p, u_row, a.uniforms ? 0u : in.step,
                                                   in.seed, counts_draw, slot, ahead);
        }
    }
    LILY_STAMP(PH_END);
    verdict(alone ? 0u : 1u, DONE);  // (a shard's record is written by then)
}

}  // namespace lily
