// The draw of a vocabulary-sharded row: the shards' records hold every candidate the
// row's top-k can contain (each shard kept its own best 64 >= k), so selecting, cutting
// and drawing over their union gives what one pass over the whole vocabulary gives.
//
// One block per row; latency bounds it. A single shard's record is in order already: one
// warp draws from it as it is. Several are ranked by counting (up to RANKSORT_MAX
// candidates, one per thread) or selected first. The parameters of up to 64 rows travel
// in the launch's own arguments, so that no copy stands between the candidates' kernel
// and this one. Measured, 64 rows of one shard behind the candidates' kernel (copies,
// launch gap and kernel): 25 -> 4 us.
#pragma once

#include "split_kernel.cuh"

namespace lily {

static __global__ void __launch_bounds__(NT, 2) merge_rows_kernel(const __grid_constant__ MergeArgs ma) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const KArgs &a = ma.a;
    extern __shared__ uint4 smem_raw[];
    SmemFixed *sm = reinterpret_cast<SmemFixed *>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const uint32_t row = a.row0 + blockIdx.x;
    if (tid == 0) {
        sm->n = 0;
        sm->err = 0;
    }
    RowIn in;
    if (a.params == nullptr) {
        in = ma.in[row];
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (a.peer.n != 0u) {
        peer_exchange_row(a, row);  // the row's records of all ranks are in the own buffer after this
    }
    if (a.params != nullptr) {
        in = row_in(a.params[row], a.steps ? a.steps[row] : 0u);
    }
    const float u = a.uniforms ? a.uniforms[row] : in.u;
    const ShardRecord *rec0 = a.merge_in + row;
    uint32_t n;
    if (a.merge_shards == 1u) {
        if (tid >= 64u) {
            return;
        }
        if (tid >= 32u) {  // (the second warp: the log-sum-exp)
            if (a.out_lse && lane == 0u) {
                a.out_lse[row] = rec0->max_adj + logf(rec0->sum_exp);
            }
            return;
        }
        const uint2 c0 = rec0->cand[lane], c1 = rec0->cand[lane + 32u];
        n = (uint32_t)__popc(__ballot_sync(FULL, c0.y != 0xFFFFFFFFu)) +
            (uint32_t)__popc(__ballot_sync(FULL, c1.y != 0xFFFFFFFFu));
        sm->key[lane] = c0.x;
        sm->id[lane] = c0.y;
        sm->key[lane + 32u] = c1.x;
        sm->id[lane + 32u] = c1.y;
        __syncwarp();
    } else {
        __syncthreads();
        const uint32_t slots = a.merge_shards * LILY_SHARD_CANDIDATES;
        for (uint32_t i = tid; i < slots; i += NT) {
            const uint2 e = rec0[(uint64_t)(i / LILY_SHARD_CANDIDATES) * a.merge_stride].cand[i % LILY_SHARD_CANDIDATES];
            if (e.y != 0xFFFFFFFFu) {
                const uint32_t at = atomicAdd(&sm->n, 1u);
                sm->key[at] = e.x;
                sm->id[at] = e.y;
            }
        }
        if (a.out_lse && tid == NT - 1u) {
            // Shards in order: the largest maximum, then the sums rescaled to it.
            float top = neg_inf();
            for (uint32_t s = 0; s < a.merge_shards; ++s) {
                top = fmaxf(top, rec0[(uint64_t)s * a.merge_stride].max_adj);
            }
            float sum = 0.0f;
            for (uint32_t s = 0; s < a.merge_shards; ++s) {
                const ShardRecord *rec = rec0 + (uint64_t)s * a.merge_stride;
                sum += rec->sum_exp * expf(rec->max_adj - top);
            }
            a.out_lse[row] = top + logf(sum);
        }
        __syncthreads();
        n = sm->n;
        const uint32_t k = in.k;
        if (tid == 0) {
            sm->n_adj = n;
        }
        __syncthreads();
        if (n <= RANKSORT_MAX) {
            rank_sort(sm, n, k);
        } else if (n > k) {
            select_topk(sm, n, k);
            if (tid < 32u) {
                sort_candidates<true>(sm, k);
            }
        }
        if (tid >= 32u) {
            return;
        }
        __syncwarp();
    }
    n = min(n, in.k);
    if (n == 0u) {
        if (lane == 0u) {
            a.out_ids[row] = 0xFFFFFFFFu;
            if (a.out_status) {
                a.out_status[row] = ROW_INTERNAL;
            }
            if (a.kept_n) {
                a.kept_n[row] = 0;
            }
            atomicOr(a.status_word, 1u << ROW_INTERNAL);
        }
        return;
    }
    if (in.flags & ROW_GREEDY) {  // (its best logit, whatever that is)
        if (lane == 0u) {
            a.out_ids[row] = sm->id[0];
            if (a.out_status) {
                a.out_status[row] = LILY_ROW_OK;
            }
            if (a.kept_n) {
                a.kept_n[row] = 1;
                a.kept_ids[(uint64_t)row * a.kept_ld] = sm->id[0];
                a.kept_probs[(uint64_t)row * a.kept_ld] = 1.0f;
            }
        }
        return;
    }
    SpecAhead ahead;
    ahead.draft = ahead.n_q = ahead.id0 = ahead.id1 = 0;
    ahead.q_draft = ahead.p0 = ahead.p1 = 0.0f;
    split_finalize<false>(sm, a, row, n, in.top_p, in.min_p, u, 0u, in.seed, false, 0u, ahead);
    if (lane == 0u && sm->err) {
        atomicOr(a.status_word, 1u << (sm->err & 31u));
    }
}

}  // namespace lily
