// The selection of a token's routes from its experts' scores, shared by the router kernels.
#ifndef S14_ROUTER_CUH
#define S14_ROUTER_CUH

#include "s14_device.cuh"

namespace s14 {

// score + bias as an integer of the same order; a NaN, whose sign means nothing, below all numbers from zero up and above the negative ones.  (Said
// here because the compiler may take `bits | sign` for a float's negative absolute value, which made a NaN such a key in one kernel and
// the largest one in another.  In integers: with v != v a block of 8 tokens of 4096 x 2048 takes 115.0 us, so 113.4.)
__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t bits = __float_as_uint(v);
    const uint32_t key = bits ^ ((uint32_t)((int)bits >> 31) | 0x80000000u);
    return (bits & 0x7FFFFFFFu) > 0x7F800000u ? 0x7FFFFFFFu : key;
}
// The picks of a warp whose lane holds the keys of experts lane, lane + 32, ... (`left`: which of them are there): lane j returns
// the expert of route j.
__device__ __forceinline__ uint32_t route_picks(const uint32_t (&key)[8], uint32_t left, uint32_t top_k, uint32_t lane) {
    // a round per pick: the largest score + bias (as an ordered integer) of what is left, the lowest expert id on ties.  A loop,
    // two warp reductions a round (eight rounds of straight code with 64-bit keys through shuffles: a block of 45 tokens 147.6 us, so
    // 146.8)
    uint32_t mine = 0u;   // lane j: the expert of route j
#pragma unroll 1
    for (uint32_t j = 0; j < top_k; ++j) {
        uint32_t best = 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) best = max(best, (left >> i & 1u) ? key[i] : 0u);
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        uint32_t id = 0xffffffffu;
#pragma unroll
        for (int i = 7; i >= 0; --i)
            if ((left >> i & 1u) && key[i] == top) id = i * 32u + lane;
        id = __reduce_min_sync(0xffffffffu, id);
        if ((id & 31u) == lane) left &= ~(1u << (id >> 5));
        if (lane == j) mine = id;
    }
    return mine;
}
// The weights of the picked experts' scores, and what else follows from a route: ids, weights and, for the one-token decode path, the
// layer's job table.  Lane j holds route j's expert and score.
__device__ __forceinline__ void route_outputs(uint32_t mine, float score, uint32_t top_k, float route_scale,
                                              int32_t *ids_out, float *weights_out, JobTable *table_out,
                                              const uint8_t *const *page_table, const uint8_t *shared_page,
                                              uint32_t shared_kind, uint32_t lane, uint32_t ep_rank,
                                              uint32_t ep_world, uint32_t shared_owner) {
    int32_t ids[8];
    float picked[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        ids[j] = (int32_t)__shfl_sync(0xffffffffu, mine, j);
        picked[j] = __shfl_sync(0xffffffffu, score, j);
    }
    if (lane != 0) return;
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if ((uint32_t)j < top_k) sum = __fadd_rn(sum, picked[j]);
    // Expert parallel: this rank keeps the jobs of the experts it owns (id mod world == rank) and,
    // if it is the shared expert's owner, the shared job; every job writes the row of its route
    // slot so that the ranks' outputs add up to the full set.
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if ((uint32_t)j >= top_k) continue;
        const float w = __fmul_rn(__fdiv_rn(picked[j], sum), route_scale);
        if (ids_out) ids_out[j] = ids[j];
        if (weights_out) weights_out[j] = w;
        if (table_out && ((uint32_t)ids[j] % ep_world) == ep_rank) {
            Job jb;
            jb.page = page_table[ids[j]];
            jb.kind = S14_PAGE_MXFP4;
            jb.token = 0;
            jb.weight = w;
            jb.is_shared = 0;
            jb.out_index = (uint32_t)j;
            table_out->jobs[n] = jb;
            table_out->token_jobs[n] = (uint8_t)n;
            ++n;
        }
    }
    if (table_out) {
        if (shared_page && shared_owner == ep_rank) {
            Job jb;
            jb.page = shared_page;
            jb.kind = shared_kind;
            jb.token = 0;
            jb.weight = 1.0f;
            jb.is_shared = 1;
            jb.out_index = top_k;
            table_out->jobs[n] = jb;
            table_out->token_jobs[n] = (uint8_t)n;
            ++n;
        }
        table_out->n_jobs = n;
        table_out->n_tokens = 1;
        table_out->token_job_begin[0] = 0;
        table_out->token_job_begin[1] = n;
    }
}
__device__ __forceinline__ void router_select(const float *scores, const float *select, uint32_t n_experts, uint32_t top_k, float route_scale,
                                              int32_t *ids_out, float *weights_out, JobTable *table_out,
                                              const uint8_t *const *page_table, const uint8_t *shared_page,
                                              uint32_t shared_kind, uint32_t lane, uint32_t ep_rank,
                                              uint32_t ep_world, uint32_t shared_owner) {
    uint32_t key[8], left = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t e = i * 32 + lane;
        key[i] = 0u;
        if (e < n_experts) {
            key[i] = order_key(__ldcg(select + e));
            left |= 1u << i;
        }
    }
    const uint32_t mine = route_picks(key, left, top_k, lane);
    const float score = lane < top_k ? __ldcg(scores + mine) : 0.0f;
    route_outputs(mine, score, top_k, route_scale, ids_out, weights_out, table_out, page_table, shared_page, shared_kind, lane, ep_rank, ep_world,
                  shared_owner);
}

}  // namespace s14

#endif
