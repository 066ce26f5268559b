// Device code of the library called by itself: tests build this file, with the library's source that it includes, on the machine
// that runs them (tests/test_gpu_parts.py).
#if defined(PART_HANDED)
#include "s14_fp8_expert.cu"
extern "C" uint32_t no_sum() { return s14::kNoSum; }
extern "C" int fp8_expert(int sms, const float *x, const uint8_t *page, float *h, float *routed, float *y, uint32_t hidden, uint32_t inter,
                          const s14::BranchPost *post) {
    return (int)s14::launch_fp8_expert(cudaStreamPerThread, sms, x, nullptr, page, h, routed, y, post, hidden, inter);
}
#elif defined(PART_BRANCH)
#include "s14_glue.cu"
extern "C" int branch_post(uint32_t hidden, float *y, const s14::BranchPost *p) {
    return (int)s14::launch_branch_post(cudaStreamPerThread, hidden, y, p->branch_out, p->residual, p->post, p->comb, p->merged);
}
#elif defined(PART_GREEDY)
#include "s14_head.cu"
extern "C" uint32_t cluster_of(uint32_t can_run) {
    return s14::cluster_that_fits([&](uint32_t n) { return n <= can_run; });
}
extern "C" int greedy(uint32_t cluster, const float *logits, uint32_t vocab, int64_t *result) {
    static bool allowed[64] = {};
    const cudaError_t e = s14::allow_wide_clusters(s14::k_greedy_argmax, allowed);
    return (int)(e != cudaSuccess ? e : s14::launch_pdl(s14::k_greedy_argmax, dim3(cluster), dim3(s14::kArgmaxThreads), 0, cudaStreamPerThread,
                                                         cluster, logits, vocab, result));
}
#elif defined(PART_QUOTIENT)
#include "s14_glue.cu"
namespace s14 {
namespace {
// Every mantissa of the divisor; dividends at random, next to ties (the product of the divisor and a number half way between two floats) and
// next to whole quotients.  wrong[0]: quotients that are not the division operator's.
__global__ void k_quotients(uint32_t rounds, unsigned long long *wrong) {
    const uint32_t mantissa = blockIdx.x * 256u + threadIdx.x;
    uint32_t state = mantissa * 2654435761u + 1u;
    auto next = [&] { return state = state * 1664525u + 1013904223u, (state >> 16 ^ state) * 2654435769u; };
    unsigned long long n = 0;
    for (uint32_t k = 0; k < rounds; ++k) {
        const int scale = (int)(next() % 100u) - 50;
        const float s = ldexpf(__uint_as_float(0x3F800000u | mantissa), scale);
        const float m = __uint_as_float(0x3F800000u | (next() & 0x7FFFFFu));
        const double tie = (double)m + ((k & 1u) ? 0x1p-24 : 0.0);
        const float near = (float)((double)s * tie);
        for (int step = -2; step <= 2; ++step) {
            const float a = __uint_as_float(__float_as_uint(near) + step);
            n += __float_as_uint(quotient(a, s)) != __float_as_uint(__fdiv_rn(a, s));
        }
        const float a = ldexpf(m, (int)(next() % 60u) - 30);
        n += __float_as_uint(quotient(a, s)) != __float_as_uint(__fdiv_rn(a, s));
    }
    if (n) atomicAdd(wrong, n);
}
}  // namespace
}  // namespace s14
extern "C" int quotients(uint32_t rounds, unsigned long long *wrong) {
    s14::k_quotients<<<(1 << 23) / 256, 256, 0, cudaStreamPerThread>>>(rounds, wrong);
    return (int)cudaGetLastError();
}
#elif defined(PART_SINKHORN)
#include "s14_glue.cu"
namespace s14 {
namespace {
__global__ void k_sinkhorn(const float *mixes, const float *scale, const float *base, uint32_t iters, float eps, float *comb) {
    const float c = sinkhorn_warp(mixes + blockIdx.x * kMixMax, scale, base, iters, eps, threadIdx.x);
    if (threadIdx.x < kHc * kHc) comb[blockIdx.x * kHc * kHc + threadIdx.x] = c;
}
}  // namespace
}  // namespace s14
extern "C" int sinkhorn(uint32_t n, const float *mixes, const float *scale, const float *base, uint32_t iters, float eps, float *comb) {
    s14::k_sinkhorn<<<n, 32, 0, cudaStreamPerThread>>>(mixes, scale, base, iters, eps, comb);
    return (int)cudaGetLastError();
}
#elif defined(PART_ROUTER)
#include "s14_router.cu"
extern "C" float near_bound(uint32_t hidden) { return s14::near_bound(hidden); }
extern "C" int near_pays(uint32_t n_tokens, uint32_t n_experts, uint32_t hidden) { return s14::near_pays(n_tokens, n_experts, hidden); }
// By the filter whatever the size.  parts: [8][n_tokens][256] sums of the approximate logits; squares: [8][256]
extern "C" int near_routes(const s14_router_desc *r, float *squares, float *parts, uint32_t *status) {
    cudaError_t err;
    s14::launch_router_near(cudaStreamPerThread, *r, parts, squares, status, &err);
    return (int)err;
}
// All scores in double whatever the size.  scores, select: [n_tokens, 256]
extern "C" int tile_routes(const s14_router_desc *r, float *scores, float *select) {
    cudaError_t err;
    s14::launch_router_tiles(cudaStreamPerThread, *r, scores, select, &err);
    return (int)err;
}
#elif defined(PART_QUICK)
#include "s14_moe_pair.cu"
namespace s14 {
namespace {
// counts[0]: pairs the fast form settles, counts[1]: of them those that differ from the exact one
__global__ void k_swiglu(const float *ups, uint32_t n_ups, const float *weights, uint32_t n_weights, unsigned long long *counts) {
    const float gate = __uint_as_float((blockIdx.x * 256u + threadIdx.x) << 16);   // every BF16 value
    unsigned long long sure = 0, wrong = 0;
    for (uint32_t i = 0; i < n_ups; ++i) {
        const float exact = swiglu_limit_f32(gate, ups[i]), pair = swiglu_pair(gate, ups[i]);
        wrong += __float_as_uint(exact) != __float_as_uint(pair) && !(exact != exact && pair != pair);
        for (uint32_t j = 0; j < n_weights; ++j) {
            float quick;
            if (!swiglu_quick(gate, ups[i], weights[j], quick)) continue;
            ++sure;
            wrong += __float_as_uint(quick) != __float_as_uint(bf16_round(__fmul_rn(exact, weights[j])));
        }
    }
    atomicAdd(counts, sure);
    atomicAdd(counts + 1, wrong);
}
__device__ uint32_t next(uint32_t &s) {
    s = s * 1664525u + 1013904223u;
    return (s >> 16 ^ s) * 2654435769u;
}
// Two tokens' six shares: random ones whose size grows by eight, some without the larger ones, many made so that the sum lies at a BF16 tie
// or next to one.
__global__ void k_sums(uint32_t rounds, unsigned long long *counts) {
    uint32_t state = blockIdx.x * 256u + threadIdx.x + 12345u;
    unsigned long long sure = 0, wrong = 0;
    for (uint32_t n = 0; n < rounds; ++n) {
        uint32_t r[16] = {};
        for (uint32_t t = 0; t < 2; ++t) {
            const uint32_t kind = next(state), top = kind & 3u ? 6u : 1u + (kind >> 2) % 6u;
            double sum = 0.0;
            for (uint32_t j = 0; j < top; ++j) {
                const float v = ((int)(next(state) >> 8) - (1 << 23)) * exp2f((float)(3 * (int)j - 40));
                r[6u * t + j] = __float_as_uint(v);
                sum += v;
            }
            if (kind & 16u) {   // the first share moves the sum to the nearest tie, or a few steps off
                const float b = __uint_as_float((__float_as_uint((float)sum) & 0xFFFF0000u) | 0x8000u);
                const int steps = (int)(next(state) % 17u) - 8;
                r[6u * t] = __float_as_uint((float)((double)b - (sum - (double)__uint_as_float(r[6u * t])) + steps * fabs((double)b) * 0x1p-24));
            }
        }
        uint32_t quick;
        if (!digit_sums_quick(r, 0, quick)) continue;
        ++sure;
        wrong += quick != digit_sums_pair(r, 0);
    }
    atomicAdd(counts, sure);
    atomicAdd(counts + 1, wrong);
}
}  // namespace
}  // namespace s14
extern "C" int swiglu(const float *ups, uint32_t n_ups, const float *weights, uint32_t n_weights, unsigned long long *counts) {
    s14::k_swiglu<<<256, 256, 0, cudaStreamPerThread>>>(ups, n_ups, weights, n_weights, counts);
    return (int)cudaGetLastError();
}
extern "C" int sums(uint32_t rounds, unsigned long long *counts) {
    s14::k_sums<<<1024, 256, 0, cudaStreamPerThread>>>(rounds, counts);
    return (int)cudaGetLastError();
}
#endif
