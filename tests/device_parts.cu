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
#endif
