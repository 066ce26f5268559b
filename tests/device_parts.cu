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
#endif
