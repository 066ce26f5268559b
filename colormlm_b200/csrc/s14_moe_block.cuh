// What the files of the grouped block path share: s14_moe_block.cu (digits, grouping, mix, the launches) and
// s14_moe_pair.cu (the contraction kernels).
#ifndef S14_MOE_BLOCK_CUH
#define S14_MOE_BLOCK_CUH

#include "s14_umma.cuh"

namespace s14 {

constexpr uint32_t kStageA = kUnitStride;                  // a unit's codes, then its scales
static_assert(kStageA % 1024u == 0u, "operand tiles keep the 1 KB alignment of the 128-byte swizzle");
constexpr uint32_t kPairsPerToken = S14_EXPERTS_PER_TOKEN + 1;   // pair = token * 7 + position in the mix (6: shared)

struct GemmArgs {
    const BlockChunk *chunks;
    const uint32_t *n_chunks;   // device memory: written by the grouping kernel
    uint32_t *why;              // the call's counts[3]: kBlockGaveUp is added by a CTA that gives up
    const uint8_t *dig;         // digit tiles of the B vectors [vector][K / 256][2048; official arithmetic: 1024]
    const uint8_t *exps;        // their block exponents + 100, [vector][K / 32]
    float *hval;                // up: the pairs' hidden values [pair][inter] (official: BF16 values, times the route weight)
    const float *weights;       // up, official arithmetic: the routes' weights [token][top_k]
    float *out;                 // down: the pairs' expert outputs [pair][hidden]
    uint32_t hidden, inter, top_k;
    uint32_t ring, stage;       // stages, bytes of a stage (set by launch_pair_gemm)
    // Expert parallel with the exchange inside the kernel: the pairs' outputs go into every rank's buffer
    // (plain stores to peer memory), and the last CTA to finish tells every rank that this rank's rows of
    // call `ep_call` are there (flags[rank] of the call's parity in every rank's buffer), unless one of the call's CTAs gave up.
    float *out_peer[kMaxEpWorld];
    unsigned long long *flag_peer[kMaxEpWorld];
    unsigned int *ep_counter;   // this GPU's arrival counter, zero at rest
    uint32_t ep_world, ep_rank, ep_call;
};

// The pair kernels (s14_moe_pair.cu): chunks of up to 2 * `half` groups of sixteen digit rows, two row tiles (slices) per item.
size_t pair_dynamic_limit();
cudaError_t launch_pair_gemm(cudaStream_t st, int sm_count, bool down, bool official, GemmArgs args, uint32_t half, uint32_t *status);

namespace {

// torch's .to(torch.bfloat16).float()
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
// two values rounded the same way: the first in the lower half of the word
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a)) | (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(b)) << 16;
}

}  // namespace
}  // namespace s14

#endif
