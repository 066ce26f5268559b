// What the two contraction kernels of the grouped block path share: s14_moe_block.cu (one CTA per item) and
// s14_moe_pair.cu (a pair of CTAs per item).
#ifndef S14_MOE_BLOCK_CUH
#define S14_MOE_BLOCK_CUH

#include "s14_umma.cuh"

namespace s14 {

constexpr uint32_t kStageA = kUnitStride;                  // a unit's codes, then its scales
static_assert(kStageA % 1024u == 0u, "operand tiles keep the 1 KB alignment of the 128-byte swizzle");
constexpr uint32_t kPairsPerToken = S14_EXPERTS_PER_TOKEN + 1;   // pair = token * 7 + position in the mix (6: shared)

// What the up kernel's epilogue leaves (the down kernel: kModeOfficial rounds its rows to BF16, the others do not)
constexpr uint32_t kModeFused = 0u;      // the digit rows of the hidden values, laid out by the epilogue itself (small blocks)
constexpr uint32_t kModeOfficial = 1u;   // the official arithmetic's BF16 hidden values, times the route weight
constexpr uint32_t kModeValues = 2u;     // the F32 hidden values; a digits launch follows (large blocks)

struct GemmArgs {
    const BlockChunk *chunks;
    const uint32_t *n_items;    // device memory: written by the grouping kernel (chunks x slices or row tiles)
    const uint8_t *dig;         // digit tiles of the B vectors [vector][K / 256][2048]
    const uint8_t *exps;        // their block exponents + 100, [vector][K / 32]
    float *out;                 // down: the pairs' expert outputs [pair][hidden]
    uint8_t *hdig, *hexp;       // up: digit tiles and exponents of the pairs' hidden values
    uint32_t by_threads;        // the token tiles come by the tile threads' own copies (large blocks), else by bulk copies
    uint32_t hidden, inter, ring, stage;   // stage: bytes of a ring stage (a unit and nt_cap token tiles)
    // Expert parallel with the exchange inside the kernel: the pairs' outputs go into every rank's buffer
    // (plain stores to peer memory), and the last CTA to finish tells every rank that this rank's rows of
    // call `ep_call` are there (flags[rank] of the call's parity in every rank's buffer).
    float *out_peer[kMaxEpWorld];
    unsigned long long *flag_peer[kMaxEpWorld];
    unsigned int *ep_counter;   // this GPU's arrival counter, zero at rest
    uint32_t ep_world, ep_rank, ep_call;
    // Up kernel, kModeOfficial / kModeValues: the pairs' hidden values [pair][inter] (official: weighted and
    // BF16-valued) and, for the official arithmetic, the routes' weights [token][top_k]
    float *hval;
    const float *weights;
    uint32_t top_k;
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
