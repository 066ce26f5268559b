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
    const uint8_t *dig;         // digit tiles of the B vectors [vector][K / 256][2048]; official arithmetic: 768, the tokens'
                                // in four forms [token][4][K / 256][768]
    const uint8_t *exps;        // their block exponents + 100, [vector][K / 32]
    float *hval;                // up: the pairs' hidden values [pair][inter]
    uint16_t *hval16;           // official: their gates and up projections as BF16 values [pair][2][inter]
    float *out;                 // down: the pairs' expert outputs [pair][hidden]
    uint16_t *out16;            // official: the same as BF16 values
    uint32_t hidden, inter;
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

// The limited SwiGLU (swiglu_limit_f32: the same bits) in F32 operations: the F32 blocks' up epilogue, where FP64 ones run at a quarter of
// their rate beside the MMAs, and what swiglu_quick does not settle.  The
// exponential by Ziv's method: e^t = 2^n e^r with r = t - n ln 2 in two floats (Cody and Waite's reduction, ln 2 in three
// parts of which n times the first is exact), e^r by its Taylor series to r^11 / 11!, the terms from r^6 on in F32 and the
// others in pairs of floats; the pair is within 2^-41 of e^t (4e7 arguments against an 80-bit exponential), so where the
// bounds 2^-38 to either side round to the same float, that is e^t correctly rounded.  The others, one in 10^4, and gates
// whose e^-g is beyond 2^57 take the FP64 path.  (1000 official tokens, when their epilogue had it: 1160 us with FP64, 1124 so.)
__device__ __noinline__ float swiglu_f64(float gate, float up) { return swiglu_limit_f32(gate, up); }
__device__ __forceinline__ float swiglu_pair(float gate, float up) {
    const float g = fminf(gate, 10.0f), u = fminf(fmaxf(up, -10.0f), 10.0f), t = -g;
    const float n = rintf(__fmul_rn(t, 1.44269502f));
    const float r0 = __fmaf_rn(n, -0x1.62e4p-1f, t);   // exact
    const float p = __fmul_rn(n, 0x1.7f7d1cp-20f), pe = __fmaf_rn(n, 0x1.7f7d1cp-20f, -p);
    const float a = __fsub_rn(r0, p), bb = __fsub_rn(a, r0);
    const float al = __fmaf_rn(n, -0x1.ef357ap-45f,
                               __fsub_rn(__fadd_rn(__fsub_rn(r0, __fsub_rn(a, bb)), __fsub_rn(-p, bb)), pe));
    const float rh = __fadd_rn(a, al), rl = __fsub_rn(al, __fsub_rn(rh, a));
    float h = __fmaf_rn(rh, 2.50521084e-8f, 2.75573192e-7f);
    h = __fmaf_rn(rh, h, 2.75573188e-6f);
    h = __fmaf_rn(rh, h, 2.48015876e-5f);
    h = __fmaf_rn(rh, h, 1.98412701e-4f);
    h = __fmaf_rn(rh, h, 1.38888892e-3f);
    float l = 0.0f;
    // (h, l) = c + r (h, l), c = 1 / 5! ... 1 / 0!
    auto horner = [&](float c, float c_low) {
        const float ph = __fmul_rn(rh, h), pl = __fmaf_rn(rl, h, __fmaf_rn(rh, l, __fmaf_rn(rh, h, -ph)));
        h = __fadd_rn(c, ph);
        l = __fadd_rn(__fsub_rn(ph, __fsub_rn(h, c)), __fadd_rn(pl, c_low));
    };
    horner(0x1.111112p-7f, -0x1.dddddep-32f);
    horner(0x1.555556p-5f, -0x1.555556p-30f);
    horner(0x1.555556p-3f, -0x1.555556p-28f);
    horner(0.5f, 0.0f);
    horner(1.0f, 0.0f);
    horner(1.0f, 0.0f);
    const float s = __fadd_rn(h, l), sl = __fsub_rn(l, __fsub_rn(s, h)), err = __fmul_rn(s, 0x1p-38f);
    const float e0 = __fadd_rn(s, __fadd_rn(sl, err)), e1 = __fadd_rn(s, __fsub_rn(sl, err));
    if (!(t < 40.0f) || e0 != e1) return swiglu_f64(gate, up);
    const float e = __fmul_rn(e0, __uint_as_float((uint32_t)((int)n + 127) << 23));
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, e)), u);
}

// (out of line, for rare callers: eight copies of it made a digits kernel of few vectors slower than its work)
__device__ __noinline__ float swiglu_once(float gate, float up) { return swiglu_pair(gate, up); }
// Official arithmetic: the limited SwiGLU times the route's weight as the BF16 value, where the fast exponential and quotient
// settle it.  __expf(-g) is within 2 + 1.173 |g| units of the last place (2^-23 of the value at most), __fdividef within two; with
// the five roundings of the exact expressions and the four here that is less than 1.1e-6 + 1.45e-7 |g| of the result, so where that much
// to either side rounds to the same BF16 value, that is the result.  False for the others (one in some hundred), gates below -80,
// results near the ends of F32's range, products that are so before the weight (they lose bits that a large weight brings
// back), zeros and NaNs.
__device__ __forceinline__ bool swiglu_quick(float gate, float up, float weight, float &out) {
    const float g = fminf(gate, 10.0f), u = fminf(fmaxf(up, -10.0f), 10.0f), ag = fabsf(g);
    const float p = __fmul_rn(__fdividef(g, __fadd_rn(1.0f, __expf(-g))), u), v = __fmul_rn(p, weight);
    const float d = __fmaf_rn(ag, 1.45e-7f, 1.1e-6f);
    const uint32_t both = bf16_pair(__fmaf_rn(v, -d, v), __fmaf_rn(v, d, v));
    out = __uint_as_float(both << 16);
    return ag <= 80.0f && fabsf(p) > 0x1p-110f && fabsf(v) > 0x1p-110f && fabsf(v) < 0x1p120f && (both >> 16) == (both & 0xFFFFu);
}

}  // namespace
}  // namespace s14

#endif
