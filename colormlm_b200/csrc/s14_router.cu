// The router for many tokens: scores of every (token, expert) and the routes picked from them, bit for bit the arithmetic of k_router
// (s14_kernels.cu), whose products and sums are double.
#include "s14_router.cuh"
#include "s14_umma.cuh"

namespace s14 {

namespace {

inline uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

}  // namespace

// ---- every score in double ----
// Scores on the FP64 matrix pipe: a CTA takes 8 * kMt tokens x 8 * kNt experts, its warps the K range in equal parts
// (their sums meet in shared memory, in warp order).  mma.m8n8k4.f64 wants one element of A (8 tokens x 4 k) and of B
// (4 k x 8 experts) per lane and step; which k an element stands for is free as long as A and B agree, so a lane
// takes eight neighbouring elements of its row (32 bytes of x, 16 of the weights) and feeds them to eight steps:
// operands go from the L2 to registers, four lanes share a cache line, nothing is staged.  Every f32 and bf16 value is
// exact in double, so is every product, and the sums are double: score and score + bias are those of k_router.
//
// Up to 64 tokens 8 x 8 tiles of sixteen warps fill the chip (x 256 experts x 4096: 8 tokens 8.3 us, 32 tokens 4.3 from the L2, in 16 x 8 tiles
// 9.6; 45 tokens x 192 experts x 2048 10); above, tiles of 16 x 16, which read a token's row once per sixteen experts, and of 16 x 8 where
// they would be fewer than two CTAs per SM.
template <uint32_t kMt, uint32_t kNt, uint32_t kWarps>
__global__ void __launch_bounds__(kWarps * 32u)
k_router_scores(const float *__restrict__ x, const uint16_t *__restrict__ wr, const float *__restrict__ bias,
                float *__restrict__ scores, float *__restrict__ select, uint32_t n_experts, uint32_t hidden,
                uint32_t n_tokens, uint32_t score_fn) {
    __shared__ double s_c[kWarps][kMt * kNt][64];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, row = lane >> 2, col = lane & 3u;
    const uint32_t e0 = blockIdx.x * (8u * kNt), t0 = blockIdx.y * (8u * kMt);
    const uint32_t part = hidden / kWarps, first = warp * part + col * 8u;   // a whole number of steps of 32 elements
    const float *xr[kMt];
    const uint16_t *wp[kNt];
    // (a token or expert past the end reads the last one again; its scores are not written)
#pragma unroll
    for (uint32_t m = 0; m < kMt; ++m) xr[m] = x + (size_t)min(t0 + m * 8u + row, n_tokens - 1u) * hidden + first;
#pragma unroll
    for (uint32_t n = 0; n < kNt; ++n) wp[n] = wr + (size_t)min(e0 + n * 8u + row, n_experts - 1u) * hidden + first;
    double c[kMt][kNt][2] = {};
    float4 xa[kMt], xb[kMt];
    uint4 q[kNt];
    auto load = [&](uint32_t k) {
#pragma unroll
        for (uint32_t n = 0; n < kNt; ++n) q[n] = __ldcg(reinterpret_cast<const uint4 *>(wp[n] + k));
#pragma unroll
        for (uint32_t m = 0; m < kMt; ++m) {
            xa[m] = __ldcg(reinterpret_cast<const float4 *>(xr[m] + k));
            xb[m] = __ldcg(reinterpret_cast<const float4 *>(xr[m] + k) + 1);
        }
    };
    dependency_wait();
    load(0);
#pragma unroll 1
    for (uint32_t k = 0; k < part; k += 32u) {
        float a[kMt][8];
        uint32_t b[kNt][4];
#pragma unroll
        for (uint32_t m = 0; m < kMt; ++m) {
            a[m][0] = xa[m].x, a[m][1] = xa[m].y, a[m][2] = xa[m].z, a[m][3] = xa[m].w;
            a[m][4] = xb[m].x, a[m][5] = xb[m].y, a[m][6] = xb[m].z, a[m][7] = xb[m].w;
        }
#pragma unroll
        for (uint32_t n = 0; n < kNt; ++n) b[n][0] = q[n].x, b[n][1] = q[n].y, b[n][2] = q[n].z, b[n][3] = q[n].w;
        if (k + 32u < part) load(k + 32u);
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            double av[kMt], bv[kNt];
#pragma unroll
            for (uint32_t m = 0; m < kMt; ++m) av[m] = (double)a[m][i];
#pragma unroll
            for (uint32_t n = 0; n < kNt; ++n)
                bv[n] = (double)__uint_as_float((i & 1u) ? b[n][i >> 1] & 0xffff0000u : b[n][i >> 1] << 16);
#pragma unroll
            for (uint32_t m = 0; m < kMt; ++m)
#pragma unroll
                for (uint32_t n = 0; n < kNt; ++n)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                                 : "+d"(c[m][n][0]), "+d"(c[m][n][1])
                                 : "d"(av[m]), "d"(bv[n]));
        }
    }
    // C (8 x 8): lane holds row lane / 4, columns 2 (lane % 4) and 2 (lane % 4) + 1
#pragma unroll
    for (uint32_t m = 0; m < kMt; ++m)
#pragma unroll
        for (uint32_t n = 0; n < kNt; ++n)
            *reinterpret_cast<double2 *>(&s_c[warp][m * kNt + n][row * 8u + col * 2u]) = make_double2(c[m][n][0], c[m][n][1]);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kMt * kNt * 64u; i += kWarps * 32u) {
        const uint32_t tile = i >> 6, at = i & 63u;
        double sum = s_c[0][tile][at];
#pragma unroll
        for (uint32_t w = 1; w < kWarps; ++w) sum += s_c[w][tile][at];
        const uint32_t t = t0 + (tile / kNt) * 8u + (at >> 3), e = e0 + (tile % kNt) * 8u + (at & 7u);
        if (t < n_tokens && e < n_experts) {
            const float sc = router_score_f32(sum, score_fn);
            scores[(size_t)t * n_experts + e] = sc;
            select[(size_t)t * n_experts + e] = __fadd_rn(sc, bias ? __ldcg(bias + e) : 0.0f);
        }
    }
}

// One warp per token picks the routes from the scores.
__global__ void __launch_bounds__(256)
k_router_select_batch(const float *__restrict__ scores, const float *__restrict__ select, uint32_t n_experts, uint32_t n_tokens,
                      uint32_t top_k, float route_scale, int32_t *__restrict__ ids_out, float *__restrict__ weights_out) {
    const uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    dependency_wait();   // (triggers behind the wait: the digits launch behind reads x without waiting for this kernel; so does k_router_pick)
    if (t >= n_tokens) return;
    router_select(scores + (size_t)t * n_experts, select + (size_t)t * n_experts, n_experts, top_k, route_scale,
                  ids_out + (size_t)t * top_k, weights_out + (size_t)t * top_k, nullptr, nullptr, nullptr, 0, threadIdx.x & 31u, 0,
                  1, 0);
}

// ---- scores in double only where they decide: large blocks of many experts ----
// Of a token's 256 scores the six largest matter, and those that come near the sixth.  So the logits are first taken
// from BF16 products (k_router_near), each with a bound on its error, and k_router_pick takes in double, for every token, the
// experts that can be among the picked ones: 6.5 on average for Gaussian rows.  Ids and weights are those of scores that are all taken in double.
// All of them on the FP64 matrix pipe in tiles of 16 tokens x 16 experts (at half of its rate) take, x 256 experts x 4096, 40 us for
// 370 tokens and 85 for 1000, and the pick 3; this 9 + 13 and 15 + 24, half of the second beside the digits launch (near_pays has the calls).
//
// k_router_near: x = hi + lo + r with BF16 values hi and lo, |r| <= 2^-18 |x|; hi and lo against the weights on tcgen05.mma
// (kind::f16, M = 128 experts, N tokens, F32 sums).  A CTA takes 128 experts, `nt` tokens and an eighth of K; the eighths' sums go to
// memory as they are ([8][token][256]) and meet in k_router_pick.  512 threads bring a stage of 64 k by copies three stages
// ahead into the 128-byte swizzle of K-major operand tiles, the weights as they are (16 KB), the tokens to be split in place; one of them
// issues the stage's eight multiplications.  It also leaves the sums of the weights' squares, for the bound.
// A wait that runs out stops the CTA: the threads agree on it at the next barrier, nothing more is loaded or issued, logits and squares
// become NaN (which sends their tokens to the scores in double, so the routes are right all the same), the status word is set, and tensor memory
// goes back when the queued multiplications are complete.
constexpr uint32_t kNearThreads = 512, kNearStages = 4, kNearSplit = 8, kNearK = 64, kNearTokens = 128, kNearW = 16384;

// kind::f16: A and B BF16 (format 1), both K-major, F32 accumulators, M = 128, N = n (a multiple of 16)
__device__ __forceinline__ constexpr uint32_t umma_idesc_bf16(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// two values rounded to BF16, the first in the lower half, and what they leave
__device__ __forceinline__ uint32_t bf16_parts(float a, float b, float &ra, float &rb) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    ra = __fsub_rn(a, __low2float(h));
    rb = __fsub_rn(b, __high2float(h));
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void copy_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

__global__ void __launch_bounds__(kNearThreads)
k_router_near(const float *__restrict__ x, const uint16_t *__restrict__ wr, float *__restrict__ part, float *__restrict__ wsq,
              uint32_t n_experts, uint32_t hidden, uint32_t n_tokens, uint32_t nt, uint32_t *status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kNearStages];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const uint32_t tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31u;
    const uint32_t e0 = blockIdx.x * 128u, t0 = blockIdx.y * nt, ks = blockIdx.z;
    const uint32_t slice = hidden / kNearSplit, steps = slice / kNearK;   // 1 .. 8 steps: hidden is a multiple of 512 up to 4096
    const uint32_t stage = kNearW + nt * 256u, bar0 = smem_u32(bars), smem0 = smem_u32(smem);   // weights, then hi and lo of the tokens
    if (tid < kNearStages) mbar_init(bar0 + tid * 8u, 1u);
    if (tid == 0) {
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kNearTokens) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        fence_before();
    }
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    // this thread's pieces of eight k: of two weight rows and of up to two tokens (an expert or token past the end is the last one again),
    // and their place in a stage
    const uint32_t row = tid >> 3, piece = tid & 7u, k0 = ks * slice + piece * 8u;
    const uint16_t *wp[2];
    const float *xp[2];
    uint32_t to[2];
    bool has[2];
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
        const uint32_t r = row + 64u * i;
        wp[i] = wr + (size_t)min(e0 + r, n_experts - 1u) * hidden + k0;
        xp[i] = x + (size_t)min(t0 + r, n_tokens - 1u) * hidden + k0;
        to[i] = r * 128u + ((piece ^ (r & 7u)) << 4);
        has[i] = r < nt;
    }
    dependency_wait();
    // step c's copies, one group (empty past the end, so that the groups can be counted).  A token's eight values come to where its two
    // parts will lie, which take as many bytes: the thread that has copied them splits them in place
    auto load = [&](uint32_t c) {
        if (c < steps) {
            const uint32_t at = smem0 + (c % kNearStages) * stage;
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                copy_async16(at + to[i], wp[i] + c * kNearK);
                if (has[i]) {
                    copy_async16(at + kNearW + to[i], xp[i] + c * kNearK);
                    copy_async16(at + kNearW + nt * 128u + to[i], xp[i] + c * kNearK + 4);
                }
            }
        }
        copy_async_commit();
    };
#pragma unroll
    for (uint32_t c = 0; c < kNearStages - 1u; ++c) load(c);
    const bool first_tile = blockIdx.y == 0u;
    float sq[2] = {0.0f, 0.0f};   // the squares of this thread's weights
    const uint32_t idesc = umma_idesc_bf16(nt);
    bool ok = true;
    uint32_t issued = 0;
#pragma unroll 1
    for (uint32_t c = 0; c < steps; ++c) {
        copy_async_wait<(int)kNearStages - 2>();   // this step's
        uint8_t *const at = smem + (c % kNearStages) * stage;
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            if (has[i]) {
                uint8_t *const hi_at = at + kNearW + to[i], *const lo_at = hi_at + nt * 128u;
                const float4 a = *reinterpret_cast<const float4 *>(hi_at), b = *reinterpret_cast<const float4 *>(lo_at);
                float r0, r1, r2, r3, r4, r5, r6, r7, none;
                uint4 hi, lo;
                hi.x = bf16_parts(a.x, a.y, r0, r1);
                hi.y = bf16_parts(a.z, a.w, r2, r3);
                hi.z = bf16_parts(b.x, b.y, r4, r5);
                hi.w = bf16_parts(b.z, b.w, r6, r7);
                lo.x = bf16_parts(r0, r1, none, none);
                lo.y = bf16_parts(r2, r3, none, none);
                lo.z = bf16_parts(r4, r5, none, none);
                lo.w = bf16_parts(r6, r7, none, none);
                *reinterpret_cast<uint4 *>(hi_at) = hi;
                *reinterpret_cast<uint4 *>(lo_at) = lo;
            }
        }
        if (first_tile) {
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const uint4 q = *reinterpret_cast<const uint4 *>(at + to[i]);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xFFFF0000u);
                    sq[i] = __fmaf_rn(lo, lo, __fmaf_rn(hi, hi, sq[i]));
                }
            }
        }
        fence_async_smem();
        ok = __syncthreads_and(ok);
        if (!ok) break;
        issued = c + 1u;
        if (warp == 0) {
            if (elect_one()) {
                const uint32_t at0 = smem0 + (c % kNearStages) * stage;
                const uint64_t a_desc = smem_desc(at0, 1, 64, 2), b_desc = smem_desc(at0 + kNearW, 1, 64, 2);
#pragma unroll
                for (uint32_t kk = 0; kk < 4; ++kk) {
                    umma_bf16(tmem, a_desc + kk * 2u, b_desc + kk * 2u, idesc, (c || kk) ? 1u : 0u);
                    umma_bf16(tmem, a_desc + kk * 2u, b_desc + nt * 8u + kk * 2u, idesc, 1u);
                }
                umma_commit(bar0 + (c % kNearStages) * 8u);
            }
            __syncwarp();
        }
        // the stage that step c + 3 takes is free when step c - 1 is complete
        if (c >= 1u && c + kNearStages - 1u < steps) ok = mbar_wait(bar0 + ((c - 1u) % kNearStages) * 8u, ((c - 1u) / kNearStages) & 1u, &abort_flag);
        if (ok) load(c + kNearStages - 1u);   // (a thread whose own wait has not run out: the stage is free)
    }
    copy_async_wait<0>();
    // all of the CTA's multiplications are complete, or none of its results count
    const uint32_t last = issued - 1u;   // (the first step is always issued)
    if (ok) ok = mbar_wait(bar0 + (last % kNearStages) * 8u, (last / kNearStages) & 1u, &abort_flag);
    ok = __syncthreads_and(ok);
    if (!ok) {
        mbar_drain(bar0 + (last % kNearStages) * 8u, (last / kNearStages) & 1u);
        if (tid == 0) atomicExch(status, 0x5509u);
    }
    fence_after();
    if (first_tile) {
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
            if (piece == 0u) wsq[ks * 256u + e0 + row + 64u * i] = ok ? sq[i] : __uint_as_float(0x7FFFFFFFu);
        }
    }
    // a lane's expert, sixteen tokens at a time
    const uint32_t quad = warp & 3u, e = e0 + quad * 32u + lane;
    for (uint32_t g = (warp >> 2) * 16u; g < nt; g += 64u) {
        uint32_t r[16];
        tmem_ld16(tmem + ((quad * 32u) << 16) + g, r);
        tmem_ld_wait();
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) {
            const uint32_t t = t0 + g + j;
            if (t < n_tokens) part[((size_t)ks * n_tokens + t) * 256u + e] = ok ? __uint_as_float(r[j]) : __uint_as_float(0x7FFFFFFFu);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kNearTokens) : "memory");
}

// A score and how much more (or less) it can be than what is returned when its logit is off by `err` at most.  The derivative s' of
// either function changes by a factor of e^err at most over `err` (|s'' / s'| <= 1); it is never above 1/3 (sigmoid 1/4).
__device__ __forceinline__ float near_score(float l, float err, uint32_t score_fn, float &off) {
    const float ex = expf(-l), sig = __fdividef(1.0f, 1.0f + ex);
    float s, slope;
    if (score_fn == S14_SCORE_SIGMOID) {
        s = sig;
        slope = sig * (1.0f - sig);
    } else {
        s = sqrtf(l > 20.0f ? l : log1pf(expf(l)));
        slope = s > 1e-18f ? __fdividef(l > 20.0f ? 0.5f : 0.5f * sig, s) : 0.0f;
    }
    off = err * (err < 1.0f ? fminf(0.5f, slope * (1.0f + 2.0f * err) + 0x1p-18f) : 0.5f);
    return s;
}

// What k_router_near's logit may be off by, of |x| |w| (see k_router_pick).
__host__ __device__ constexpr float near_bound(uint32_t hidden) { return 4.3e-6f + 3.37e-8f * (float)hidden; }

// One CTA per token: the logits' parts are added, a bound on their error is made, and the experts that can be among the top_k are
// scored in double, each warp an eighth of K; then the first warp picks.
//
// The bound.  S = |x| |w| (lengths of the rows) is no less than an expert's sum of |x_k w_k|.  What hi and lo leave of x moves a logit by
// 2^-18 S at most.  A multiplication adds sixteen exact products to a sum in F32; whatever the order and the roundings in it, with 23 bits
// kept of the largest of the seventeen terms it is off by 18 x 2^-23 of what the magnitudes so far add up to.  An eighth of K is a chain of
// n = 2 x hidden / 8 / 16 multiplications, and where the row's magnitude lies in a chain's first elements all n of them meet all of it: n x 18 x
// 2^-23 of the chain's part of S, so of S for the eight together, whose F32 sum adds 7 x 2^-24; hi and lo together are 1 + 2^-8 of x at most.
// That is near_bound: 1.42e-4 for 4096, 2.2e-5 for 512.  (Half of the chain's magnitude in place of all of it, the mean for rows whose
// magnitude is spread evenly, is no bound: with such a row the arithmetic described here is off by 1.2 times what that gives.)  Gaussian rows of
// 4096: 0.012 of a logit whose deviation is 1.3.  Squares
// that underflow are made up for by 2^-114; an S that is not finite, or a logit that is not, makes every expert a candidate.
//
// What it spends its time on, for a token alone on its SM and with two others beside it, in clocks: the parts and the token 1000 / 2000, scores and
// bound 1000, the candidates 1700, their weights and products 4000 / 5800 (loads: rows 8 KB apart; four lanes to a row and 64 bytes a load
// took 9000), scores in double 1200 / 1900, pick and weights 1700 (selection rounds by warp reductions 4000 in all).
__global__ void __launch_bounds__(256, 3)
k_router_pick(const float *__restrict__ x, const uint16_t *__restrict__ wr, const float *__restrict__ bias, const float *__restrict__ part,
              const float *__restrict__ wsq, uint32_t n_experts, uint32_t hidden, uint32_t n_tokens, uint32_t score_fn,
              uint32_t top_k, float route_scale, int32_t *__restrict__ ids_out, float *__restrict__ weights_out) {
    __shared__ float s_sq[8], s_sel[256], s_score[256];
    __shared__ double s_sum[8][8];
    __shared__ __align__(16) uint32_t s_top[32];
    __shared__ __align__(16) uint32_t s_least[256];
    __shared__ uint32_t s_n, s_most[256], s_has[8], s_bar[8];
    __shared__ uint16_t s_list[256];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, t = blockIdx.x, mine_e = min(tid, n_experts - 1u);
    const uint32_t pieces = hidden >> 6, piece0 = warp * pieces + lane;   // of eight elements, this warp's: 8 .. 64
    if (tid == 0) s_n = 0u;
    dependency_wait();
    float p[kNearSplit], q[kNearSplit];
    float4 xa[2] = {}, xb[2] = {};
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u)
        if (lane + 32u * u < pieces) {
            const float4 *const at = reinterpret_cast<const float4 *>(x + (size_t)t * hidden) + 2u * (piece0 + 32u * u);
            xa[u] = __ldcg(at);
            xb[u] = __ldcg(at + 1);
        }
#pragma unroll
    for (uint32_t k = 0; k < kNearSplit; ++k) p[k] = __ldcg(part + ((size_t)k * n_tokens + t) * 256u + mine_e);
#pragma unroll
    for (uint32_t k = 0; k < kNearSplit; ++k) q[k] = __ldcg(wsq + k * 256u + mine_e);
    const bool there = tid < n_experts;
    const float b = there && bias ? __ldcg(bias + tid) : 0.0f;
    float x2 = 0.0f;
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
        x2 = __fmaf_rn(xa[u].x, xa[u].x, __fmaf_rn(xa[u].y, xa[u].y, __fmaf_rn(xa[u].z, xa[u].z, __fmaf_rn(xa[u].w, xa[u].w, x2))));
        x2 = __fmaf_rn(xb[u].x, xb[u].x, __fmaf_rn(xb[u].y, xb[u].y, __fmaf_rn(xb[u].z, xb[u].z, __fmaf_rn(xb[u].w, xb[u].w, x2))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x2 += __shfl_xor_sync(0xffffffffu, x2, o);
    if (lane == 0) s_sq[warp] = x2;
    float logit = 0.0f, w2 = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < kNearSplit; ++k) {
        logit += p[k];
        w2 += q[k];
    }
    __syncthreads();
    x2 = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < 8; ++w) x2 += s_sq[w];
    // (1.001: the sums' own roundings)
    const float err = near_bound(hidden) * sqrtf(__fmaf_rn(x2, 1.001f, 0x1p-114f)) * sqrtf(__fmaf_rn(w2, 1.001f, 0x1p-114f));
    float off;
    const float s = near_score(logit, err, score_fn, off), sel = s + b;
    // the score's own evaluation and the roundings here (a bias beyond 3e38 - a mask's, infinite or the type's lowest - is the sum whatever the
    // score is)
    off += 0x1p-18f * (fabsf(s) + (fabsf(b) <= 3e38f ? fabsf(b) : 0.0f) + 0x1p-20f);
    const bool all = __syncthreads_or(there && !(fabsf(s) <= 3e38f && off <= 3e38f && b == b));
    // a token of zeros (padding): every logit is zero; one that holds a NaN (padding that nobody has written): every logit is none
    const uint32_t bits = __float_as_uint(xa[0].x) | __float_as_uint(xa[0].y) | __float_as_uint(xa[0].z) | __float_as_uint(xa[0].w) |
                          __float_as_uint(xb[0].x) | __float_as_uint(xb[0].y) | __float_as_uint(xb[0].z) | __float_as_uint(xb[0].w) |
                          __float_as_uint(xa[1].x) | __float_as_uint(xa[1].y) | __float_as_uint(xa[1].z) | __float_as_uint(xa[1].w) |
                          __float_as_uint(xb[1].x) | __float_as_uint(xb[1].y) | __float_as_uint(xb[1].z) | __float_as_uint(xb[1].w);
    const bool none = x2 != x2, alike = none || (x2 == 0.0f && !__syncthreads_or((bits << 1) != 0u) && !all);
    // No more than the top_k-th largest of what the experts have at least: the largest of every one, two, four or eight experts, of 32 such
    // groups at most, and of those the top_k-th (where two of the largest are in one group it is the next one's: a candidate more).  Every
    // warp finds it.
    uint32_t key = there ? order_key(sel - off) : 0u;
    const uint32_t shift = n_experts <= 32u ? 0u : (n_experts <= 64u ? 1u : (n_experts <= 128u ? 2u : 3u));
#pragma unroll 1
    for (uint32_t o = (1u << shift) >> 1; o > 0u; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
    if ((tid & ((1u << shift) - 1u)) == 0u && (tid >> shift) < 32u) s_top[tid >> shift] = key;
    __syncthreads();
    key = s_top[lane];
    uint32_t above = 0u;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint4 k4 = reinterpret_cast<const uint4 *>(s_top)[i];
        above += (k4.x > key) + (k4.y > key) + (k4.z > key) + (k4.w > key);
    }
    const uint32_t least = __reduce_min_sync(0xffffffffu, above < top_k ? key : 0xffffffffu);
    const bool cand = there && (all || order_key(sel + off) >= least);
    const uint32_t mine = __ballot_sync(0xffffffffu, cand);
    uint32_t at = 0u;
    if (lane == 0) {
        s_has[warp] = mine;
        at = atomicAdd(&s_n, (uint32_t)__popc(mine));
    }
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(mine & ((1u << lane) - 1u));
    if (cand) s_list[at] = (uint16_t)tid;
    s_least[tid] = there ? order_key(sel - off) : 0u;
    if (cand) s_most[tid] = order_key(sel + off);
    __syncthreads();
    uint32_t n = s_n;
    if (n > 32u && !all) {
        // where masks leave fewer groups than top_k with an expert that counts: by the top_k-th largest of all that the experts have at least
        const uint32_t low = s_least[tid];
        above = 0u;
#pragma unroll 8
        for (uint32_t i = 0; i < 64u; ++i) {
            const uint4 k4 = reinterpret_cast<const uint4 *>(s_least)[i];
            above += (k4.x > low) + (k4.y > low) + (k4.z > low) + (k4.w > low);
        }
        const uint32_t bar = __reduce_min_sync(0xffffffffu, above < top_k ? low : 0xffffffffu);
        if (lane == 0) s_bar[warp] = bar;
        __syncthreads();
        uint32_t bars = s_bar[0];
#pragma unroll
        for (uint32_t w = 1; w < 8u; ++w) bars = min(bars, s_bar[w]);
        const uint32_t who = __ballot_sync(0xffffffffu, cand && s_most[tid] >= bars);
        if (lane == 0) s_has[warp] = who;
        __syncthreads();
        at = __popc(who & ((1u << lane) - 1u));
        n = 0u;
#pragma unroll
        for (uint32_t w = 0; w < 8u; ++w) {
            if (w < warp) at += __popc(s_has[w]);
            n += __popc(s_has[w]);
        }
        if (who >> lane & 1u) s_list[at] = (uint16_t)tid;
        __syncthreads();
    }
    if (n > 8u && n <= 32u && !all) {
        // more than the groups below: by the top_k-th largest itself, which is among them
        uint32_t e = lane < n ? s_list[lane] : 0u, low = lane < n ? s_least[e] : 0u, before = 0u;
#pragma unroll 1
        for (uint32_t i = 0; i < n; ++i) before += __shfl_sync(0xffffffffu, low, i) > low;
        const uint32_t bar = __reduce_min_sync(0xffffffffu, lane < n && before < top_k ? low : 0xffffffffu);
        const bool stays = lane < n && s_most[e] >= bar;
        const uint32_t who = __ballot_sync(0xffffffffu, stays);
        __syncthreads();
        if (warp == 0 && stays) s_list[__popc(who & ((1u << lane) - 1u))] = (uint16_t)e;
        n = __popc(who);
        __syncthreads();
    }
    // Eight candidates at a time, each warp its part of K, the loads of a piece of all eight in flight together.  A BF16 weight's bits, moved
    // three to the right, are the double of 2^-896 times its value, subnormal ones included, so nothing has to be converted (a conversion takes
    // an SM four times as long as a multiplication); with the token times 2^800 no product leaves the range of normal doubles, and the sum has
    // the bits of the plain one times 2^-96.  Weights that are not finite come with `all`, and so does this loop's other form.
    if (alike) {
        s_score[tid] = router_score_f32(none ? __longlong_as_double(-1ll) : 0.0, score_fn);
        s_sel[tid] = __fadd_rn(s_score[tid], b);
        __syncthreads();
    }
#pragma unroll 1
    for (uint32_t c0 = alike ? n : 0u; c0 < n; c0 += 8u) {
        double acc[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) acc[k] = 0.0;
#pragma unroll 1
        for (uint32_t u = 0; u < 64u && u < pieces; u += 32u) {
            const bool in = lane + u < pieces;
            const uint16_t *const at_w = wr + (size_t)(piece0 + u) * 8u;
            uint4 wq[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
                wq[k] = in ? __ldcg(reinterpret_cast<const uint4 *>(at_w + (size_t)s_list[min(c0 + k, n - 1u)] * hidden)) : make_uint4(0u, 0u, 0u, 0u);
            const float4 fa = u ? xa[1] : xa[0], fb = u ? xb[1] : xb[0];
            const double xd[8] = {fa.x * 0x1p800, fa.y * 0x1p800, fa.z * 0x1p800, fa.w * 0x1p800,
                                  fb.x * 0x1p800, fb.y * 0x1p800, fb.z * 0x1p800, fb.w * 0x1p800};
            if (!all) {
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) {
                    const uint32_t w[4] = {wq[k].x, wq[k].y, wq[k].z, wq[k].w};
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        acc[k] = __fma_rn(xd[2u * j], __hiloint2double(((int)(w[j] << 16) >> 3) & (int)0x8FFFFFFF, 0), acc[k]);
                        acc[k] = __fma_rn(xd[2u * j + 1u], __hiloint2double(((int)w[j] >> 3) & (int)0x8FFFE000, 0), acc[k]);
                    }
                }
            } else {
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) {
                    const uint32_t w[4] = {wq[k].x, wq[k].y, wq[k].z, wq[k].w};
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        acc[k] = __fma_rn(xd[2u * j], (double)__uint_as_float(w[j] << 16) * 0x1p-896, acc[k]);
                        acc[k] = __fma_rn(xd[2u * j + 1u], (double)__uint_as_float(w[j] & 0xffff0000u) * 0x1p-896, acc[k]);
                    }
                }
            }
        }
        // the lanes' sums: a lane gives away half of what it holds, and ends with candidate lane / 4
#pragma unroll
        for (uint32_t h = 4; h > 0; h >>= 1) {
            const bool upper = lane & (4u * h);
#pragma unroll
            for (uint32_t k = 0; k < h; ++k) {
                const double give = upper ? acc[k] : acc[k + h], keep = upper ? acc[k + h] : acc[k];
                acc[k] = keep + __shfl_xor_sync(0xffffffffu, give, 4u * h);
            }
        }
        double sum = acc[0];
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if ((lane & 3u) == 0u) s_sum[warp][lane >> 2] = sum;
        __syncthreads();
        if (tid < 8u && c0 + tid < n) {
            sum = s_sum[0][tid];
#pragma unroll
            for (uint32_t w = 1; w < 8; ++w) sum += s_sum[w][tid];
            const uint32_t e = s_list[c0 + tid];
            const float sc = router_score_f32(sum * 0x1p96, score_fn);
            s_score[e] = sc;
            s_sel[e] = __fadd_rn(sc, bias ? __ldcg(bias + e) : 0.0f);
        }
        __syncthreads();
    }
    if (warp) return;
    uint32_t picked;
    if (n <= 32u) {
        // a candidate per lane: its place is the number of those before it
        const uint32_t e = lane < n ? s_list[lane] : 0u, key = lane < n ? order_key(s_sel[e]) : 0u;
        uint32_t place = 0u;
#pragma unroll 1
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t k = __shfl_sync(0xffffffffu, key, i), id = __shfl_sync(0xffffffffu, e, i);
            place += k > key || (k == key && id < e);
        }
        if (lane < n && place < top_k) s_top[place] = e;
        __syncwarp();
        picked = lane < top_k ? s_top[lane] : 0u;
    } else {
        uint32_t keys[8], left = 0u;
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            keys[i] = 0u;
            if (s_has[i] >> lane & 1u) {
                keys[i] = order_key(s_sel[i * 32u + lane]);
                left |= 1u << i;
            }
        }
        picked = route_picks(keys, left, top_k, lane);
    }
    const float score = lane < top_k ? s_score[picked] : 0.0f;
    float sum = 0.0f;
#pragma unroll 1
    for (uint32_t j = 0; j < top_k; ++j) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, score, j));
    if (lane < top_k) {
        ids_out[(size_t)t * top_k + lane] = (int32_t)picked;
        weights_out[(size_t)t * top_k + lane] = __fmul_rn(__fdiv_rn(score, sum), route_scale);
    }
}

static int launch_router_near(cudaStream_t st, const s14_router_desc &r, float *part, float *wsq, uint32_t *status, cudaError_t *err) {
    const uint32_t nt = std::min(ceil_div(ceil_div(r.n_tokens, 9u), 16u) * 16u, kNearTokens), mt = ceil_div(r.n_experts, 128u);
    const size_t smem = (size_t)kNearStages * (kNearW + nt * 256u);
    static bool allowed[64] = {};
    int dev = -1;
    *err = cudaGetDevice(&dev);
    if (*err == cudaSuccess && (dev < 0 || dev >= 64)) *err = cudaErrorInvalidDevice;
    if (*err == cudaSuccess && !allowed[dev]) {
        *err = cudaFuncSetAttribute(k_router_near, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kNearStages * (kNearW + kNearTokens * 256u)));
        allowed[dev] = *err == cudaSuccess;
    }
    // (two tiles of experts, up to nine of tokens, eight parts of K: as many CTAs as SMs)
    if (*err == cudaSuccess)
        *err = launch_pdl(k_router_near, dim3(mt, ceil_div(r.n_tokens, nt), kNearSplit), dim3(kNearThreads), smem, st, 0u, r.x, r.router_weight_bf16,
                          part, wsq, r.n_experts, r.hidden, r.n_tokens, nt, status);
    if (*err == cudaSuccess)
        *err = launch_pdl(k_router_pick, dim3(r.n_tokens), dim3(256), 0, st, 0u, r.x, r.router_weight_bf16, r.bias,
                          (const float *)part, (const float *)wsq, r.n_experts, r.hidden, r.n_tokens, r.score_fn, r.top_k,
                          r.route_scale, r.ids_out, r.weights_out);
    return *err == cudaSuccess ? 2 : 0;
}

// Which of the two ways.  All scores in double take time by tokens x experts x hidden; k_router_near by tiles of 128 experts, and k_router_pick, a CTA per
// token, hardly less for few experts than for many.  us of the call (inter 512 or 1024), all in double / by the filter: 256 experts x 4096, 80
// tokens 116.6 both, 150 156.9 / 152.1, 1000 official 366 / 319; 256 x 2048, 100 tokens 116.2 / 116.4, 370 235 / 224; 256 x 1024, 250 97.1 / 97.3, 370
// 125.5 / 122.1; 192 x 2048, 250 123.9 / 124.4, 370 161.1 / 158.8; 160 x 2048, 250 121.9 / 124.4, 700 261 / 256; but rows so short that
// the pick is most of it, 256 x 512, 1000 tokens 208.3 / 208.8, official 118.2 / 119.3.  One tile of experts: 128 x 4096, 370 tokens official 155.1 / 156.6,
// 700 235 / 221; 128 x 2048, 1000 tokens 501 / 499; 64 x 4096, 1000 tokens 370 / 378; 64 x 512, 250 tokens 46.2 / 50.6; 8 x 1024, 1000 tokens 100 / 114.
constexpr uint32_t kNearFrom = 64;   // (up to 64 tokens the 8 x 8 tiles are the faster for all sizes)
static bool near_pays(uint32_t n_tokens, uint32_t n_experts, uint32_t hidden) {
    const uint64_t row = (uint64_t)n_experts * hidden, work = row * n_tokens;
    if (n_tokens <= kNearFrom) return false;
    return n_experts > 128u ? row >= 1ull << 18 && work * n_experts >= 1ull << 34 : work >= 1ull << 28;
}

static int launch_router_tiles(cudaStream_t st, const s14_router_desc &r, float *scores, float *select, cudaError_t *err) {
    auto run = [&](auto kernel, uint32_t mt, uint32_t nt, uint32_t warps) {
        return launch_pdl(kernel, dim3(ceil_div(r.n_experts, 8u * nt), ceil_div(r.n_tokens, 8u * mt)), dim3(warps * 32u), 0, st, 0u, r.x,
                          r.router_weight_bf16, r.bias, scores, select, r.n_experts, r.hidden, r.n_tokens, r.score_fn);
    };
    if (r.n_tokens <= 64u) *err = run(k_router_scores<1, 1, 16>, 1, 1, 16);
    else if (ceil_div(r.n_tokens, 16u) * ceil_div(r.n_experts, 16u) < 296u) *err = run(k_router_scores<2, 1, 8>, 2, 1, 8);
    else *err = run(k_router_scores<2, 2, 8>, 2, 2, 8);
    if (*err != cudaSuccess) return 0;
    *err = launch_pdl(k_router_select_batch, dim3(ceil_div(r.n_tokens, 8)), dim3(256), 0, st, 0u, (const float *)scores,
                      (const float *)select, r.n_experts, r.n_tokens, r.top_k, r.route_scale, r.ids_out, r.weights_out);
    return 2;
}

int launch_router_batch(cudaStream_t st, const s14_router_desc &r, float *scores, float *select, float *parts, uint32_t *status, cudaError_t *err) {
    *err = cudaErrorInvalidValue;
    if (r.hidden % 512u || r.hidden > 4096u) return 0;   // (a block object's hidden size)
    return near_pays(r.n_tokens, r.n_experts, r.hidden) ? launch_router_near(st, r, parts, scores, status, err)
                                                        : launch_router_tiles(st, r, scores, select, err);
}

}  // namespace s14
