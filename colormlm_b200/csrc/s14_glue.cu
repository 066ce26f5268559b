// The steps on either side of the MoE inside one layer: hyper-connection reduce (hc_pre) and expand
// (hc_post), RMSNorm, the head's reduce and the hash route of the first layers.  Reference:
//   fast16/research/polaris_meridian_v1/local_s14_primitives/hc.py:19-148
//   fast16/research/polaris_meridian_v1/local_s14_primitives/final_head.py:43-110
//   fast16/research/polaris_meridian_v1/s14_first_real_token/executor.py:638-668
// The Python code computes in F32 and leaves the order of its long sums and its exp to torch's CPU
// kernels.  Here the long sums (mean of squares, the dot products with hc_fn and with the router
// rows) are accumulated in double and rounded to F32 once, exp is evaluated in double and rounded
// once, and everything else follows the Python expressions operation by operation in F32 with
// separate multiplies and adds (no FMA), the sums over the four streams in stream order - the
// arithmetic of the CPU restatement the tests compare with.
// A token's state is hc = 4 streams of `hidden` values, F32 or BF16 (the reference's state is BF16
// [1, 1, 4, 4096]); results are rounded to the streams' type where the Python code casts back.
#include <type_traits>

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "s14_umma.cuh"

namespace s14 {

namespace cg = cooperative_groups;

namespace {

constexpr uint32_t kHc = 4;
constexpr uint32_t kMixMax = (2 + kHc) * kHc;

// What an earlier kernel wrote is read from the L2: these kernels may be resident before that kernel ends, and
// an SM's L1 may still hold the line's earlier contents.
template <bool kBf16>
__device__ __forceinline__ float stream_ld(const void *p, size_t i) {
    if constexpr (kBf16) return __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const uint16_t *>(p) + i) << 16);
    else return __ldcg(reinterpret_cast<const float *>(p) + i);
}
template <bool kBf16>
__device__ __forceinline__ void stream_st(void *p, size_t i, float v) {
    if constexpr (kBf16) reinterpret_cast<__nv_bfloat16 *>(p)[i] = __float2bfloat16_rn(v);
    else reinterpret_cast<float *>(p)[i] = v;
}

// N consecutive stream values, back and forth: eight BF16 or four F32 values are one 16-byte access, four BF16 values one of 8
// bytes, eight F32 values two of 16 (which a warp's lanes make 32 bytes apart); one by one where a caller's buffer is
// not aligned to 16 bytes (`vec`): all of hc_post and rms_norm, and hc_pre's reduced vector.  Those kernels are compiled once for
// each (with both forms in one kernel 370 tokens of 4096 took hc_post 7.6 us, now 6.2, and F32 norms 3.7, now 3.0), the norm also
// for either, which some sizes are faster with (launch_rms_norm).  The dot products of hc_pre and of the head always read four
// values of x and of hc_fn at a time; the calls refuse what is not aligned for that.
template <bool kBf16, int N>
__device__ __forceinline__ void stream_ldn(const void *p, size_t i, float (&v)[N], bool vec) {
    static_assert(N == 4 || N == 8, "values per thread");
    if (!vec) {
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = stream_ld<kBf16>(p, i + k);
        return;
    }
    if constexpr (kBf16) {
        uint32_t w[N / 2];
        const uint16_t *at = reinterpret_cast<const uint16_t *>(p) + i;
        if constexpr (N == 8) {
            const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(at));
            w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
        } else {
            const uint2 q = __ldcg(reinterpret_cast<const uint2 *>(at));
            w[0] = q.x, w[1] = q.y;
        }
#pragma unroll
        for (int k = 0; k < N / 2; ++k) v[2 * k] = __uint_as_float(w[k] << 16), v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
    } else {
        const float4 *at = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p) + i);
#pragma unroll
        for (int k = 0; k < N / 4; ++k) {
            const float4 a = __ldcg(at + k);
            v[4 * k] = a.x, v[4 * k + 1] = a.y, v[4 * k + 2] = a.z, v[4 * k + 3] = a.w;
        }
    }
}
template <bool kBf16, int N>
__device__ __forceinline__ void stream_stn(void *p, size_t i, const float (&v)[N], bool vec) {
    if (!vec) {
#pragma unroll
        for (int k = 0; k < N; ++k) stream_st<kBf16>(p, i + k, v[k]);
        return;
    }
    if constexpr (kBf16) {
        uint32_t w[N / 2];
#pragma unroll
        for (int k = 0; k < N / 2; ++k) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
            w[k] = *reinterpret_cast<const uint32_t *>(&b);
        }
        uint16_t *at = reinterpret_cast<uint16_t *>(p) + i;
        if constexpr (N == 8) *reinterpret_cast<uint4 *>(at) = make_uint4(w[0], w[1], w[2], w[3]);
        else *reinterpret_cast<uint2 *>(at) = make_uint2(w[0], w[1]);
    } else {
        float4 *at = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p) + i);
#pragma unroll
        for (int k = 0; k < N / 4; ++k) at[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
}

__device__ __forceinline__ float sigmoid_f32(float v) { return (float)(1.0 / (1.0 + exp(-(double)v))); }
__device__ __forceinline__ float rsqrt_of(float mean_sq, float eps) { return (float)(1.0 / sqrt((double)__fadd_rn(mean_sq, eps))); }

// scale [3] (kHead: [1]) and base into shared memory by threads 0 .. 31, early in a kernel: read where they are used, they
// would stand in the serial chain of the coefficients.
template <bool kHead>
__device__ __forceinline__ void load_coefficients(float *s_coef, const float *scale, const float *base, uint32_t tid) {
    if (tid < (kHead ? 1u : 3u)) s_coef[tid] = __ldcg(scale + tid);
    if (tid < (kHead ? kHc : kMixMax)) s_coef[3u + tid] = __ldcg(base + tid);
}

// a / s rounded to nearest, by Markstein's method (IBM Journal of Research and Development 34, 1990): a reciprocal y with its error taken
// out once, q = a y, and q corrected by y times the remainder a - q s, which a fused multiply-add gives exactly.  For positive numbers from 2^-60
// to 2^60 (from_range below kInRange), where nothing on the way leaves the range of normal numbers.  The division operator looks
// at its operands first and costs a serial chain twice as much.
__device__ __forceinline__ float quotient(float a, float s) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    y = __fmaf_rn(__fmaf_rn(-s, y, 1.0f), y, y);
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-s, q, a), y, q);
}
constexpr uint32_t kInRange = 120u << 23;
__device__ __forceinline__ uint32_t from_range(float v) { return __float_as_uint(v) - (67u << 23); }

// hc.py:19-84: 24 logits -> pre [4], post [4], comb [4][4], F32 in the reference's order, in two warps, as comb is a chain several
// times as long as the rest.  Both make the logits of the sums (lane m: row m's; lane n_mix: the sum of squares) and leave them in a row of
// shared memory of their own.
template <bool kHead>
__device__ __forceinline__ void mix_logits(double sum, uint32_t n, float norm_eps, uint32_t lane, float *s_mix) {
    constexpr uint32_t n_mix = kHead ? kHc : kMixMax;
    const float rs = rsqrt_of((float)(__shfl_sync(0xffffffffu, sum, n_mix) / (double)n), norm_eps);
    if (lane < n_mix) s_mix[lane] = __fmul_rn((float)sum, rs);
    __syncwarp();
}
// lanes 0 .. 3
__device__ __forceinline__ float pre_of(const float *mixes, const float *scale, const float *base, float eps, uint32_t lane) {
    return __fadd_rn(sigmoid_f32(__fadd_rn(__fmul_rn(mixes[lane], scale[0]), base[lane])), eps);
}
__device__ __forceinline__ float post_of(const float *mixes, const float *scale, const float *base, uint32_t lane) {
    return __fmul_rn(2.0f, sigmoid_f32(__fadd_rn(__fmul_rn(mixes[kHc + lane], scale[1]), base[kHc + lane])));
}
// comb by a warp: lane l < 16 owns comb[l / 4][l % 4]; a row's or column's four values are fetched with shuffles and added in
// index order, as the Python sums do.  All 32 lanes call it.
__device__ __forceinline__ float sinkhorn_warp(const float *mixes, const float *scale, const float *base, uint32_t iters, float eps,
                                               uint32_t lane) {
    const uint32_t l = lane & 15u, i = l >> 2, j = l & 3u;
    float c = __fadd_rn(__fmul_rn(mixes[2 * kHc + l], scale[2]), base[2 * kHc + l]);
    auto row_sum = [&](float v, bool is_max) {
        const float r0 = __shfl_sync(0xffffffffu, v, i * 4u), r1 = __shfl_sync(0xffffffffu, v, i * 4u + 1u);
        const float r2 = __shfl_sync(0xffffffffu, v, i * 4u + 2u), r3 = __shfl_sync(0xffffffffu, v, i * 4u + 3u);
        if (is_max) return fmaxf(fmaxf(fmaxf(r0, r1), r2), r3);
        return __fadd_rn(__fadd_rn(__fadd_rn(r0, r1), r2), r3);
    };
    auto col_sum = [&](float v) {
        const float r0 = __shfl_sync(0xffffffffu, v, j), r1 = __shfl_sync(0xffffffffu, v, 4u + j);
        const float r2 = __shfl_sync(0xffffffffu, v, 8u + j), r3 = __shfl_sync(0xffffffffu, v, 12u + j);
        return __fadd_rn(__fadd_rn(__fadd_rn(r0, r1), r2), r3);
    };
    // stable row softmax, + eps
    c = (float)exp((double)__fsub_rn(c, row_sum(c, true)));
    const float first = __fadd_rn(__fdiv_rn(c, row_sum(c, false)), eps);   // (may be as small as eps, and the quotient a zero)
    auto rounds = [&](auto divide) {
        c = first;
        if (iters) c = divide(c, __fadd_rn(col_sum(c), eps));
#pragma unroll 1
        for (uint32_t it = 1; it < iters; ++it) {
            c = divide(c, __fadd_rn(row_sum(c, false), eps));
            c = divide(c, __fadd_rn(col_sum(c), eps));
        }
    };
    // 2 x 20 half rounds one after the other: 142 clocks each with the division operator, 108 so.  A value out of `quotient`'s range on the
    // way (an eps far below 1e-18, an infinity): once more with the operator.
    uint32_t out = 0u;
    rounds([&](float a, float d) {
        out = max(out, max(from_range(a), from_range(d)));
        return quotient(a, d);
    });
    if (__any_sync(0xffffffffu, out >= kInRange)) rounds([](float a, float d) { return __fdiv_rn(a, d); });
    return c;
}

// sum_h pre[h] v[h] in stream order
template <int N>
__device__ __forceinline__ void sum_streams(const float (&v)[kHc][N], const float (&pre)[kHc], float (&acc)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
        acc[k] = __fmul_rn(pre[0], v[0][k]);
#pragma unroll
        for (uint32_t h = 1; h < kHc; ++h) acc[k] = __fadd_rn(acc[k], __fmul_rn(pre[h], v[h][k]));
    }
}
// reduced[d] = sum_h pre[h] x[h][d] for N consecutive d.
template <bool kBf16, int N>
__device__ __forceinline__ void reduce_streams(const void *x, size_t x0, uint32_t hidden, uint32_t d, const float (&pre)[kHc],
                                               float (&acc)[N], bool vec) {
    float v[kHc][N];
#pragma unroll
    for (uint32_t h = 0; h < kHc; ++h) stream_ldn<kBf16, N>(x, x0 + (size_t)h * hidden + d, v[h], vec);
    sum_streams<N>(v, pre, acc);
}

// `v` to the same shared-memory variable of CTA `r` of the cluster, counted in bytes on its barrier
__device__ __forceinline__ void store_counted(uint32_t at, uint32_t bar, uint32_t r, double v) {
    asm volatile(
        "{\n.reg .b32 a, b;\n"
        "mapa.shared::cluster.u32 a, %0, %2;\n"
        "mapa.shared::cluster.u32 b, %1, %2;\n"
        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [a], %3, [b];\n}" ::"r"(at),
        "r"(bar), "r"(r), "l"(__double_as_longlong(v))
        : "memory");
}
// Whether all that is counted on the barrier's first phase has come, bounded (kSpin); by a whole warp, which then reads it.
__device__ __forceinline__ bool counted_stores_come(uint32_t bar) {
    bool come = false;
#pragma unroll 1
    for (uint32_t i = 0; i < kSpin && !(come = mbar_try(bar, 0u)); ++i) {
    }
    // (the stores are other CTAs', and the tries are at this one's scope)
    uint32_t seen;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
        "selp.b32 %0, 1, 0, p;\n}"
        : "=r"(seen)
        : "r"(bar)
        : "memory");
    return __all_sync(0xffffffffu, come && seen);
}

// hc_pre (and, kHead, the head's reduce, final_head.py:43-81: hc logits, pre = sigmoid(mix * scale + base) + eps
// only) of few tokens: one cluster of sixteen CTAs per token (the head fewer for more tokens: launch_hc_pre).  The call is all
// latency: 1.5 MB of fn per token, then a serial chain of 20 Sinkhorn rounds.  Every CTA takes its share of the
// flattened streams against all rows of fn (98 KB, all loads in flight together), the partial sums cross in
// shared memory, every CTA makes the coefficients itself and reduces its share of the hidden vector: no scratch, no second
// launch, no vote.  One token of 4096, calls one after another: 10.9 us in the two launches of then, 8.1 with clusters, 5.9 now.  Marks of the 8.1,
// in clocks: start and cluster barrier 1200, rows and products 3550, the warps' sums 2100, their exchange 1700, logits and pre 1400, comb
// 6400 (20 Sinkhorn rounds of one warp); now 1200, 3050, 350, 1400, and comb 5700 straight behind its logits, with pre beside it.
constexpr uint32_t kPreThreads = 512, kPreRow = (kPreThreads - 32u) * 8u;   // most elements of a CTA's share of the hidden vector
template <bool kBf16, bool kHead, uint32_t kCluster>
__global__ void __launch_bounds__(kPreThreads)
k_hc_pre(const void *__restrict__ x, const float *__restrict__ fn, const float *__restrict__ scale, const float *__restrict__ base,
         uint32_t hidden, float norm_eps, uint32_t iters, float hc_eps, void *__restrict__ reduced, float *__restrict__ post_out,
         float *__restrict__ comb_out, float *__restrict__ pre_out, uint32_t vec, uint32_t *status) {
    constexpr uint32_t n_mix = kHead ? kHc : kMixMax, kRows = n_mix / 2u;   // rows per half of the CTA
    __shared__ double s_warp[kPreThreads / 32][kRows + 1];
    __shared__ double s_part[kCluster][n_mix + 1];                      // [n_mix]: the sum of squares
    __shared__ float s_mix[2][n_mix], s_pre[kHc], s_coef[3 + n_mix];         // [3 + n_mix]: scale, base
    __shared__ __align__(8) uint64_t s_bar;                                  // all CTAs' sums are in s_part
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), t = blockIdx.y, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t n = kHc * hidden, share = n / kCluster, k0 = rank * share;   // a multiple of 64
    const uint32_t half = tid >> 8, c = tid & 255u;                          // half of the rows, column of four elements
    constexpr uint32_t kSums = kHead ? 4u : 16u;   // the rows of a half and the squares, rounded up
    double acc[kSums], ss = 0.0;
#pragma unroll
    for (uint32_t m = 0; m < kSums; ++m) acc[m] = 0.0;
    float4 f[kRows];
    auto fetch = [&](uint32_t i) {
#pragma unroll
        for (uint32_t m = 0; m < kRows; ++m) f[m] = __ldcg(reinterpret_cast<const float4 *>(fn + (size_t)(half * kRows + m) * n + k0 + i));
    };
    if (tid == 0u) {
        mbar_init(smem_u32(&s_bar), 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_arrive_expect(smem_u32(&s_bar), kCluster * (n_mix + 1u) * (uint32_t)sizeof(double));
    }
    cluster.barrier_arrive();
    dependency_wait();
    if (c * 4u < share) fetch(c * 4u);
    load_coefficients<kHead>(s_coef, scale, base, tid);
    for (uint32_t i = c * 4u; i < share; i += 1024u) {
        float v[4];
        if constexpr (kBf16) {
            const uint2 q = __ldcg(reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(x) + (size_t)t * n + k0 + i));
            v[0] = __uint_as_float(q.x << 16), v[1] = __uint_as_float(q.x & 0xffff0000u);
            v[2] = __uint_as_float(q.y << 16), v[3] = __uint_as_float(q.y & 0xffff0000u);
        } else {
            const float4 q = __ldcg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(x) + (size_t)t * n + k0 + i));
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        }
        if (i != c * 4u) fetch(i);
        const double d0 = v[0], d1 = v[1], d2 = v[2], d3 = v[3];
#pragma unroll
        for (uint32_t m = 0; m < kRows; ++m) acc[m] += (d0 * (double)f[m].x + d1 * (double)f[m].y) + (d2 * (double)f[m].z + d3 * (double)f[m].w);
        if (half == 0u) ss += (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
    }
    // (thirteen values by five exchanges each, 130 shuffles a warp and sixteen warps, were a microsecond of the chain)
    acc[kRows] = ss;
    const double sum = warp_sums(acc, lane);
    constexpr uint32_t kLanes = 32u / kSums;
    if (lane % kLanes == 0u && lane / kLanes <= kRows) s_warp[warp][lane / kLanes] = sum;
    __syncthreads();
    cluster.barrier_wait();  // every CTA of the cluster runs: its shared memory may be written
    if (tid <= n_mix) {
        const uint32_t w0 = tid < n_mix ? (tid / kRows) * 8u : 0u, m = tid < n_mix ? tid % kRows : kRows;
        double s = 0.0;
#pragma unroll
        for (uint32_t w = 0; w < 8u; ++w) s += s_warp[w0 + w][m];
        // counted stores: a barrier of the cluster behind plain ones takes 1200 clocks
#pragma unroll
        for (uint32_t r = 0; r < kCluster; ++r) store_counted(smem_u32(&s_part[rank][tid]), smem_u32(&s_bar), r, s);
    }
    const uint32_t part = hidden / kCluster;   // a multiple of 16
    const bool comb_here = !kHead && rank == 0u;
    // A CTA leaves when all sums have come, so none is stored into one that has left.  Sums that do not come make the coefficients NaN and set the
    // status word; the warps that have waited for them then stay until every other CTA of the cluster has left or stays likewise, and
    // once more a wait's length for what is on its way.
    bool come = true;
    if (warp == 0u || warp == 1u) come = counted_stores_come(smem_u32(&s_bar));
    auto leave = [&] {
        if (come) return;
        if (lane == 0u) atomicExch(status, 0x550Au);
        __syncwarp();
        cluster.barrier_arrive();
        cluster.barrier_wait();
        mbar_drain(smem_u32(&s_bar), 0u);
    };
    if (warp == 1u || (warp == 0u && comb_here)) {
        double s = come ? 0.0 : __longlong_as_double(-1ll);
        if (lane <= n_mix) {
#pragma unroll
            for (uint32_t r = 0; r < kCluster; ++r) s += s_part[r][lane];
        }
        mix_logits<kHead>(s, n, norm_eps, lane, s_mix[warp]);
    }
    if (warp == 0u) {
        // comb, while the others go on; this warp has no part of the streams
        if (comb_here) {
            const float comb = sinkhorn_warp(s_mix[0], s_coef, s_coef + 3, iters, hc_eps, lane);
            if (lane < kHc * kHc) comb_out[(size_t)t * kHc * kHc + lane] = comb;
        }
        leave();
        return;
    }
    if (warp == 1u && lane < kHc) {
        const float pre = pre_of(s_mix[1], s_coef, s_coef + 3, hc_eps, lane);
        s_pre[lane] = pre;
        if (pre_out && rank == 0u) pre_out[(size_t)t * kHc + lane] = pre;
    }
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(kPreThreads - 32u) : "memory");
    if (!kHead && rank == 0u && warp == 1u && lane < kHc) post_out[(size_t)t * kHc + lane] = post_of(s_mix[1], s_coef, s_coef + 3, lane);
    const float pre[kHc] = {s_pre[0], s_pre[1], s_pre[2], s_pre[3]};
    // (from the last thread on: the first warp, which has left, would come in above kPreRow elements)
    for (uint32_t i = (kPreThreads - 1u - tid) * 8u; i < part; i += kPreThreads * 8u) {
        float v[8];
        reduce_streams<kBf16, 8>(x, (size_t)t * n, hidden, rank * part + i, pre, v, vec != 0u);
        stream_stn<kBf16, 8>(reduced, (size_t)t * hidden + rank * part + i, v, vec != 0u);
    }
    leave();
}

// The dot products of many tokens with the rows of fn, and the sums of squares, on mma.m8n8k4.f64: a CTA takes
// sixteen tokens and a slice of K, each of its eight warps a part of the slice.  A vector kernel with a CTA per
// (row, token) read every token 24 times and every row once per token and converted all of it to double each
// time (70 us for 370 tokens of 4096); here a row's element serves sixteen tokens and a token's 24 rows (12 us:
// the FP64 pipe's 64 products per clock and SM bound it at 8).  K is permuted inside steps of sixteen: lane q of
// a quad takes four consecutive elements as its slots of four MMAs.  Writes partial sums [slice][token][25] in double.
constexpr uint32_t kDotTokens = 16, kHcSlices = 64;
template <bool kBf16, bool kHead>
__global__ void __launch_bounds__(256)
k_hc_dots(const void *__restrict__ x, const float *__restrict__ fn, uint32_t n, uint32_t n_tokens, double *__restrict__ partial) {
    constexpr uint32_t kMix = kHead ? kHc : kMixMax, kTiles = (kMix + 7u) / 8u;   // rows of fn, tiles of eight of them
    __shared__ double s_acc[8][kDotTokens][kMix + 1];
    dependency_wait();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, g = lane >> 2, q = lane & 3u;
    // steps of sixteen k, dealt to the warps of all slices as evenly as whole steps go
    const uint32_t steps = n >> 4, parts = gridDim.y * 8u, me = blockIdx.y * 8u + warp;
    const uint32_t t0 = blockIdx.x * kDotTokens, k0 = steps * me / parts * 16u + q * 4u, k1 = steps * (me + 1u) / parts * 16u + q * 4u;
    const uint32_t ta = min(t0 + g, n_tokens - 1u), tb = min(t0 + g + 8u, n_tokens - 1u);
    double c[2][kTiles][2] = {}, ss[2] = {0.0, 0.0};
    auto load4 = [&](uint32_t t, uint32_t k, float (&v)[4]) {
        if constexpr (kBf16) {
            const uint2 w = __ldcg(reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(x) + (size_t)t * n + k));
            v[0] = __uint_as_float(w.x << 16), v[1] = __uint_as_float(w.x & 0xffff0000u);
            v[2] = __uint_as_float(w.y << 16), v[3] = __uint_as_float(w.y & 0xffff0000u);
        } else {
            const float4 w = __ldcg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(x) + (size_t)t * n + k));
            v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
        }
    };
#pragma unroll 2
    for (uint32_t k = k0; k < k1; k += 16u) {
        float va[4], vb[4];
        load4(ta, k, va);
        load4(tb, k, vb);
        float4 w[kTiles];   // (the head's four rows twice: columns 4..7 of its tile are not used)
#pragma unroll
        for (uint32_t m = 0; m < kTiles; ++m) w[m] = __ldcg(reinterpret_cast<const float4 *>(fn + (size_t)((m * 8u + g) % kMix) * n + k));
#pragma unroll
        for (uint32_t s = 0; s < 4; ++s) {
            const double a = va[s], b = vb[s];
            ss[0] += a * a;
            ss[1] += b * b;
#pragma unroll
            for (uint32_t m = 0; m < kTiles; ++m) {
                const double f = s == 0u ? w[m].x : (s == 1u ? w[m].y : (s == 2u ? w[m].z : w[m].w));
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                             : "+d"(c[0][m][0]), "+d"(c[0][m][1])
                             : "d"(a), "d"(f));
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                             : "+d"(c[1][m][0]), "+d"(c[1][m][1])
                             : "d"(b), "d"(f));
            }
        }
    }
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
#pragma unroll
        for (uint32_t m = 0; m < kTiles; ++m)
#pragma unroll
            for (uint32_t e = 0; e < 2; ++e)
                if (m * 8u + 2u * q + e < kMix) s_acc[warp][h * 8u + g][m * 8u + 2u * q + e] = c[h][m][e];
        ss[h] += __shfl_xor_sync(0xffffffffu, ss[h], 1);
        ss[h] += __shfl_xor_sync(0xffffffffu, ss[h], 2);
        if (q == 0u) s_acc[warp][h * 8u + g][kMix] = ss[h];
    }
    __syncthreads();
    for (uint32_t i = tid; i < kDotTokens * (kMix + 1u); i += 256u) {
        const uint32_t t = i / (kMix + 1u), m = i - t * (kMix + 1u);
        double s = 0.0;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) s += s_acc[w][t][m];
        if (t0 + t < n_tokens) partial[((size_t)blockIdx.y * n_tokens + t0 + t) * (kMix + 1u) + m] = s;
    }
}

// One CTA per token: the coefficients from the partial sums (one warp), then the reduced vector.  All latency: the slices' sums
// (added one after the other by one warp, four loads in flight, they were half of a call of 20 tokens: 10.5 us, now 8.1), the
// coefficients, the streams (a call of 20 tokens of 4096 8.2 us, 7.0 with comb in a warp of its own and its rounds shorter, 370 tokens 20.1 and
// 19.0).  kAhead: a thread reads its first N values of every stream in front of the wait for the sums (the rule
// is the launch's).
template <bool kBf16, bool kHead, int N, bool vec, bool kAhead>
__global__ void __launch_bounds__(256)
k_hc_reduce(const void *__restrict__ x, const double *__restrict__ partial, uint32_t slices, const float *__restrict__ scale,
            const float *__restrict__ base, uint32_t hidden, float norm_eps, uint32_t iters, float hc_eps, void *__restrict__ reduced,
            float *__restrict__ post_out, float *__restrict__ comb_out, float *__restrict__ pre_out) {
    constexpr uint32_t kMix = kHead ? kHc : kMixMax;
    __shared__ double s_sum[8][kMix + 1];
    __shared__ float s_pre[kHc], s_mix[2][kMix], s_coef[3 + kMix];
    // k_hc_dots in front of this launch has waited, so everything in front of that kernel is complete: the launch behind may be
    // set up at once, and the streams may be read in front of the wait for the sums.
    cudaTriggerProgrammaticLaunchCompletion();
    const uint32_t t = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr uint32_t kFirst = kHead ? 0u : 32u;   // (the coefficients' warp has no part of the streams)
    uint32_t d = (threadIdx.x - kFirst) * N;        // (that warp's is beyond them)
    float v[kHc][N];
    if (kAhead && d < hidden) {
#pragma unroll
        for (uint32_t h = 0; h < kHc; ++h) stream_ldn<kBf16, N>(x, ((size_t)t * kHc + h) * hidden + d, v[h], vec);
    }
    cudaGridDependencySynchronize();
    // the slices' sums: a warp takes every eighth, at most eight of them, all loads in flight together
    if (lane <= kMix) {
        double u[8], s = 0.0;
#pragma unroll
        for (uint32_t k = 0; k < 8u; ++k) {
            const uint32_t p = warp + 8u * k;
            u[k] = p < slices ? __ldcg(partial + ((size_t)p * gridDim.x + t) * (kMix + 1u) + lane) : 0.0;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8u; ++k) s += u[k];
        s_sum[warp][lane] = s;
    }
    if (warp == 0u) load_coefficients<kHead>(s_coef, scale, base, lane);
    __syncthreads();
    constexpr uint32_t kPreWarp = kHead ? 0u : 1u;
    if (warp <= kPreWarp) {
        double s = 0.0;
        if (lane <= kMix) {
#pragma unroll
            for (uint32_t w = 0; w < 8u; ++w) s += s_sum[w][lane];
        }
        mix_logits<kHead>(s, kHc * hidden, norm_eps, lane, s_mix[warp]);
    }
    if (!kHead && warp == 0u) {  // the other warps reduce the streams meanwhile
        const float comb = sinkhorn_warp(s_mix[0], s_coef, s_coef + 3, iters, hc_eps, lane);
        if (lane < kHc * kHc) comb_out[(size_t)t * kHc * kHc + lane] = comb;
        return;
    }
    if (warp == kPreWarp && lane < kHc) {
        const float pre = pre_of(s_mix[kPreWarp], s_coef, s_coef + 3, hc_eps, lane);
        s_pre[lane] = pre;
        if (kHead) pre_out[(size_t)t * kHc + lane] = pre;
    }
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(256u - kFirst) : "memory");
    if (!kHead && warp == kPreWarp && lane < kHc) post_out[(size_t)t * kHc + lane] = post_of(s_mix[kPreWarp], s_coef, s_coef + 3, lane);
    const float pre[kHc] = {s_pre[0], s_pre[1], s_pre[2], s_pre[3]};
    if constexpr (kAhead) {
        if (d < hidden) {
            float o[N];
            sum_streams<N>(v, pre, o);
            stream_stn<kBf16, N>(reduced, (size_t)t * hidden + d, o, vec);
        }
        d += (256u - kFirst) * N;
    }
    for (; d < hidden; d += (256u - kFirst) * N) {
        float o[N];
        reduce_streams<kBf16, N>(x, (size_t)t * kHc * hidden, hidden, d, pre, o, vec);
        stream_stn<kBf16, N>(reduced, (size_t)t * hidden + d, o, vec);
    }
}

// hc.py:127-148: merged[t][o][d] = post[o] * branch[d] + sum_h comb[h][o] * residual[h][d]; N d per thread.  A
// token's twenty coefficients are the same for all its threads, so they are read through the L1; F32 values go four to a
// thread, because the lanes' 16-byte accesses then meet in whole lines (4096, us, before these two and now: 150 tokens
// F32 7.1 -> 3.3, 1024 28.2 -> 24.5; BF16 16 tokens 2.1 -> 1.7, 1024 10.6 -> 10.2).
template <bool kBf16, int N, bool vec, bool kTight = false>
__global__ void __launch_bounds__(128, kTight ? 8 : 0)
k_hc_post(const void *__restrict__ branch, const void *__restrict__ residual, const float *__restrict__ post,
          const float *__restrict__ comb, uint32_t hidden, void *__restrict__ merged) {
    const uint32_t d = (blockIdx.x * 128u + threadIdx.x) * N, t = blockIdx.y;
    dependency_wait();
    if (d >= hidden) return;
    float r[kHc][N], b[N], c[kHc * kHc], p[kHc];
#pragma unroll
    for (uint32_t h = 0; h < kHc; ++h) {
        stream_ldn<kBf16, N>(residual, ((size_t)t * kHc + h) * hidden + d, r[h], vec);
        p[h] = ld_f32(post + (size_t)t * kHc + h);
    }
    stream_ldn<kBf16, N>(branch, (size_t)t * hidden + d, b, vec);
#pragma unroll
    for (uint32_t i = 0; i < kHc * kHc; ++i) c[i] = ld_f32(comb + (size_t)t * kHc * kHc + i);
#pragma unroll
    for (uint32_t o = 0; o < kHc; ++o) {
        float v[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            float s = __fmul_rn(c[o], r[0][k]);
#pragma unroll
            for (uint32_t h = 1; h < kHc; ++h) s = __fadd_rn(s, __fmul_rn(c[h * kHc + o], r[h][k]));
            v[k] = __fadd_rn(__fmul_rn(p[o], b[k]), s);
        }
        stream_stn<kBf16, N>(merged, ((size_t)t * kHc + o) * hidden + d, v, vec);
    }
}

// final_head.py:84-110: out = w * (x * rsqrt(mean(x^2) + eps)); one CTA per token, N values per thread and step, kSteps
// steps.  kHeld: the token stays in registers and is read once.  The weight is the same for all tokens and comes
// through the L1.  All tokens read and written at once bound it, so the registers have to leave room for them: kBlocks
// CTAs per SM (the launch's rule).  kVec: the buffers are aligned to 16 bytes, are not, or either (`aligned` says which).
constexpr int kUnaligned = 0, kAligned = 1, kEither = 2;
template <bool kBf16, int N, int kSteps, int kBlocks, bool kHeld, int kVec>
__global__ void __launch_bounds__(256, kBlocks)
k_rms_norm(const void *__restrict__ x, const float *__restrict__ w, uint32_t hidden, float eps, void *__restrict__ out, uint32_t aligned) {
    __shared__ double red[8];
    const bool vec = kVec == kEither ? aligned != 0u : kVec == kAligned;
    const uint32_t t = blockIdx.x;
    dependency_wait();
    float v[kHeld ? kSteps : 1][N];
    double ss = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < kSteps; ++i) {
        const uint32_t d = (i * 256u + threadIdx.x) * N;
        float(&vi)[N] = v[kHeld ? i : 0];
        if (d < hidden) {
            stream_ldn<kBf16, N>(x, (size_t)t * hidden + d, vi, vec);
#pragma unroll
            for (int k = 0; k < N; ++k) ss += (double)vi[k] * (double)vi[k];
        }
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31u) == 0u) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += red[i];
    const float rs = rsqrt_of((float)(ss / (double)hidden), eps);
#pragma unroll
    for (uint32_t i = 0; i < kSteps; ++i) {
        const uint32_t d = (i * 256u + threadIdx.x) * N;
        float(&vi)[N] = v[kHeld ? i : 0];
        if (d < hidden) {
            if (!kHeld) stream_ldn<kBf16, N>(x, (size_t)t * hidden + d, vi, vec);
            float wv[N];
#pragma unroll
            for (int k = 0; k < N; k += 4) {
                if (vec) {
                    const float4 q = ld_f32x4(reinterpret_cast<const float4 *>(w + d + k));
                    wv[k] = q.x, wv[k + 1] = q.y, wv[k + 2] = q.z, wv[k + 3] = q.w;
                } else {
                    wv[k] = ld_f32(w + d + k), wv[k + 1] = ld_f32(w + d + k + 1), wv[k + 2] = ld_f32(w + d + k + 2), wv[k + 3] = ld_f32(w + d + k + 3);
                }
            }
#pragma unroll
            for (int k = 0; k < N; ++k) wv[k] = __fmul_rn(wv[k], __fmul_rn(vi[k], rs));
            stream_stn<kBf16, N>(out, (size_t)t * hidden + d, wv, vec);
        }
    }
}

// executor.py:638-668 for the hash-routed layers: the ids are the token's row of tid2eid, the weights the
// router's scores of those experts, normalised and scaled.  One CTA per token, warp j scores expert j.
__global__ void __launch_bounds__(256)
k_router_hash(const float *__restrict__ x, const uint16_t *__restrict__ wr, const long long *__restrict__ tid2eid,
              uint32_t n_experts, uint32_t hidden, uint32_t top_k, uint32_t score_fn, float route_scale,
              int32_t *__restrict__ ids_out, float *__restrict__ weights_out) {
    __shared__ float s_sc[8];
    const uint32_t t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (warp < top_k) {
        const long long e = tid2eid[(size_t)t * top_k + warp];
        double acc = 0.0;
        if (e >= 0 && (unsigned long long)e < n_experts) {
            const uint16_t *row = wr + (size_t)e * hidden;
            for (uint32_t k = lane; k < hidden; k += 32u)
                acc += (double)__ldg(x + (size_t)t * hidden + k) * (double)__uint_as_float((uint32_t)__ldg(row + k) << 16);
        }
        acc = warp_sum(acc);
        if (lane == 0) {
            s_sc[warp] = router_score_f32(acc, score_fn);
            ids_out[(size_t)t * top_k + warp] = (int32_t)e;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
        for (uint32_t j = 0; j < top_k; ++j) sum = __fadd_rn(sum, s_sc[j]);
        for (uint32_t j = 0; j < top_k; ++j) weights_out[(size_t)t * top_k + j] = __fmul_rn(__fdiv_rn(s_sc[j], sum), route_scale);
    }
}

__global__ void __launch_bounds__(256) k_bf16_to_f32(const uint16_t *__restrict__ in, float *__restrict__ out, uint32_t n) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i < n) out[i] = __uint_as_float((uint32_t)__ldg(in + i) << 16);
}
// The end of the executor's expert step: the branch rounded to BF16 (left in branch_out if the caller wants it)
// and expanded into the four streams as k_hc_post does.  One token.  y: the layer's sums, or kNoSum where it wrote none.
__global__ void __launch_bounds__(256)
k_branch_post(float *__restrict__ y, uint16_t *__restrict__ branch_out, const void *__restrict__ residual,
              const float *__restrict__ post, const float *__restrict__ comb, uint32_t hidden, void *__restrict__ merged) {
    const uint32_t d = blockIdx.x * 256u + threadIdx.x;
    dependency_wait();
    if (d >= hidden) return;
    float r[kHc], c[kHc * kHc], p[kHc];
#pragma unroll
    for (uint32_t h = 0; h < kHc; ++h) {
        r[h] = stream_ld<true>(residual, (size_t)h * hidden + d);
        p[h] = __ldcg(post + h);
    }
#pragma unroll
    for (uint32_t i = 0; i < kHc * kHc; ++i) c[i] = __ldcg(comb + i);
    const float v = __ldcg(y + d);
    y[d] = __uint_as_float(kNoSum);
    if (__float_as_uint(v) == kNoSum) return;
    const __nv_bfloat16 b16 = __float2bfloat16_rn(v);
    if (branch_out) branch_out[d] = *reinterpret_cast<const uint16_t *>(&b16);
    const float b = __bfloat162float(b16);
#pragma unroll
    for (uint32_t o = 0; o < kHc; ++o) {
        float s = __fmul_rn(c[o], r[0]);
#pragma unroll
        for (uint32_t h = 1; h < kHc; ++h) s = __fadd_rn(s, __fmul_rn(c[h * kHc + o], r[h]));
        stream_st<true>(merged, (size_t)o * hidden + d, __fadd_rn(__fmul_rn(p[o], b), s));
    }
}

}  // namespace

cudaError_t launch_bf16_to_f32(cudaStream_t st, const uint16_t *in, float *out, uint32_t n) {
    k_bf16_to_f32<<<(n + 255u) / 256u, 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}
cudaError_t launch_branch_post(cudaStream_t st, uint32_t hidden, float *y, uint16_t *branch_out, const void *residual,
                               const float *post, const float *comb, void *merged) {
    return launch_pdl(k_branch_post, dim3((hidden + 255u) / 256u), dim3(256), 0, st, 0u, y, branch_out, residual, post, comb, hidden,
                      merged);
}

// The partial sums of launch_hc_pre_many.
size_t hc_scratch_bytes(uint32_t max_tokens, int sm_count) {
    // a row per slice and token: slices times groups of sixteen tokens come to six CTAs per SM at most (launch_hc_pre_many)
    return (size_t)std::max(std::max(max_tokens, kHcSlices * kDotTokens), 6u * kDotTokens * (uint32_t)sm_count) * (kMixMax + 1u) * sizeof(double);
}

// Whether all the addresses are multiples of 16 (rows of 256 and more elements keep that).
template <class... P>
static uint32_t aligned16(P... p) {
    return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) == 0u ? 1u : 0u;
}

template <bool kBf16, bool kHead, uint32_t kCluster>
static cudaError_t launch_hc_pre_cluster(cudaStream_t st, uint32_t n_tokens, uint32_t hidden, const void *x, const float *fn,
                                         const float *scale, const float *base, float norm_eps, uint32_t iters, float hc_eps,
                                         void *reduced, float *post, float *comb, float *pre, uint32_t *status) {
    static bool done[64] = {};
    if (hidden / kCluster > kPreRow) return cudaErrorInvalidValue;
    const cudaError_t e = allow_wide_clusters(k_hc_pre<kBf16, kHead, kCluster>, done);
    if (e != cudaSuccess) return e;
    return launch_pdl(k_hc_pre<kBf16, kHead, kCluster>, dim3(kCluster, n_tokens), dim3(kPreThreads), 0, st, kCluster, x, fn, scale, base,
                      hidden, norm_eps, iters, hc_eps, reduced, post, comb, pre, aligned16(x, reduced), status);
}

template <bool kBf16, bool kHead>
static cudaError_t launch_hc_pre_many(cudaStream_t st, int sm_count, uint32_t n_tokens, uint32_t hidden, const void *x, const float *fn,
                                      const float *scale, const float *base, float norm_eps, uint32_t iters, float hc_eps,
                                      double *partial, void *reduced, float *post, float *comb, float *pre) {
    // Slices of K: as many as make the CTAs fit the SMs side by side, three to an SM by their registers (the head's, with four rows
    // in place of 24, six of BF16 streams and five of F32 ones, which with six took a second round: 1024 tokens of 7168 54.3 us, so
    // 48.9, 900 of 512 8.1 and 7.4; but 300 of 7168, whose warps have five steps then, 13.6 and with five slices 15.3): one round,
    // no tail.  At most 64, which the second kernel adds up, and a step of sixteen k for every warp.  us of both launches with
    // eight or sixteen slices and a second kernel that added them in one warp, and now: 20 tokens of 4096 10.5 and 8.1, 370 23.3
    // and 20.9, 700 34.1 and 30.9, 1000 45.8 and 40.3; 900 of 1024 20.6 and 16.0.  The head: 460 of 4096 18.7 and 11.5, 1000 30.1
    // and 23.3, 704 of 512 7.5 and 6.3.
    const uint32_t groups = (n_tokens + kDotTokens - 1u) / kDotTokens, n = kHc * hidden, sms = (uint32_t)sm_count;
    const uint32_t per_sm = !kHead ? 3u : kBf16 || (hidden >= 4096u && groups * 6u <= sms) ? 6u : 5u;
    const uint32_t slices = std::max(1u, std::min({kHcSlices, hidden / 32u, per_sm * sms / groups}));
    const cudaError_t e = launch_pdl(k_hc_dots<kBf16, kHead>, dim3(groups, slices), dim3(256), 0, st, 0u, x, fn, n, n_tokens, partial);
    if (e != cudaSuccess) return e;
    auto reduce = [&](auto kernel) {
        return launch_pdl(kernel, dim3(n_tokens), dim3(256), 0, st, 0u, x, (const double *)partial, slices, scale, base, hidden, norm_eps, iters,
                          hc_eps, reduced, post, comb, pre);
    };
    constexpr int kN = kBf16 ? 8 : 4;
    if (!aligned16(x, reduced)) return reduce(k_hc_reduce<kBf16, kHead, kN, false, false>);
    // The streams in front of the wait while all CTAs are resident with the registers that takes (64, F32 48: four and five to an
    // SM).  us of the site, with and without: 370 tokens of 4096 30.6 and 32.3, 550 44.4 and 46.0, 650 46.7 and 43.3; F32 600 46.0 and 47.9,
    // 1000 80.0 and 76.2.  (Twice the values: two CTAs to an SM, 370 tokens 34.5.)
    const bool ahead = n_tokens <= (kBf16 ? 4u : 5u) * sms;
    return ahead ? reduce(k_hc_reduce<kBf16, kHead, kN, true, true>) : reduce(k_hc_reduce<kBf16, kHead, kN, true, false>);
}

// hc_pre by a cluster of CTAs per token, for as many tokens as leave a fifth of the SMs (launch_hc_pre has the figures).
static bool hc_pre_in_clusters(uint32_t n_tokens, uint32_t sms) { return 16u * n_tokens * 5u <= sms * 4u; }

// scratch: hc_scratch_bytes of the most tokens; status: the context's word (0x550A: the sums of a token's other CTAs have not come).  Returns the number of kernels launched.
int launch_hc_pre(cudaStream_t st, int sm_count, bool bf16, bool head, uint32_t n_tokens, uint32_t hidden, const void *x, const float *fn,
                  const float *scale, const float *base, float norm_eps, uint32_t iters, float hc_eps, double *scratch, void *reduced,
                  float *post, float *comb, float *pre, uint32_t *status, cudaError_t *err) {
    // one cluster per token while the clusters fit the GPU side by side, else two launches for all tokens
    auto run = [&](auto is_bf16, auto is_head, auto size) {
        constexpr bool kB = decltype(is_bf16)::value, kH = decltype(is_head)::value;
        constexpr uint32_t kC = decltype(size)::value;
        if constexpr (kC != 0u) {
            *err = launch_hc_pre_cluster<kB, kH, kC>(st, n_tokens, hidden, x, fn, scale, base, norm_eps, iters, hc_eps, reduced, post, comb, pre,
                                                     status);
            return 1;
        } else {
            *err = launch_hc_pre_many<kB, kH>(st, sm_count, n_tokens, hidden, x, fn, scale, base, norm_eps, iters, hc_eps, scratch, reduced,
                                              post, comb, pre);
            return 2;
        }
    };
    auto of_size = [&](auto is_head, auto size) { return bf16 ? run(std::true_type{}, is_head, size) : run(std::false_type{}, is_head, size); };
    using U = uint32_t;
    const uint32_t sms = (uint32_t)sm_count;
    if (!head) {
        // A CTA with 24 rows fills an SM: on 148 SMs seven clusters of sixteen run together (4096, us: one token 5.9, seven 6.0, the
        // two launches of eight tokens 6.9).  Fourteen clusters of eight took
        // 9.7 for fourteen tokens, the two launches 8.3 (7168 11.3 and 9.7; both before what is a microsecond and more faster now).
        if (hc_pre_in_clusters(n_tokens, sms)) return of_size(std::false_type{}, std::integral_constant<U, 16>{});
        return of_size(std::false_type{}, std::integral_constant<U, 0>{});
    }
    // The head's four rows leave room for two CTAs, and smaller clusters pack closer: the largest whose CTAs come to at most
    // one and a half per SM (4096, us: 8 tokens 4.0, 20 4.5, 55 5.5, the two launches 4.7, 5.0, 6.7).  Clusters of two only of short
    // rows: up to 1024, or 1792 while their CTAs have an SM each (us, F32 streams, 64 and 111 tokens, the two launches: 512 3.3 and 3.7, 3.8 and
    // 4.6; 1024 4.0 and 4.4, 4.4 and 4.5; 1536 4.4 and 5.1, 4.9 and 5.0; 2048 5.0 and 5.9, 4.9 and 5.8; 4096, 80 tokens, 8.2 and 6.8).
    const uint32_t room = sms + sms / 2u;
    if (16u * n_tokens <= room) return of_size(std::true_type{}, std::integral_constant<U, 16>{});
    if (8u * n_tokens <= room) return of_size(std::true_type{}, std::integral_constant<U, 8>{});
    if (4u * n_tokens <= room) return of_size(std::true_type{}, std::integral_constant<U, 4>{});
    if (2u * n_tokens <= (hidden <= 1024u ? room : hidden <= 1792u ? sms : 0u)) return of_size(std::true_type{}, std::integral_constant<U, 2>{});
    return of_size(std::true_type{}, std::integral_constant<U, 0>{});
}

cudaError_t launch_hc_post(cudaStream_t st, int sm_count, bool bf16, uint32_t n_tokens, uint32_t hidden, const void *branch, const void *residual,
                           const float *post, const float *comb, void *merged) {
    const uint32_t vec = aligned16(branch, residual, merged);
    // BF16: four values a thread (8-byte accesses) while their CTAs come to at most five per SM (one token of 4096 1.4 us, eight
    // values 1.6; 64 tokens 1.9 and 2.0), above that eight (1024 tokens 9.6 us, four values 11.9).  With four and five CTAs per SM
    // calls one after another are faster with eight (148 tokens of 2048 2.04 us and 2.16), whole sites with four (370 of 1024
    // 14.8 us and 15.3, 150 of 2048 14.7 and 15.1), and values one by one much so (300 of 1024 3.0 us and 5.4).
    const bool few = (uint64_t)n_tokens * hidden <= (uint64_t)sm_count * 5u * 512u;
    // 8 to 32 tokens (two groups of k_hc_dots): the SMs divided as that kernel needs them, three CTAs of 26 KB.  Its CTAs, the next
    // site's, are to start while this kernel runs, and once the two need more than the SMs they have to share some, which an SM divided
    // otherwise makes them wait for.  Sites one after another, us: 10 tokens of 7168 17.7, so 14.4, 14 of 5120 15.7 and 13.1, 12 of 4096 12.9
    // and 12.0, 32 of 4096 14.6 and 13.1; from 64 tokens of 5120 on it gains nothing (150 of 4096 18.1 and 18.5).
    // (Fewer tokens' hc_pre is one launch, and the division itself costs one token 0.1 us.)
    const size_t divided = !hc_pre_in_clusters(n_tokens, (uint32_t)sm_count) && n_tokens <= 2u * kDotTokens ? 80u << 10 : 0u;
    auto run = [&](auto kernel, uint32_t per_thread) {
        return launch_dependent(kernel, dim3((hidden + 128u * per_thread - 1u) / (128u * per_thread), n_tokens), dim3(128), 0, st, 0u, divided,
                                branch, residual, post, comb, hidden, merged);
    };
    if (!bf16) return vec ? run(k_hc_post<false, 4, true>, 4) : run(k_hc_post<false, 4, false>, 4);
    if (!vec) return few ? run(k_hc_post<true, 4, false>, 4) : run(k_hc_post<true, 8, false, true>, 8);
    if (few) return run(k_hc_post<true, 4, true>, 4);
    // Eight values a thread take 72 registers, seven CTAs to an SM.  In 64 there are eight, so a call of four per SM starts while the
    // one in front of it runs out (148 tokens of 4096 3.2 us, so 2.45; values one by one 592 tokens of 1024 13.2 and 8.2); more CTAs are
    // faster with 72 (148 tokens of 7168 3.25 and 3.55, 900 of 4096 8.3 and 8.5).
    const bool tight = (uint64_t)((hidden + 1023u) / 1024u) * n_tokens <= 4u * (uint64_t)sm_count;
    return tight ? run(k_hc_post<true, 8, true, true>, 8) : run(k_hc_post<true, 8, true>, 8);
}

// F32 tokens: eight values per thread while a token has an SM to itself (the fewest steps in series), else four, whose
// 16-byte accesses meet in whole lines, with registers for as many CTAs per SM as there are tokens; above 4096 the
// largest batches would spill and read the token twice.  us of 4096, one form for all / now: 16 tokens 2.7 / 2.6,
// 300 5.2 / 3.6, 700 7.8 / 4.9, 1024 9.5 / 6.7; 8192 and 1024 tokens 16.4 / 12.0.  BF16 tokens are half the bytes, eight
// values to a thread always: 4096 and 700 tokens 5.8 / 3.7.
template <bool kBf16, int kSteps, int kVec>
static cudaError_t launch_rms_steps(cudaStream_t st, uint32_t sms, uint32_t n_tokens, uint32_t hidden, const void *x, const float *w, float eps,
                                    void *out, uint32_t aligned) {
    auto run = [&](auto kernel) { return launch_pdl(kernel, dim3(n_tokens), dim3(256), 0, st, 0u, x, w, hidden, eps, out, aligned); };
    if (kBf16 || n_tokens <= sms) return run(k_rms_norm<kBf16, 8, kSteps, 1, true, kVec>);
    if constexpr (!kBf16) {
        constexpr int kFour = 2 * kSteps;   // steps of four values
        if (kSteps == 1 && hidden <= 1024u) return run(k_rms_norm<false, 4, 1, 8, true, kVec>);
        if (n_tokens <= 4u * sms) return run(k_rms_norm<false, 4, kFour, 1, true, kVec>);
        if (n_tokens <= 6u * sms) return run(k_rms_norm<false, 4, kFour, 6, true, kVec>);
        return run(k_rms_norm<false, 4, kFour, 8, (kFour < 8), kVec>);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_rms_norm(cudaStream_t st, int sm_count, bool bf16, uint32_t n_tokens, uint32_t hidden, const void *x, const float *w,
                            float eps, void *out) {
    const uint32_t sms = (uint32_t)sm_count, aligned = aligned16(x, w, out);
    // The form for either kind of buffer, where it is the faster one.  us of it and of the other: aligned, short rows of few tokens (F32
    // 250 tokens of 1024 1.76 and 1.84, 8 of 2048 1.68 and 1.79; but BF16 592 of 1024 2.35 and 2.25, F32 150 of 2048 2.34 and 2.05, 4096
    // 2.7 and 2.4); not aligned, many BF16 tokens (592 of 4096 10.4 and 10.9, 1024 of 1024 5.4 and 6.0; but 148 of 2048 2.65 and 2.40),
    // many F32 ones of short rows (592 of 1024 2.65 and 2.85; but 148 2.26 and 2.22, 592 of 4096 7.5 and 7.1) and few of long ones (148
    // of 7168 6.5 and 7.0; but 250 7.8 and 7.2).
    const bool either = aligned ? n_tokens <= (hidden <= 1024u ? 3u * sms : hidden <= 2048u ? sms : 0u)
                                : n_tokens > sms ? bf16 || hidden <= 1024u : !bf16 && hidden > 4096u;
    auto run = [&](auto steps) {
        constexpr int kS = decltype(steps)::value;
        auto form = [&](auto vec) {
            constexpr int kV = decltype(vec)::value;
            return bf16 ? launch_rms_steps<true, kS, kV>(st, sms, n_tokens, hidden, x, w, eps, out, aligned)
                        : launch_rms_steps<false, kS, kV>(st, sms, n_tokens, hidden, x, w, eps, out, aligned);
        };
        if (either) return form(std::integral_constant<int, kEither>{});
        return aligned ? form(std::integral_constant<int, kAligned>{}) : form(std::integral_constant<int, kUnaligned>{});
    };
    if (hidden <= 2048u) return run(std::integral_constant<int, 1>{});
    if (hidden <= 4096u) return run(std::integral_constant<int, 2>{});
    return run(std::integral_constant<int, 4>{});
}

cudaError_t launch_router_hash(cudaStream_t st, const s14_router_desc &r, const int64_t *tid2eid) {
    k_router_hash<<<r.n_tokens, 256, 0, st>>>(r.x, r.router_weight_bf16, reinterpret_cast<const long long *>(tid2eid), r.n_experts,
                                             r.hidden, r.top_k, r.score_fn, r.route_scale, r.ids_out, r.weights_out);
    return cudaGetLastError();
}

}  // namespace s14
