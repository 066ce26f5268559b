// The shared expert of one decode token when its page is the checkpoint's FP8 page (E4M3 weights, one UE8M0
// scale per 128 x 128): w1 | w3 with the limited SwiGLU, then w2, as two launches behind the tensor-core
// layer kernel, which runs the routed MXFP4 experts; the second adds this expert's output to theirs, last in the mix's order
// (examples/s14_vulkan_numeric.rs:929-947), and in the executor's step goes on to what follows (branch and hc_post).
//
// A matvec of 25 MB: the weight stream bounds it (3.8 us at 6.55 TB/s), so every warp owns one row pair (one row
// of w2 at a time), splits K over its lanes in 16-byte pieces and has all of a row's loads in flight at once
// (115 KB per SM).  The layer kernel asks the page into the L2 while its last hand-offs leave the memory idle, and the first
// launch needs nothing of that kernel, so it runs on the SMs that kernel has left.  The vector lies in shared memory as [quarter
// of a piece][piece]: the lanes of a warp, which hold consecutive pieces, read consecutive 16 bytes.  Sums as in the FP8
// register kernels: F32 inside a piece, double across pieces and lanes, one rounding.  Measured at 4096 x 2048, other pages every
// time: the executor's step, which is the layer kernel's six experts and these two launches, takes 32.6 us.  With both launches and
// their own stream from memory in front of the layer kernel and a launch for branch and expand behind it: 39.9; behind it but
// waiting for it: 35.5; on the register kernels, which ran all seven experts, 77.2.
#include "s14_device.cuh"

namespace s14 {

namespace {

constexpr uint32_t kF8Threads = 512, kF8Warps = kF8Threads / 32u;

// n values into shared memory, transposed as above
__device__ __forceinline__ void stage_vector(float *sx, const float *x, uint32_t n) {
    const uint32_t pieces = n >> 4;
    for (uint32_t i = threadIdx.x; i < (n >> 2); i += kF8Threads)
        reinterpret_cast<float4 *>(sx)[(i & 3u) * pieces + (i >> 2)] = __ldcg(reinterpret_cast<const float4 *>(x) + i);
}
__device__ __forceinline__ void stage_vector_bf16(float *sx, const uint16_t *x, uint32_t n) {
    const uint32_t pieces = n >> 4;
    for (uint32_t i = threadIdx.x; i < (n >> 2); i += kF8Threads) {
        const uint2 b = __ldcg(reinterpret_cast<const uint2 *>(x) + i);
        reinterpret_cast<float4 *>(sx)[(i & 3u) * pieces + (i >> 2)] =
            make_float4(__uint_as_float(b.x << 16), __uint_as_float(b.x & 0xffff0000u), __uint_as_float(b.y << 16),
                        __uint_as_float(b.y & 0xffff0000u));
    }
}

// F32 dots of one 16-byte piece of N rows with the piece's sixteen staged values
template <uint32_t N>
__device__ __forceinline__ void dot_piece(const uint4 *const (&q)[N], const float *sx, uint32_t piece, uint32_t pieces, float (&dot)[N]) {
    float2 acc[N];
#pragma unroll
    for (uint32_t n = 0; n < N; ++n) acc[n] = make_float2(0.f, 0.f);
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        const float4 v = reinterpret_cast<const float4 *>(sx)[i * pieces + piece];
#pragma unroll
        for (uint32_t n = 0; n < N; ++n) {
            uint32_t h0, h1;
            e4m3x4_to_h2x2(i == 0u ? q[n]->x : (i == 1u ? q[n]->y : (i == 2u ? q[n]->z : q[n]->w)), h0, h1);
            acc[n] = __ffma2_rn(h2_to_f2(h0), make_float2(v.x, v.y), acc[n]);
            acc[n] = __ffma2_rn(h2_to_f2(h1), make_float2(v.z, v.w), acc[n]);
        }
    }
#pragma unroll
    for (uint32_t n = 0; n < N; ++n) dot[n] = acc[n].x + acc[n].y;
}

// P: 16-byte pieces of a row per lane (K / 512)
template <uint32_t P>
__device__ __forceinline__ void load_row(uint4 (&q)[P], const uint8_t *row, uint32_t lane) {
#pragma unroll
    for (uint32_t j = 0; j < P; ++j) q[j] = ld_stream(reinterpret_cast<const uint4 *>(row) + j * 32u + lane);
}
// scales: a row's codes, one per 128 elements (a piece's: piece / 8)
template <uint32_t P>
__device__ __forceinline__ float dot_row(const uint4 (&qa)[P], const uint8_t *scales, const float *sx, uint32_t lane) {
    double acc = 0.0;
#pragma unroll
    for (uint32_t j = 0; j < P; ++j) {
        const uint32_t p = j * 32u + lane;
        const uint4 *const q[1] = {&qa[j]};
        float dot[1];
        dot_piece<1>(q, sx, p, P * 32u, dot);
        acc += (double)dot[0] * ue8m0_to_f64(ld_u8(scales + (p >> 3)));
    }
    return (float)warp_sum(acc);
}
// Two rows piece by piece, so that the vector is read once and never held whole (which would not fit the registers)
template <uint32_t P>
__device__ __forceinline__ void dot_rows(const uint4 (&qa)[P], const uint4 (&qb)[P], const uint8_t *sa, const uint8_t *sb, const float *sx,
                                         uint32_t lane, float &va, float &vb) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (uint32_t j = 0; j < P; ++j) {
        const uint32_t p = j * 32u + lane;
        const uint4 *const q[2] = {&qa[j], &qb[j]};
        float dot[2];
        dot_piece<2>(q, sx, p, P * 32u, dot);
        a += (double)dot[0] * ue8m0_to_f64(ld_u8(sa + (p >> 3)));
        b += (double)dot[1] * ue8m0_to_f64(ld_u8(sb + (p >> 3)));
    }
    va = (float)warp_sum(a);
    vb = (float)warp_sum(b);
}

// h[i] = swiglu(w1[i] . x, w3[i] . x); x F32 or BF16
template <uint32_t P>
__global__ void __launch_bounds__(kF8Threads, 1)
k_fp8_expert_up(const float *__restrict__ x, const uint16_t *__restrict__ x_bf16, const uint8_t *__restrict__ page, float *__restrict__ h,
                uint32_t inter) {
    constexpr uint32_t hidden = P * 512u;
    __shared__ __align__(16) float sx[hidden];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, step = gridDim.x * kF8Warps;
    const PageView pv = page_view(page, S14_PAGE_FP8, hidden, inter);
    uint32_t row = warp * gridDim.x + blockIdx.x;  // the CTAs' numbers of rows differ by one at most
    uint4 q1[P], q3[P];
    // No wait in front: the layer kernel, which this launch follows, lets it start behind its own wait (so everything in front of
    // that kernel is complete) and touches neither the token, the page nor h.  The wait comes last, for the launch behind.
    if (row < inter) {
        load_row<P>(q1, pv.w1 + (size_t)row * hidden, lane);
        load_row<P>(q3, pv.w3 + (size_t)row * hidden, lane);
    }
    if (x_bf16) stage_vector_bf16(sx, x_bf16, hidden);
    else stage_vector(sx, x, hidden);
    __syncthreads();
#pragma unroll 1
    while (row < inter) {
        const size_t srow = (size_t)(row >> 7) * (hidden >> 7);
        float gate, up;
        dot_rows<P>(q1, q3, pv.s1 + srow, pv.s3 + srow, sx, lane, gate, up);
        if (lane == 0u) h[row] = swiglu_limit_f32(gate, up);
        row += step;
        if (row < inter) {
            load_row<P>(q1, pv.w1 + (size_t)row * hidden, lane);
            load_row<P>(q3, pv.w3 + (size_t)row * hidden, lane);
        }
    }
    dependency_wait();
}

// v[n] = routed[n] + w2[n] . h (where the layer kernel has left a sum: kNoSum): to y, or (kPost) the branch of the executor's step,
// rounded to BF16, and hc_post over the post-attention state, lane o the o-th stream (hc.py:127-148; the operations of
// k_branch_post, whose launch it saves)
template <uint32_t P, bool kPost>
__global__ void __launch_bounds__(kF8Threads, 1)
k_fp8_expert_down(const uint8_t *__restrict__ page, const float *__restrict__ h, float *routed, float *__restrict__ y,
                  const __grid_constant__ BranchPost post, uint32_t hidden) {
    constexpr uint32_t inter = P * 512u;
    __shared__ __align__(16) float sx[inter];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, step = gridDim.x * kF8Warps, o = lane & 3u;
    const PageView pv = page_view(page, S14_PAGE_FP8, hidden, inter);
    uint32_t row = warp * gridDim.x + blockIdx.x;
    uint4 qa[P], qb[P];  // this row and the warp's next one
    // what a row's result is made of beside the dot product: its sum and the streams.  Asked for in front of the row's weights, as
    // behind them it comes microseconds later (the store of kNoSum keeps the compiler from moving it: the step of 1024 x 2048 then took
    // 22.0 us instead of 19.4)
    struct Row {
        float base;
        uint32_t r[4];
    } ra = {}, rb = {};
    auto load_in = [&](Row &in, uint32_t at) {
        in.base = __ldcg(routed + at);
        if constexpr (kPost) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) in.r[i] = __ldcg(static_cast<const uint16_t *>(post.residual) + (size_t)i * hidden + at);
        }
    };
    dependency_wait();
    if (row < hidden) load_in(ra, row);
    if (row + step < hidden) load_in(rb, row + step);
    if (row < hidden) load_row<P>(qa, pv.w2 + (size_t)row * inter, lane);
    if (row + step < hidden) load_row<P>(qb, pv.w2 + (size_t)(row + step) * inter, lane);
    float c[4], p = 0.0f;
    if constexpr (kPost) {
        p = __ldcg(post.post + o);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) c[i] = __ldcg(post.comb + i * 4u + o);
    }
    stage_vector(sx, h, inter);
    __syncthreads();
#pragma unroll 1
    while (row < hidden) {
        const float base = ra.base;
        const float v = __fadd_rn(base, dot_row<P>(qa, pv.s2 + (size_t)(row >> 7) * (inter >> 7), sx, lane));
        const bool there = __float_as_uint(base) != kNoSum;
        if (lane == 0u) routed[row] = __uint_as_float(kNoSum);   // (every lane has its copy: dot_row's shuffles lie in between)
        if constexpr (kPost) {
            if (there && lane < 4u) {
                const __nv_bfloat16 b16 = __float2bfloat16_rn(v);
                if (lane == 0u && post.branch_out) post.branch_out[row] = __bfloat16_as_ushort(b16);
                float s = __fmul_rn(c[0], __uint_as_float(ra.r[0] << 16));
#pragma unroll
                for (uint32_t i = 1; i < 4; ++i) s = __fadd_rn(s, __fmul_rn(c[i], __uint_as_float(ra.r[i] << 16)));
                static_cast<uint16_t *>(post.merged)[(size_t)o * hidden + row] =
                    __bfloat16_as_ushort(__float2bfloat16_rn(__fadd_rn(__fmul_rn(p, __bfloat162float(b16)), s)));
            }
        } else {
            if (there && lane == 0u) y[row] = v;
        }
        row += step;
        ra = rb;
#pragma unroll
        for (uint32_t j = 0; j < P; ++j) qa[j] = qb[j];
        if (row + step < hidden) {
            load_in(rb, row + step);
            load_row<P>(qb, pv.w2 + (size_t)(row + step) * inter, lane);
        }
    }
}

}  // namespace

cudaError_t launch_fp8_expert(cudaStream_t st, int sm_count, const float *x, const uint16_t *x_bf16, const uint8_t *page,
                              float *h, float *routed, float *y, const BranchPost *post, uint32_t hidden, uint32_t inter) {
    const dim3 grid(sm_count), block(kF8Threads);
    cudaError_t e;
    switch (hidden >> 9) {
    case 2: e = launch_pdl(k_fp8_expert_up<2>, grid, block, 0, st, 0u, x, x_bf16, page, h, inter); break;
    case 4: e = launch_pdl(k_fp8_expert_up<4>, grid, block, 0, st, 0u, x, x_bf16, page, h, inter); break;
    default: e = launch_pdl(k_fp8_expert_up<8>, grid, block, 0, st, 0u, x, x_bf16, page, h, inter); break;
    }
    if (e != cudaSuccess) return e;
    const BranchPost bp = post ? *post : BranchPost{};
    auto down = [&](auto plain, auto with_post) {
        return launch_pdl(post ? with_post : plain, grid, block, 0, st, 0u, page, (const float *)h, routed, y, bp, hidden);
    };
    switch (inter >> 9) {
    case 2: return down(k_fp8_expert_down<2, false>, k_fp8_expert_down<2, true>);
    case 4: return down(k_fp8_expert_down<4, false>, k_fp8_expert_down<4, true>);
    default: return down(k_fp8_expert_down<8, false>, k_fp8_expert_down<8, true>);
    }
}

}  // namespace s14
