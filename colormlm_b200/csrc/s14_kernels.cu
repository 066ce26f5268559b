// sm_100a kernels of the S14 MoE expert hot path.
//
// Two summation orders are implemented for every matvec (see S14_ACCUM_* in
// include/polaris_s14_cuda.h):
//   pairwise  - a warp owns an output row, its lanes split K in 16-byte pieces
//               (128-bit coalesced loads), decode E2M1 / E4M3 with the hardware
//               cvt to f16x2, multiply-accumulate in F32 inside one scale block,
//               then carry block sums, lane sums and the final value in F64;
//   reference - a thread owns an output row and walks k in ascending order with
//               the reference's separate multiply / multiply / add per element
//               (examples/s14_vulkan_numeric.rs:1669-1714), bit-identical to it.
// The elementwise steps (limit-10 SwiGLU, route mix, ordered accumulate) use
// separate F32 multiplies and adds in both modes, as the reference does.
#include "s14_device.cuh"
#include "s14_router.cuh"

namespace s14 {

// F32 dot of 32 E2M1 codes (one 16-byte piece = one scale block) with 32
// activations held in registers; two independent even/odd chains on the packed
// F32x2 pipe.
__device__ __forceinline__ float dot32_e2m1(const uint4 &q, const float *__restrict__ xr) {
    float2 acc = make_float2(0.f, 0.f);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t h0, h1, h2, h3;
        e2m1x8_to_h2x4(w[i], h0, h1, h2, h3);
        acc = __ffma2_rn(h2_to_f2(h0), make_float2(xr[i * 8 + 0], xr[i * 8 + 1]), acc);
        acc = __ffma2_rn(h2_to_f2(h1), make_float2(xr[i * 8 + 2], xr[i * 8 + 3]), acc);
        acc = __ffma2_rn(h2_to_f2(h2), make_float2(xr[i * 8 + 4], xr[i * 8 + 5]), acc);
        acc = __ffma2_rn(h2_to_f2(h3), make_float2(xr[i * 8 + 6], xr[i * 8 + 7]), acc);
    }
    return acc.x + acc.y;
}

// F32 dot of 16 E4M3 codes (one 16-byte piece) with 16 activations.
__device__ __forceinline__ float dot16_e4m3(const uint4 &q, const float *__restrict__ xr) {
    float2 acc = make_float2(0.f, 0.f);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t h0, h1;
        e4m3x4_to_h2x2(w[i], h0, h1);
        acc = __ffma2_rn(h2_to_f2(h0), make_float2(xr[i * 4 + 0], xr[i * 4 + 1]), acc);
        acc = __ffma2_rn(h2_to_f2(h1), make_float2(xr[i * 4 + 2], xr[i * 4 + 3]), acc);
    }
    return acc.x + acc.y;
}

// ------------------------------------------------- primitive operators ------

// y[n] = sum_k x[k] * e2m1(w[n,k]) * 2^(s[n,k/32]-127).  A matrix of the checkpoint's sizes is 4 MB: launch, first
// byte and the x reads bound the call, not the bandwidth.  A warp owns NR rows at a time and splits K over its
// lanes in 16-byte pieces (one scale block each), the pieces of its rows (four each per step) in flight together and
// the first ones brought to the L2 before the wait for the kernel in front (l2_hint).  x lies in
// shared memory as [eighth of a piece][piece], so that a warp's lanes read consecutive 16 bytes; reading it
// through the L1 with a 128-byte stride between lanes, one piece in flight, took 10.6 us for 2048 x 4096
// (this kernel: 3.3).  Two rows per warp halve the x reads, which cost more than the weights (128 bytes for 16),
// once there are two rows for every warp.
constexpr uint32_t kMvThreads = 512, kMvBatch = 4, kMvMaxK = 32768;
template <uint32_t NR>
__global__ void __launch_bounds__(kMvThreads, 1)
k_mxfp4_matvec_pairwise(const float *__restrict__ x, const uint8_t *__restrict__ w, const uint8_t *__restrict__ s,
                        float *__restrict__ y, uint32_t n_rows, uint32_t k) {
    extern __shared__ __align__(16) float sx[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, groups = k >> 5;
    const uint32_t n_warps = gridDim.x * (kMvThreads / 32u);
    const uint32_t batches = (groups + 32u * kMvBatch - 1u) / (32u * kMvBatch);
    uint4 q[NR][kMvBatch];
    uint32_t sc[NR][kMvBatch];
    // rows n, n + n_warps of the step (row, batch); pieces past a row's end and rows past the matrix count as zeros
    auto fetch = [&](uint32_t n, uint32_t batch) {
#pragma unroll
        for (uint32_t r = 0; r < NR; ++r) {
            const uint32_t row = n + r * n_warps;
#pragma unroll
            for (uint32_t j = 0; j < kMvBatch; ++j) {
                const uint32_t p = (batch * kMvBatch + j) * 32u + lane;
                const bool there = row < n_rows && p < groups;
                q[r][j] = there ? ld_stream(reinterpret_cast<const uint4 *>(w + (size_t)row * (k >> 1)) + p) : make_uint4(0u, 0u, 0u, 0u);
                sc[r][j] = there ? ld_u8(s + (size_t)row * groups + p) : 0u;
            }
        }
    };
    uint32_t n = warp * gridDim.x + blockIdx.x;  // the CTAs' numbers of rows differ by one at most
#pragma unroll
    for (uint32_t r = 0; r < NR; ++r)
#pragma unroll
        for (uint32_t j = 0; j < kMvBatch; ++j) {
            const uint32_t row = n + r * n_warps, p = j * 32u + lane;
            if (row < n_rows && p < groups) {
                l2_hint(w + (size_t)row * (k >> 1) + p * 16u);
                l2_hint(s + (size_t)row * groups + p);
            }
        }
    dependency_wait();
    if (n < n_rows) fetch(n, 0u);
    for (uint32_t i = threadIdx.x; i < (k >> 2); i += kMvThreads)
        reinterpret_cast<float4 *>(sx)[(i & 7u) * groups + (i >> 3)] = __ldcg(reinterpret_cast<const float4 *>(x) + i);
    __syncthreads();
    while (n < n_rows) {
        double acc[NR];
#pragma unroll
        for (uint32_t r = 0; r < NR; ++r) acc[r] = 0.0;
        const uint32_t next = n + NR * n_warps;
        for (uint32_t b = 0; b < batches; ++b) {
            uint4 cur[NR][kMvBatch];
            uint32_t cs[NR][kMvBatch];
#pragma unroll
            for (uint32_t r = 0; r < NR; ++r)
#pragma unroll
                for (uint32_t j = 0; j < kMvBatch; ++j) cur[r][j] = q[r][j], cs[r][j] = sc[r][j];
            if (b + 1u < batches) fetch(n, b + 1u);
            else if (next < n_rows) fetch(next, 0u);
#pragma unroll
            for (uint32_t j = 0; j < kMvBatch; ++j) {
                const uint32_t p = (b * kMvBatch + j) * 32u + lane;
                if (p >= groups) break;
                float2 part[NR];
#pragma unroll
                for (uint32_t r = 0; r < NR; ++r) part[r] = make_float2(0.f, 0.f);
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const float4 xa = reinterpret_cast<const float4 *>(sx)[(2u * i) * groups + p];
                    const float4 xb = reinterpret_cast<const float4 *>(sx)[(2u * i + 1u) * groups + p];
#pragma unroll
                    for (uint32_t r = 0; r < NR; ++r) {
                        const uint4 &c = cur[r][j];
                        uint32_t h0, h1, h2, h3;
                        e2m1x8_to_h2x4(i == 0u ? c.x : (i == 1u ? c.y : (i == 2u ? c.z : c.w)), h0, h1, h2, h3);
                        part[r] = __ffma2_rn(h2_to_f2(h0), make_float2(xa.x, xa.y), part[r]);
                        part[r] = __ffma2_rn(h2_to_f2(h1), make_float2(xa.z, xa.w), part[r]);
                        part[r] = __ffma2_rn(h2_to_f2(h2), make_float2(xb.x, xb.y), part[r]);
                        part[r] = __ffma2_rn(h2_to_f2(h3), make_float2(xb.z, xb.w), part[r]);
                    }
                }
#pragma unroll
                for (uint32_t r = 0; r < NR; ++r) acc[r] += (double)(part[r].x + part[r].y) * ue8m0_to_f64(cs[r][j]);
            }
        }
#pragma unroll
        for (uint32_t r = 0; r < NR; ++r) {
            const double v = warp_sum(acc[r]);
            if (lane == 0u && n + r * n_warps < n_rows) y[n + r * n_warps] = (float)v;
        }
        n = next;
    }
}

// The same for rows longer than x fits shared memory: a warp per row, x through the L1.
__global__ void __launch_bounds__(256)
k_mxfp4_matvec_long(const float *__restrict__ x, const uint8_t *__restrict__ w,
                        const uint8_t *__restrict__ s, float *__restrict__ y, uint32_t n_rows,
                        uint32_t k) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t groups = k >> 5;
    for (uint32_t n = warp; n < n_rows; n += n_warps) {
        const uint4 *wrow = reinterpret_cast<const uint4 *>(w + (size_t)n * (k >> 1));
        const uint8_t *srow = s + (size_t)n * groups;
        double acc = 0.0;
        for (uint32_t g = lane; g < groups; g += 32u) {
            const uint4 q = ldg_stream(wrow + g);
            float xr[32];
            const float4 *xp = reinterpret_cast<const float4 *>(x + (size_t)g * 32u);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 v = __ldg(xp + i);
                xr[i * 4 + 0] = v.x;
                xr[i * 4 + 1] = v.y;
                xr[i * 4 + 2] = v.z;
                xr[i * 4 + 3] = v.w;
            }
            acc += (double)dot32_e2m1(q, xr) * ue8m0_to_f64(__ldg(srow + g));
        }
        acc = warp_sum(acc);
        if (lane == 0) y[n] = (float)acc;
    }
}

// Reference order: thread per row, k ascending, (x*e)*s then add.
__global__ void __launch_bounds__(128)
k_mxfp4_matvec_reference(const float *__restrict__ x, const uint8_t *__restrict__ w,
                         const uint8_t *__restrict__ s, float *__restrict__ y, uint32_t n_rows,
                         uint32_t k) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n_rows) return;
    const uint32_t groups = k >> 5;
    const uint4 *wrow = reinterpret_cast<const uint4 *>(w + (size_t)n * (k >> 1));
    const uint8_t *srow = s + (size_t)n * groups;
    float sum = 0.0f;
    for (uint32_t g = 0; g < groups; ++g) {
        const uint4 q = __ldg(wrow + g);
        const float sc = ue8m0_to_f32(__ldg(srow + g));
        const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
        const float *xg = x + (size_t)g * 32u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t h[4];
            e2m1x8_to_h2x4(wd[i], h[0], h[1], h[2], h[3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 e = h2_to_f2(h[j]);
                sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(__ldg(xg + i * 8 + j * 2), e.x), sc));
                sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(__ldg(xg + i * 8 + j * 2 + 1), e.y), sc));
            }
        }
    }
    y[n] = sum;
}

__device__ __forceinline__ float e4m3_to_f32(uint32_t code) {
    const __half_raw hr = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)code, __NV_E4M3);
    return __half2float(__half(hr));
}

template <bool F32_SCALE>
__device__ __forceinline__ double fp8_block_scale_f64(const void *scale, size_t idx) {
    if (F32_SCALE) return (double)ld_f32(reinterpret_cast<const float *>(scale) + idx);
    return ue8m0_to_f64(ld_u8(reinterpret_cast<const uint8_t *>(scale) + idx));
}

template <bool F32_SCALE>
__device__ __forceinline__ float fp8_block_scale_f32(const void *scale, size_t idx) {
    if (F32_SCALE) return __ldg(reinterpret_cast<const float *>(scale) + idx);
    return ue8m0_to_f32(__ldg(reinterpret_cast<const uint8_t *>(scale) + idx));
}

// y[t,n] = sum_k x[t,k] * e4m3(w[n,k]) * scale[n/128][k/128]; warp per row, any k,
// NT tokens per weight pass.  Lanes take 16-byte pieces when the row is 16-byte
// aligned and k is a multiple of 16, single bytes otherwise.
template <int NT, bool F32_SCALE>
__global__ void __launch_bounds__(256)
k_fp8_matvec_pairwise(const float *__restrict__ x, const uint8_t *__restrict__ w,
                      const void *__restrict__ scale, float *__restrict__ y, uint32_t n_rows,
                      uint32_t k) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t k_groups = (k + 127u) >> 7;
    const bool vec_ok = ((k & 15u) == 0u) && ((reinterpret_cast<uintptr_t>(w) & 15u) == 0u) &&
                        ((reinterpret_cast<uintptr_t>(x) & 15u) == 0u);
    for (uint32_t n = warp; n < n_rows; n += n_warps) {
        const uint8_t *wrow = w + (size_t)n * k;
        const size_t srow = (size_t)(n >> 7) * k_groups;
        double acc[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t] = 0.0;
        if (vec_ok) {
            const uint32_t pieces = k >> 4;
            for (uint32_t p = lane; p < pieces; p += 32u) {
                const uint4 q = ldg_stream(reinterpret_cast<const uint4 *>(wrow) + p);
                const double sc = fp8_block_scale_f64<F32_SCALE>(scale, srow + (p >> 3));
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    float xr[16];
                    const float4 *xp =
                        reinterpret_cast<const float4 *>(x + (size_t)t * k + (size_t)p * 16u);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 v = __ldg(xp + i);
                        xr[i * 4 + 0] = v.x;
                        xr[i * 4 + 1] = v.y;
                        xr[i * 4 + 2] = v.z;
                        xr[i * 4 + 3] = v.w;
                    }
                    acc[t] += (double)dot16_e4m3(q, xr) * sc;
                }
            }
        } else {
            for (uint32_t kk = lane; kk < k; kk += 32u) {
                const double wv = (double)e4m3_to_f32(__ldg(wrow + kk)) *
                                  fp8_block_scale_f64<F32_SCALE>(scale, srow + (kk >> 7));
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[t] += (double)__ldg(x + (size_t)t * k + kk) * wv;
            }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const double v = warp_sum(acc[t]);
            if (lane == 0) y[(size_t)t * n_rows + n] = (float)v;
        }
    }
}

// The same product for a block of tokens and a matrix of few rows (the 1024 x 4096 projection of
// the decode step, 1 / 4 / 8 tokens): with a warp per row every warp would fetch the activations of
// all tokens for itself (134 MB of L2 reads for 4 MB of weights at 8 tokens).  Here a CTA of sixteen
// warps takes eight rows, two warps per row (the halves of K), the tokens' activations are staged
// once per CTA in shared memory, a 16-byte piece of weights is decoded once for all tokens, and the
// two halves of a row are added through shared memory.  k a multiple of 32, 16-byte aligned operands.
// A dependent launch: the first weights are brought to the L2 before the wait for the kernel in front, the next ones are
// asked for while a piece is worked on (us a call in a queue of calls, before and after: 1024 x 4096 x 8 tokens 12.3 ->
// 9.8, 4700 x 640 x 8 14.4 -> 11.4, 700 x 8192 x 5 14.4 -> 11.5; one token of 1024 x 4096 7.8 -> 3.1, half of it host time).
// One token, more CTAs than SMs and long rows: a dependent launch's CTAs fill the slots that the launch in front leaves
// and pile up on some SMs (2048 x 8192 one after the other: 9.7 us, an ordinary launch 7.2; 2048 x 4096 4.8 and 3.9;
// short rows gain from it, 4096 x 1024 3.2 and 3.9), and with many CTAs per SM the piece ahead (kAhead) costs more
// registers than it hides (4096 x 8192: 14.4 us, without 12.1).
constexpr uint32_t kFp8BlockRows = 8, kFp8BlockThreads = 512;
template <int NT, bool F32_SCALE, bool kAhead>
__global__ void __launch_bounds__(kFp8BlockThreads)
k_fp8_matvec_block(const float *__restrict__ x, const uint8_t *__restrict__ w, const void *__restrict__ scale,
                   float *__restrict__ y, uint32_t n_rows, uint32_t k) {
    extern __shared__ __align__(16) float sx[];  // [NT][k]
    __shared__ double red[kFp8BlockRows][NT];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t r = warp & (kFp8BlockRows - 1u), half = warp >> 3;
    const uint32_t n = blockIdx.x * kFp8BlockRows + r;
    // staged as [token][quarter of a piece][piece]: the lanes of a warp, which hold consecutive pieces,
    // then read consecutive 16 bytes (no bank conflicts)
    const uint32_t pieces = k >> 4, per = pieces >> 1;
    const uint4 *wrow = reinterpret_cast<const uint4 *>(w + (size_t)n * k);
    uint4 ahead = make_uint4(0u, 0u, 0u, 0u);
    if (n < n_rows && lane < per) l2_hint(wrow + half * per + lane);
    dependency_wait();
    if (kAhead && n < n_rows && lane < per) ahead = ld_stream(wrow + half * per + lane);
    for (uint32_t i = threadIdx.x; i < (NT * k) >> 2; i += kFp8BlockThreads) {
        const uint32_t t = i / (k >> 2), j = i % (k >> 2);
        reinterpret_cast<float4 *>(sx)[(size_t)t * (k >> 2) + (j & 3u) * pieces + (j >> 2)] =
            __ldcg(reinterpret_cast<const float4 *>(x) + i);
    }
    __syncthreads();
    const uint32_t k_groups = (k + 127u) >> 7;
    double acc[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t] = 0.0;
    if (n < n_rows) {
        const size_t srow = (size_t)(n >> 7) * k_groups;
        for (uint32_t p = half * per + lane; p < (half + 1u) * per; p += 32u) {
            const uint4 q = kAhead ? ahead : ld_stream(wrow + p);
            if (kAhead && p + 32u < (half + 1u) * per) ahead = ld_stream(wrow + p + 32u);
            const double sc = fp8_block_scale_f64<F32_SCALE>(scale, srow + (p >> 3));
            const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
            float2 wf[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t h0, h1;
                e4m3x4_to_h2x2(wd[i], h0, h1);
                wf[i * 2] = h2_to_f2(h0);
                wf[i * 2 + 1] = h2_to_f2(h1);
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const float4 *xp = reinterpret_cast<const float4 *>(sx) + (size_t)t * (k >> 2) + p;
                float2 part = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 v = xp[(size_t)i * pieces];
                    part = __ffma2_rn(wf[i * 2], make_float2(v.x, v.y), part);
                    part = __ffma2_rn(wf[i * 2 + 1], make_float2(v.z, v.w), part);
                }
                acc[t] += (double)(part.x + part.y) * sc;
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const double v = warp_sum(acc[t]);
        if (lane == 0 && half == 1u) red[r][t] = v;
        acc[t] = v;
    }
    __syncthreads();
    if (lane == 0 && half == 0u && n < n_rows) {
#pragma unroll
        for (int t = 0; t < NT; ++t) y[(size_t)t * n_rows + n] = (float)(acc[t] + red[r][t]);
    }
}

// Reference order: thread per (row, token), k ascending, (x*e)*s then add
// (examples/s14_vulkan_numeric.rs:1698-1714).
template <bool F32_SCALE>
__global__ void __launch_bounds__(128)
k_fp8_matvec_reference(const float *__restrict__ x, const uint8_t *__restrict__ w,
                       const void *__restrict__ scale, float *__restrict__ y, uint32_t n_rows,
                       uint32_t k, uint32_t n_tokens) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t t = blockIdx.y;
    if (n >= n_rows || t >= n_tokens) return;
    const uint32_t k_groups = (k + 127u) >> 7;
    const uint8_t *wrow = w + (size_t)n * k;
    const float *xt = x + (size_t)t * k;
    const size_t srow = (size_t)(n >> 7) * k_groups;
    float sum = 0.0f;
    for (uint32_t kg = 0; kg < k_groups; ++kg) {
        const float sc = fp8_block_scale_f32<F32_SCALE>(scale, srow + kg);
        const uint32_t k_end = min(kg * 128u + 128u, k);
        for (uint32_t kk = kg * 128u; kk < k_end; ++kk)
            sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(__ldg(xt + kk), e4m3_to_f32(__ldg(wrow + kk))), sc));
    }
    y[(size_t)t * n_rows + n] = sum;
}

// The element-wise operators wait for the kernel in front of them inside the launch (launch_pdl) and read what it
// wrote from the L2.
// s14_swiglu_limit.comp:14-20
__global__ void k_swiglu_limit(const float *__restrict__ gate, const float *__restrict__ up,
                               float *__restrict__ y, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    dependency_wait();
    if (i < n) y[i] = swiglu_limit_f32(__ldcg(gate + i), __ldcg(up + i));
}

// s14_route_mix.comp:16-20
__global__ void k_route_mix(const float *__restrict__ expert, float *__restrict__ routed, uint32_t n,
                            float weight) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    dependency_wait();
    if (i < n) routed[i] = __fmul_rn(weight, __ldcg(expert + i));
}

// s14_moe_accumulate.comp:17-21
__global__ void k_moe_accumulate(const float *__restrict__ expert, float *__restrict__ acc,
                                 uint32_t n, float weight) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    dependency_wait();
    if (i < n) acc[i] = __fadd_rn(__ldcg(acc + i), __fmul_rn(weight, __ldcg(expert + i)));
}

// ------------------------------------------------------- fused MoE layer ----
//
// A job is one (expert page, token) pair.  Jobs of the same expert are adjacent
// so that the second and later tokens of an expert find its page in L2.
//   up   : h[job, i]    = swiglu(w1[i,:] . x_t, w3[i,:] . x_t)      i < inter
//   down : d[job, n]    = w2[n,:] . h[job,:]                        n < hidden
//   mix  : y[t, n]      = sum over the token's jobs, in route order, of
//                         weight * d[job, n]  (shared last, weight 1)

// One MXFP4 row against register-resident activations.  KC = K / 1024; lane l
// owns the 32 elements k = j*1024 + l*32 ... of every 1024-wide slice j, which is
// one 16-byte piece and one scale block.
template <int KC>
struct RowFrag {
    uint4 q[KC];
    uint32_t sc[KC];
};

// MAT: 0 = w1, 1 = w3 (rows of [inter, hidden]), 2 = w2 (rows of [hidden, inter]); `other` is the
// matrix's other dimension (inter for w1 / w3 rows of K = hidden, hidden for w2 rows of K = inter).
template <int KC, int MAT>
__device__ __forceinline__ void load_row_mxfp4(RowFrag<KC> &f, const PageView &pv, uint32_t row, uint32_t lane,
                                               uint32_t other) {
#pragma unroll
    for (int j = 0; j < KC; ++j) {
        const uint32_t kb = (uint32_t)j * 32u + lane;
        if (MAT < 2) {
            constexpr uint32_t hidden = KC * 1024;
            f.q[j] = ldg_stream(reinterpret_cast<const uint4 *>(pv.base + mxfp4_up_chunk_offset(MAT, row, kb, hidden)));
            f.sc[j] = __ldg(pv.base + mxfp4_up_scale_offset(MAT, row, kb, hidden, other));
        } else {
            constexpr uint32_t inter = KC * 1024;
            f.q[j] = ldg_stream(reinterpret_cast<const uint4 *>(pv.base + mxfp4_down_chunk_offset(row, kb, other, inter)));
            f.sc[j] = __ldg(pv.base + mxfp4_down_scale_offset(row, kb, other, inter));
        }
    }
}

template <int KC>
__device__ __forceinline__ double dot_row_mxfp4(const RowFrag<KC> &f, const float *__restrict__ xr) {
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < KC; ++j)
        acc += (double)dot32_e2m1(f.q[j], xr + j * 32) * ue8m0_to_f64(f.sc[j]);
    return acc;
}

// One FP8 row with the same lane-to-k mapping (two 16-byte pieces per slice).
template <int KC>
__device__ __forceinline__ double dot_row_fp8(const uint8_t *w, const uint8_t *s, uint32_t row,
                                              uint32_t lane, const float *__restrict__ xr) {
    const uint8_t *wrow = w + (size_t)row * (KC * 1024);
    const uint8_t *srow = s + (size_t)(row >> 7) * (KC * 8);
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < KC; ++j) {
        const uint4 *p = reinterpret_cast<const uint4 *>(wrow + j * 1024 + lane * 32);
        const uint4 q0 = __ldg(p), q1 = __ldg(p + 1);
        const float part = dot16_e4m3(q0, xr + j * 32) + dot16_e4m3(q1, xr + j * 32 + 16);
        acc += (double)part * ue8m0_to_f64(__ldg(srow + j * 8 + (lane >> 2)));
    }
    return acc;
}

template <int KC>
__device__ __forceinline__ void load_x_regs(float *xr, const float *__restrict__ x, uint32_t lane) {
#pragma unroll
    for (int j = 0; j < KC; ++j) {
        const float4 *xp = reinterpret_cast<const float4 *>(x + j * 1024 + lane * 32);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 v = xp[i];
            xr[j * 32 + i * 4 + 0] = v.x;
            xr[j * 32 + i * 4 + 1] = v.y;
            xr[j * 32 + i * 4 + 2] = v.z;
            xr[j * 32 + i * 4 + 3] = v.w;
        }
    }
}

// Up phase, pairwise order.  grid = n_tokens * ctas_per_token; the warps of a CTA
// keep their token's x in registers and stride over that token's (job, row) space.
template <int KC>
__global__ void __launch_bounds__(256, 1)
k_expert_up_pairwise(const JobTable *__restrict__ dev_table,
                     const __grid_constant__ JobTable param_table, const float *__restrict__ x,
                     float *__restrict__ h, uint32_t inter, uint32_t ctas_per_token) {
    const JobTable &tab = table_of(dev_table, param_table);
    constexpr uint32_t hidden = KC * 1024;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t token = blockIdx.x / ctas_per_token;
    const uint32_t cta_in_token = blockIdx.x - token * ctas_per_token;
    const uint32_t warp = cta_in_token * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t n_warps = ctas_per_token * (blockDim.x >> 5);
    const uint32_t job0 = tab.token_job_begin[token];
    const uint32_t n_jobs = tab.token_job_begin[token + 1] - job0;
    const uint32_t items = n_jobs * inter;

    float xr[KC * 32];
    load_x_regs<KC>(xr, x + (size_t)token * hidden, lane);

    RowFrag<KC> g0, u0, g1, u1;
    uint32_t it = warp;
    auto issue = [&](RowFrag<KC> &g, RowFrag<KC> &u, uint32_t item) {
        const uint32_t job = job0 + item / inter, row = item % inter;
        const Job jb = tab.jobs[tab.token_jobs[job]];
        if (jb.kind == S14_PAGE_MXFP4) {
            const PageView pv = page_view(jb.page, jb.kind, hidden, inter);
            load_row_mxfp4<KC, 0>(g, pv, row, lane, inter);
            load_row_mxfp4<KC, 1>(u, pv, row, lane, inter);
        }
    };
    auto finish = [&](const RowFrag<KC> &g, const RowFrag<KC> &u, uint32_t item) {
        const uint32_t job = job0 + item / inter, row = item % inter;
        const uint32_t jid = tab.token_jobs[job];
        const Job jb = tab.jobs[jid];
        double gate, up;
        if (jb.kind == S14_PAGE_MXFP4) {
            gate = dot_row_mxfp4<KC>(g, xr);
            up = dot_row_mxfp4<KC>(u, xr);
        } else {
            const PageView pv = page_view(jb.page, jb.kind, hidden, inter);
            gate = dot_row_fp8<KC>(pv.w1, pv.s1, row, lane, xr);
            up = dot_row_fp8<KC>(pv.w3, pv.s3, row, lane, xr);
        }
        gate = warp_sum(gate);
        up = warp_sum(up);
        if (lane == 0) h[(size_t)jid * inter + row] = swiglu_limit_f32((float)gate, (float)up);
    };
    if (it < items) issue(g0, u0, it);
    while (it < items) {
        const uint32_t nx = it + n_warps;
        if (nx < items) issue(g1, u1, nx);
        finish(g0, u0, it);
        it = nx;
        if (it >= items) break;
        const uint32_t nx2 = it + n_warps;
        if (nx2 < items) issue(g0, u0, nx2);
        finish(g1, u1, it);
        it = nx2;
    }
}

// Down phase, pairwise order.  grid = n_jobs * ctas_per_job; a CTA's warps keep the
// job's h in registers and stride over the rows of w2.
template <int KC>
__global__ void __launch_bounds__(256, (KC >= 4 ? 1 : 2))
k_expert_down_pairwise(const JobTable *__restrict__ dev_table,
                       const __grid_constant__ JobTable param_table, const float *__restrict__ h,
                       float *__restrict__ d, uint32_t hidden, uint32_t ctas_per_job) {
    const JobTable &tab = table_of(dev_table, param_table);
    constexpr uint32_t inter = KC * 1024;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t jid = blockIdx.x / ctas_per_job;
    const uint32_t cta_in_job = blockIdx.x - jid * ctas_per_job;
    const uint32_t warp = cta_in_job * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t n_warps = ctas_per_job * (blockDim.x >> 5);
    if (jid >= tab.n_jobs) return;
    const Job jb = tab.jobs[jid];
    const PageView pv = page_view(jb.page, jb.kind, hidden, inter);

    float xr[KC * 32];
    load_x_regs<KC>(xr, h + (size_t)jid * inter, lane);
    float *out = d + (size_t)jb.out_index * hidden;

    if (jb.kind != S14_PAGE_MXFP4) {
        for (uint32_t row = warp; row < hidden; row += n_warps) {
            const double v = warp_sum(dot_row_fp8<KC>(pv.w2, pv.s2, row, lane, xr));
            if (lane == 0) out[row] = (float)v;
        }
        return;
    }
    RowFrag<KC> a0, a1, b0, b1;
    uint32_t row = warp;
    const uint32_t step = n_warps;
    // two rows per stage, two stages in flight
    auto issue2 = [&](RowFrag<KC> &p, RowFrag<KC> &q, uint32_t r) {
        if (r < hidden) load_row_mxfp4<KC, 2>(p, pv, r, lane, hidden);
        if (r + step < hidden) load_row_mxfp4<KC, 2>(q, pv, r + step, lane, hidden);
    };
    auto finish2 = [&](const RowFrag<KC> &p, const RowFrag<KC> &q, uint32_t r) {
        if (r < hidden) {
            const double v = warp_sum(dot_row_mxfp4<KC>(p, xr));
            if (lane == 0) out[r] = (float)v;
        }
        if (r + step < hidden) {
            const double v = warp_sum(dot_row_mxfp4<KC>(q, xr));
            if (lane == 0) out[r + step] = (float)v;
        }
    };
    if (row < hidden) issue2(a0, a1, row);
    while (row < hidden) {
        const uint32_t nx = row + 2 * step;
        if (nx < hidden) issue2(b0, b1, nx);
        finish2(a0, a1, row);
        row = nx;
        if (row >= hidden) break;
        const uint32_t nx2 = row + 2 * step;
        if (nx2 < hidden) issue2(a0, a1, nx2);
        finish2(b0, b1, row);
        row = nx2;
    }
}

// Reference-order dot of one MXFP4 row: sequential k, (x*e)*s, separate add.
// x is read from shared memory (every lane reads the same address: broadcast).
// MAT: 0 = w1, 1 = w3, 2 = w2 of an expert page; k is the row's length.
template <int MAT>
__device__ __forceinline__ float dot_row_mxfp4_reference(const PageView &pv, uint32_t row, uint32_t k, uint32_t hidden,
                                                         uint32_t inter, const float *__restrict__ xs) {
    const uint32_t groups = k >> 5;
    float sum = 0.0f;
    for (uint32_t g4 = 0; g4 < groups; g4 += 4) {
        uint4 q[4];
        uint32_t scw;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            q[j] = __ldg(reinterpret_cast<const uint4 *>(
                pv.base + (MAT < 2 ? mxfp4_up_chunk_offset(MAT, row, g4 + j, hidden)
                                   : mxfp4_down_chunk_offset(row, g4 + j, hidden, inter))));
        scw = __ldg(reinterpret_cast<const uint32_t *>(
            pv.base + (MAT < 2 ? mxfp4_up_scale_offset(MAT, row, g4, hidden, inter)
                               : mxfp4_down_scale_offset(row, g4, hidden, inter))));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float sc = ue8m0_to_f32((scw >> (8 * j)) & 0xffu);
            const uint32_t wd[4] = {q[j].x, q[j].y, q[j].z, q[j].w};
            const float *xg = xs + (size_t)(g4 + j) * 32u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t hh[4];
                e2m1x8_to_h2x4(wd[i], hh[0], hh[1], hh[2], hh[3]);
                const float4 xa = *reinterpret_cast<const float4 *>(xg + i * 8);
                const float4 xb = *reinterpret_cast<const float4 *>(xg + i * 8 + 4);
                const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float2 e = h2_to_f2(hh[p]);
                    sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(xv[p * 2], e.x), sc));
                    sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(xv[p * 2 + 1], e.y), sc));
                }
            }
        }
    }
    return sum;
}

__device__ __forceinline__ float dot_row_fp8_reference(const uint8_t *w, const uint8_t *s,
                                                       uint32_t row, uint32_t k,
                                                       const float *__restrict__ xs) {
    const uint32_t k_groups = (k + 127u) >> 7;
    const uint4 *wrow = reinterpret_cast<const uint4 *>(w + (size_t)row * k);
    const uint8_t *srow = s + (size_t)(row >> 7) * k_groups;
    float sum = 0.0f;
    for (uint32_t kg = 0; kg < k_groups; ++kg) {
        const float sc = ue8m0_to_f32(__ldg(srow + kg));
        for (uint32_t p = 0; p < 8; ++p) {
            const uint4 q = __ldg(wrow + kg * 8 + p);
            const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
            const float *xg = xs + kg * 128u + p * 16u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t h0, h1;
                e4m3x4_to_h2x2(wd[i], h0, h1);
                const float4 xa = *reinterpret_cast<const float4 *>(xg + i * 4);
                const float2 e0 = h2_to_f2(h0), e1 = h2_to_f2(h1);
                sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(xa.x, e0.x), sc));
                sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(xa.y, e0.y), sc));
                sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(xa.z, e1.x), sc));
                sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(xa.w, e1.y), sc));
            }
        }
    }
    return sum;
}

// Up phase, reference order: a thread owns gate row i and up row i of one job.
// grid = (ceil(inter/32), n_jobs), block = 32.
__global__ void __launch_bounds__(32)
k_expert_up_reference(const JobTable *__restrict__ dev_table,
                      const __grid_constant__ JobTable param_table, const float *__restrict__ x,
                      float *__restrict__ h, uint32_t hidden, uint32_t inter) {
    extern __shared__ __align__(16) float xs[];
    const JobTable &tab = table_of(dev_table, param_table);
    const uint32_t jid = blockIdx.y;
    if (jid >= tab.n_jobs) return;
    const Job jb = tab.jobs[jid];
    const float *xt = x + (size_t)jb.token * hidden;
    for (uint32_t i = threadIdx.x; i < hidden; i += blockDim.x) xs[i] = xt[i];
    __syncthreads();
    const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= inter) return;
    const PageView pv = page_view(jb.page, jb.kind, hidden, inter);
    float gate, up;
    if (jb.kind == S14_PAGE_MXFP4) {
        gate = dot_row_mxfp4_reference<0>(pv, row, hidden, hidden, inter, xs);
        up = dot_row_mxfp4_reference<1>(pv, row, hidden, hidden, inter, xs);
    } else {
        gate = dot_row_fp8_reference(pv.w1, pv.s1, row, hidden, xs);
        up = dot_row_fp8_reference(pv.w3, pv.s3, row, hidden, xs);
    }
    h[(size_t)jid * inter + row] = swiglu_limit_f32(gate, up);
}

// Down phase, reference order.  grid = (ceil(hidden/32), n_jobs), block = 32.
__global__ void __launch_bounds__(32)
k_expert_down_reference(const JobTable *__restrict__ dev_table,
                        const __grid_constant__ JobTable param_table, const float *__restrict__ h,
                        float *__restrict__ d, uint32_t hidden, uint32_t inter) {
    extern __shared__ __align__(16) float xs[];
    const JobTable &tab = table_of(dev_table, param_table);
    const uint32_t jid = blockIdx.y;
    if (jid >= tab.n_jobs) return;
    const Job jb = tab.jobs[jid];
    const float *hj = h + (size_t)jid * inter;
    for (uint32_t i = threadIdx.x; i < inter; i += blockDim.x) xs[i] = hj[i];
    __syncthreads();
    const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= hidden) return;
    const PageView pv = page_view(jb.page, jb.kind, hidden, inter);
    const float v = (jb.kind == S14_PAGE_MXFP4)
                        ? dot_row_mxfp4_reference<2>(pv, row, inter, hidden, inter, xs)
                        : dot_row_fp8_reference(pv.w2, pv.s2, row, inter, xs);
    d[(size_t)jb.out_index * hidden + row] = v;
}

// Ordered mix (examples/s14_vulkan_numeric.rs:936-946): acc = 0; acc += w * d for the
// token's routed jobs in route order; acc += d_shared.  Separate multiply and add.
__global__ void __launch_bounds__(256)
k_moe_mix(const JobTable *__restrict__ dev_table, const __grid_constant__ JobTable param_table,
          const float *__restrict__ d, float *__restrict__ y, uint32_t hidden) {
    const JobTable &tab = table_of(dev_table, param_table);
    const uint32_t token = blockIdx.y;
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= hidden) return;
    const uint32_t j0 = tab.token_job_begin[token], j1 = tab.token_job_begin[token + 1];
    float acc = 0.0f;
    for (uint32_t j = j0; j < j1; ++j) {
        const uint32_t jid = tab.token_jobs[j];
        const Job jb = tab.jobs[jid];
        const float v = d[(size_t)jb.out_index * hidden + n];
        acc = jb.is_shared ? __fadd_rn(acc, v) : __fadd_rn(acc, __fmul_rn(jb.weight, v));
    }
    y[(size_t)token * hidden + n] = acc;
}

// Ordered mix of gathered per-slot expert outputs (expert-parallel combine): slots [n_routed (+1)]
// [hidden], weights on the device; same operations and order as k_moe_mix.
__global__ void __launch_bounds__(256)
k_mix_slots(const float *__restrict__ slots, const float *__restrict__ weights, uint32_t n_routed,
            int has_shared, float *__restrict__ y, uint32_t hidden) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= hidden) return;
    float acc = 0.0f;
    for (uint32_t j = 0; j < n_routed; ++j)
        acc = __fadd_rn(acc, __fmul_rn(weights[j], slots[(size_t)j * hidden + n]));
    if (has_shared) acc = __fadd_rn(acc, slots[(size_t)n_routed * hidden + n]);
    y[n] = acc;
}

// ------------------------------------------------------------- router -------

// One CTA of two warps per (token, expert) row of BF16 weights: logit in double (every product
// f32 x bf16 is exact in double), score and score + bias in F32.  The last CTA to finish
// (a counter in global memory, no waiting) selects the top-k of every token, normalises the
// weights and, for the one-token decode path, writes the job table of the layer.
__global__ void __launch_bounds__(64)
k_router(const float *__restrict__ x, const uint16_t *__restrict__ wr, const float *__restrict__ bias,
         float *__restrict__ scores, float *__restrict__ select, uint32_t n_experts, uint32_t hidden,
         uint32_t n_tokens, uint32_t score_fn, uint32_t top_k, float route_scale,
         int32_t *__restrict__ ids_out, float *__restrict__ weights_out, JobTable *__restrict__ table_out,
         const uint8_t *const *__restrict__ page_table, const uint8_t *shared_page, uint32_t shared_kind,
         unsigned int *__restrict__ counter, uint32_t ep_rank, uint32_t ep_world, uint32_t shared_owner) {
    __shared__ bool is_last;
    // a dependent launch (the up phase) may start its own prologue now; it reads what this
    // kernel writes only after cudaGridDependencySynchronize()
    cudaTriggerProgrammaticLaunchCompletion();
    __shared__ double half_sum[2];
    const uint32_t lane = threadIdx.x & 31u, half = threadIdx.x >> 5;
    {
        const uint32_t t = blockIdx.x / n_experts, e = blockIdx.x - t * n_experts;
        const uint32_t pieces = hidden >> 4;  // 16-byte pieces (8 weights) per half row
        const uint4 *row = reinterpret_cast<const uint4 *>(wr + (size_t)e * hidden) + half * pieces;
        const float *xt = x + (size_t)t * hidden + (size_t)half * (hidden >> 1);
        double acc0 = 0.0, acc1 = 0.0;
        for (uint32_t p0 = lane; p0 < pieces; p0 += 32u * 8u) {
            uint4 q[8];
            float4 xa[8], xb[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t p = p0 + u * 32u;
                if (p < pieces) {
                    q[u] = __ldg(row + p);
                    xa[u] = __ldg(reinterpret_cast<const float4 *>(xt + p * 8));
                    xb[u] = __ldg(reinterpret_cast<const float4 *>(xt + p * 8 + 4));
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (p0 + u * 32u < pieces) {
                    const uint32_t wd[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
                    const float xv[8] = {xa[u].x, xa[u].y, xa[u].z, xa[u].w, xb[u].x, xb[u].y, xb[u].z, xb[u].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        acc0 += (double)xv[i * 2] * (double)__uint_as_float(wd[i] << 16);
                        acc1 += (double)xv[i * 2 + 1] * (double)__uint_as_float(wd[i] & 0xffff0000u);
                    }
                }
            }
        }
        const double part = warp_sum(acc0 + acc1);
        if (lane == 0) half_sum[half] = part;
        __syncthreads();
        if (threadIdx.x == 0) {
            const float s = router_score_f32(half_sum[0] + half_sum[1], score_fn);
            scores[(size_t)t * n_experts + e] = s;
            select[(size_t)t * n_experts + e] = __fadd_rn(s, bias ? bias[e] : 0.0f);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(counter, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (uint32_t t = threadIdx.x >> 5; t < n_tokens; t += blockDim.x >> 5)
        router_select(scores + (size_t)t * n_experts, select + (size_t)t * n_experts, n_experts, top_k,
                      route_scale, ids_out ? ids_out + (size_t)t * top_k : nullptr,
                      weights_out ? weights_out + (size_t)t * top_k : nullptr, table_out, page_table,
                      shared_page, shared_kind, lane, ep_rank, ep_world, shared_owner);
    if (threadIdx.x == 0) *counter = 0u;  // ready for the next launch
}

// ------------------------------------------------------------- launchers ----

static inline uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// Shared memory for the longest x the row kernels hold, once per device.
static cudaError_t matvec_smem_attribute() {
    static bool done[64] = {};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return e != cudaSuccess ? e : cudaErrorInvalidDevice;
    if (done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(k_mxfp4_matvec_pairwise<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kMvMaxK * sizeof(float)));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mxfp4_matvec_pairwise<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kMvMaxK * sizeof(float)));
    done[dev] = e == cudaSuccess;
    return e;
}

cudaError_t launch_mxfp4_matvec(cudaStream_t st, uint32_t mode, int sm_count, const float *x,
                                const uint8_t *w, const uint8_t *s, float *y, uint32_t n, uint32_t k) {
    if (mode == S14_ACCUM_REFERENCE) {
        k_mxfp4_matvec_reference<<<ceil_div(n, 128), 128, 0, st>>>(x, w, s, y, n, k);
    } else {
        if (k > kMvMaxK) {
            k_mxfp4_matvec_long<<<min(ceil_div(n, 8), (uint32_t)sm_count * 8u), 256, 0, st>>>(x, w, s, y, n, k);
            return cudaGetLastError();
        }
        // one CTA of sixteen warps per SM; two rows per warp when every warp has two
        const cudaError_t e = matvec_smem_attribute();
        if (e != cudaSuccess) return e;
        const size_t smem = (size_t)k * sizeof(float);
        const dim3 grid(min(n, (uint32_t)sm_count)), block(kMvThreads);
        if (n >= 2u * (kMvThreads / 32u) * (uint32_t)sm_count)
            return launch_pdl(k_mxfp4_matvec_pairwise<2>, grid, block, smem, st, 0u, x, w, s, y, n, k);
        return launch_pdl(k_mxfp4_matvec_pairwise<1>, grid, block, smem, st, 0u, x, w, s, y, n, k);
    }
    return cudaGetLastError();
}

// Largest dynamic shared memory k_fp8_matvec_block may ask for on the current device (0: not set).
template <int NT, bool F32S, bool kAhead>
static bool fp8_block_smem_ok(size_t bytes) {
    static int configured[64] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!configured[dev]) {
        configured[dev] = cudaFuncSetAttribute(k_fp8_matvec_block<NT, F32S, kAhead>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               160 * 1024) == cudaSuccess ? 1 : -1;
    }
    return configured[dev] == 1 && bytes <= 160u * 1024u;
}

// Whether the block kernel takes the call; *err: its launch's result.
template <int NT, bool F32S>
static bool try_fp8_block(cudaStream_t st, int sm_count, const float *x, const uint8_t *w, const void *s, float *y,
                          uint32_t n, uint32_t k, cudaError_t *err) {
    // few rows (a warp per row would leave most SMs with a handful of warps), k in whole scale
    // blocks, 16-byte aligned operands, the tokens' activations fit shared memory
    const size_t bytes = (size_t)NT * k * sizeof(float);
    if (n > (uint32_t)sm_count * 32u || (k & 31u) || ((uintptr_t)w & 15u) || ((uintptr_t)x & 15u)) return false;
    const dim3 grid((n + kFp8BlockRows - 1) / kFp8BlockRows), block(kFp8BlockThreads);
    if constexpr (NT == 1) {
        if (grid.x > (uint32_t)sm_count && k >= 4096u) {
            const bool ahead = grid.x <= 2u * (uint32_t)sm_count;
            if (!(ahead ? fp8_block_smem_ok<NT, F32S, true>(bytes) : fp8_block_smem_ok<NT, F32S, false>(bytes))) return false;
            if (ahead) k_fp8_matvec_block<NT, F32S, true><<<grid, block, bytes, st>>>(x, w, s, y, n, k);
            else k_fp8_matvec_block<NT, F32S, false><<<grid, block, bytes, st>>>(x, w, s, y, n, k);
            *err = cudaGetLastError();
            return true;
        }
    }
    if (!fp8_block_smem_ok<NT, F32S, true>(bytes)) return false;
    *err = launch_pdl(k_fp8_matvec_block<NT, F32S, true>, grid, block, bytes, st, 0u, x, w, s, y, n, k);
    return true;
}

template <bool F32S>
static cudaError_t launch_fp8_pairwise_nt(cudaStream_t st, int sm_count, uint32_t blocks, uint32_t nt, const float *x,
                                          const uint8_t *w, const void *s, float *y, uint32_t n, uint32_t k) {
    bool done = false;
    cudaError_t err = cudaSuccess;
    switch (nt) {
    case 1: done = try_fp8_block<1, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    case 2: done = try_fp8_block<2, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    case 3: done = try_fp8_block<3, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    case 4: done = try_fp8_block<4, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    case 5: done = try_fp8_block<5, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    case 6: done = try_fp8_block<6, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    case 7: done = try_fp8_block<7, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    default: done = try_fp8_block<8, F32S>(st, sm_count, x, w, s, y, n, k, &err); break;
    }
    if (done) return err;
    switch (nt) {
    case 1: k_fp8_matvec_pairwise<1, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    case 2: k_fp8_matvec_pairwise<2, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    case 3: k_fp8_matvec_pairwise<3, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    case 4: k_fp8_matvec_pairwise<4, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    case 5: k_fp8_matvec_pairwise<5, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    case 6: k_fp8_matvec_pairwise<6, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    case 7: k_fp8_matvec_pairwise<7, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    default: k_fp8_matvec_pairwise<8, F32S><<<blocks, 256, 0, st>>>(x, w, s, y, n, k); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_fp8_matvec(cudaStream_t st, uint32_t mode, int sm_count, uint32_t scale_format,
                              uint32_t n_tokens, const float *x, const uint8_t *w, const void *s,
                              float *y, uint32_t n, uint32_t k) {
    if (mode == S14_ACCUM_REFERENCE) {
        dim3 grid(ceil_div(n, 128), n_tokens);
        if (scale_format == S14_SCALE_F32)
            k_fp8_matvec_reference<true><<<grid, 128, 0, st>>>(x, w, s, y, n, k, n_tokens);
        else
            k_fp8_matvec_reference<false><<<grid, 128, 0, st>>>(x, w, s, y, n, k, n_tokens);
    } else {
        const uint32_t blocks = min(ceil_div(n, 8), (uint32_t)sm_count * 8u);
        if (scale_format == S14_SCALE_F32)
            return launch_fp8_pairwise_nt<true>(st, sm_count, blocks, n_tokens, x, w, s, y, n, k);
        return launch_fp8_pairwise_nt<false>(st, sm_count, blocks, n_tokens, x, w, s, y, n, k);
    }
    return cudaGetLastError();
}

cudaError_t launch_swiglu_limit(cudaStream_t st, const float *gate, const float *up, float *y,
                                uint32_t n) {
    return launch_pdl(k_swiglu_limit, dim3(ceil_div(n, 256)), dim3(256), 0, st, 0u, gate, up, y, n);
}

cudaError_t launch_route_mix(cudaStream_t st, const float *expert, float *routed, uint32_t n,
                             float weight) {
    return launch_pdl(k_route_mix, dim3(ceil_div(n, 256)), dim3(256), 0, st, 0u, expert, routed, n, weight);
}

cudaError_t launch_moe_accumulate(cudaStream_t st, const float *expert, float *acc, uint32_t n,
                                  float weight) {
    return launch_pdl(k_moe_accumulate, dim3(ceil_div(n, 256)), dim3(256), 0, st, 0u, expert, acc, n, weight);
}

template <int KC>
static void launch_up_pairwise(cudaStream_t st, const JobTable *dev, const JobTable &param,
                               const float *x, float *h, uint32_t inter, uint32_t n_tokens,
                               uint32_t ctas_per_token) {
    k_expert_up_pairwise<KC><<<n_tokens * ctas_per_token, 256, 0, st>>>(dev, param, x, h, inter,
                                                                        ctas_per_token);
}

template <int KC>
static void launch_down_pairwise(cudaStream_t st, const JobTable *dev, const JobTable &param,
                                 const float *h, float *d, uint32_t hidden, uint32_t n_jobs,
                                 uint32_t ctas_per_job) {
    k_expert_down_pairwise<KC><<<n_jobs * ctas_per_job, 256, 0, st>>>(dev, param, h, d, hidden,
                                                                      ctas_per_job);
}

// which implementation the calling thread's last launch_moe_layer chose (S14_LAYER_PATH_*)
static thread_local uint32_t t_last_layer_path = 0;
uint32_t last_layer_path() { return t_last_layer_path; }

int launch_moe_layer(cudaStream_t st, uint32_t mode, int sm_count, const JobTable *dev_table,
                     const JobTable &param_table, uint32_t n_tokens, uint32_t n_jobs_max,
                     uint32_t hidden, uint32_t inter, const float *x, float *h, float *d, float *y,
                     cudaError_t *err, const KernelMarks *km, bool all_mxfp4, unsigned int *counters,
                     const UmmaScratch *umma, const FusedRouter *router, const EpExchange *ep, const uint16_t *x_bf16,
                     float *x_stage, BranchPost *post) {
    int launches = 0;
    *err = cudaSuccess;
    t_last_layer_path = 0;
    // the checkpoint's page kinds: routed MXFP4 experts and an FP8 shared expert
    const uint8_t *shared = nullptr;
    if (n_tokens == 1u && y && !ep && counters) {
        if (router && router->ep_world <= 1u && router->shared_kind == S14_PAGE_FP8) shared = router->shared_page;
        if (!router && !dev_table)
            for (uint32_t j = 0; j < param_table.n_jobs; ++j)
                if (param_table.jobs[j].is_shared && param_table.jobs[j].kind == S14_PAGE_FP8) shared = param_table.jobs[j].page;
    }
    if (shared) {
        JobTable routed = {};
        uint32_t n_routed = 0;
        FusedRouter rt = {};
        if (router) {
            rt = *router;
            rt.shared_page = nullptr;
            n_routed = umma_router_ok(sm_count, rt.n_experts) ? rt.top_k : 0u;
        } else {
            routed.n_tokens = 1;
            for (uint32_t i = param_table.token_job_begin[0]; i < param_table.token_job_begin[1]; ++i) {
                Job jb = param_table.jobs[param_table.token_jobs[i]];
                if (jb.is_shared) continue;
                jb.out_index = n_routed;
                routed.jobs[n_routed] = jb;
                routed.token_jobs[n_routed] = (uint8_t)n_routed;
                ++n_routed;
            }
            routed.n_jobs = routed.token_job_begin[1] = n_routed;
        }
        if (fp8_shared_layer_ok(sm_count, mode, umma, n_routed, hidden, inter)) {
            // the expert's kernel reads a BF16 token in 8-byte pieces; a token on another boundary is converted first
            if (!fp8_expert_takes(x_bf16)) {
                *err = launch_bf16_to_f32(st, x_bf16, x_stage, hidden);
                if (*err != cudaSuccess) return launches;
                ++launches;
                x_bf16 = nullptr;
            }
            if (km) cudaEventRecord(km->ev[0], st), cudaEventRecord(km->ev[1], st);
            launches += launch_layer_fp8_shared(st, sm_count, routed, router ? &rt : nullptr, shared, x, x_bf16, h, d, y,
                                                counters, umma, hidden, inter, err, post);
            if (km)  // as for the layer kernel alone (below): all of it is booked as the up phase
                for (int i = 2; i < 5; ++i) cudaEventRecord(km->ev[i], st);
            t_last_layer_path = S14_LAYER_PATH_TENSOR | S14_LAYER_PATH_FP8_SHARED_KERNEL;
            return launches;
        }
    }
    if (x_bf16) {
        *err = launch_bf16_to_f32(st, x_bf16, x_stage, hidden * n_tokens);
        if (*err != cudaSuccess) return launches;
        ++launches;
    }
    const bool tensor_path = mode != S14_ACCUM_REFERENCE && all_mxfp4 && counters && umma &&
                             umma_layer_ok(sm_count, n_tokens, n_jobs_max, hidden, inter);
    if (ep && ep->world > 1u && !(tensor_path && router && umma_router_ok(sm_count, router->n_experts))) {
        *err = cudaErrorNotSupported;  // the exchange over peer memory is part of the tensor-core layer kernel
        return launches;
    }
    if (router && !(tensor_path && umma_router_ok(sm_count, router->n_experts))) {
        // the routes come from a kernel of their own, which fills the device job table
        s14_router_desc r = {};
        r.x = x;
        r.router_weight_bf16 = router->weight;
        r.bias = router->bias;
        r.n_experts = router->n_experts;
        r.hidden = hidden;
        r.n_tokens = 1;
        r.score_fn = router->score_fn;
        r.top_k = router->top_k;
        r.route_scale = router->route_scale;
        r.ids_out = router->ids_out;
        r.weights_out = router->weights_out;
        launches += launch_router(st, r, router->scores, router->select, router->table_out, router->page_table,
                                  router->shared_page, router->shared_kind, counters, err, km, router->ep_rank,
                                  router->ep_world, router->shared_owner);
        if (*err != cudaSuccess) return launches;
        dev_table = router->table_out;
        router = nullptr;
        t_last_layer_path |= S14_LAYER_PATH_ROUTER_KERNEL;
    } else if (router && km) {
        cudaEventRecord(km->ev[0], st);
    }
    if (km) cudaEventRecord(km->ev[1], st);
    // A block of several tokens whose routes the caller gives (a verify block of up to eight tokens):
    // the tensor-core kernel takes one token per launch, so the block is one launch per token, each
    // with the token's own jobs in its mix order.  Launches follow one another in the stream (each a
    // programmatic dependent of the one before), a page that several tokens of the block use (the
    // shared expert always) is read from HBM by the first and found in the L2 by the others, and every
    // token's result is, bit for bit, that of its own one-token call.
    const bool block_on_tensor_path = mode != S14_ACCUM_REFERENCE && all_mxfp4 && counters && umma && n_tokens > 1u &&
                                      !router && !ep && !dev_table && y &&
                                      umma_layer_ok(sm_count, 1u, S14_EXPERTS_PER_TOKEN + 1u, hidden, inter);
    if (block_on_tensor_path) {
        bool fits = true;
        for (uint32_t t = 0; t < n_tokens; ++t)
            fits = fits && param_table.token_job_begin[t + 1] - param_table.token_job_begin[t] <= S14_EXPERTS_PER_TOKEN + 1u &&
                   param_table.token_job_begin[t + 1] > param_table.token_job_begin[t];
        if (fits) {
            for (uint32_t t = 0; t < n_tokens && *err == cudaSuccess; ++t) {
                JobTable one = {};
                const uint32_t b = param_table.token_job_begin[t], e = param_table.token_job_begin[t + 1];
                one.n_jobs = e - b;
                one.n_tokens = 1;
                one.token_job_begin[0] = 0;
                one.token_job_begin[1] = e - b;
                for (uint32_t i = b; i < e; ++i) {
                    Job jb = param_table.jobs[param_table.token_jobs[i]];
                    jb.token = 0;
                    jb.out_index = i - b;
                    one.jobs[i - b] = jb;
                    one.token_jobs[i - b] = (uint8_t)(i - b);
                }
                *err = launch_moe_layer_umma(st, sm_count, nullptr, one, x + (size_t)t * hidden, d, y + (size_t)t * hidden,
                                             umma->tiles, counters, umma->status, hidden, inter, nullptr, nullptr,
                                             umma->trace);
                launches += 1;
            }
            if (km) {
                cudaEventRecord(km->ev[2], st);
                cudaEventRecord(km->ev[3], st);
                cudaEventRecord(km->ev[4], st);
            }
            t_last_layer_path |= S14_LAYER_PATH_TENSOR_PER_TOKEN;
            return launches;
        }
    }
    if (mode == S14_ACCUM_REFERENCE) {
        dim3 gu(ceil_div(inter, 32), n_jobs_max), gd(ceil_div(hidden, 32), n_jobs_max);
        k_expert_up_reference<<<gu, 32, hidden * sizeof(float), st>>>(dev_table, param_table, x, h,
                                                                      hidden, inter);
        if (km) cudaEventRecord(km->ev[2], st);
        k_expert_down_reference<<<gd, 32, inter * sizeof(float), st>>>(dev_table, param_table, h, d,
                                                                       hidden, inter);
        launches += 2;
        t_last_layer_path |= S14_LAYER_PATH_REFERENCE;
    } else if (tensor_path) {
        *err = launch_moe_layer_umma(st, sm_count, dev_table, param_table, x, d, y, umma->tiles, counters,
                                     umma->status, hidden, inter, router, ep, umma->trace);
        launches += 1;
        t_last_layer_path |= S14_LAYER_PATH_TENSOR;
        if (km) {  // one kernel runs both phases and the mix: its time is booked as the up phase
            cudaEventRecord(km->ev[2], st);
            cudaEventRecord(km->ev[3], st);
            cudaEventRecord(km->ev[4], st);
        }
        return launches;
    } else {
        const uint32_t ctas_per_token = max(1u, (uint32_t)sm_count / n_tokens);
        switch (hidden >> 10) {
        case 1: launch_up_pairwise<1>(st, dev_table, param_table, x, h, inter, n_tokens, ctas_per_token); break;
        case 2: launch_up_pairwise<2>(st, dev_table, param_table, x, h, inter, n_tokens, ctas_per_token); break;
        default: launch_up_pairwise<4>(st, dev_table, param_table, x, h, inter, n_tokens, ctas_per_token); break;
        }
        if (km) cudaEventRecord(km->ev[2], st);
        const uint32_t ctas_per_job = max(1u, ceil_div(2u * (uint32_t)sm_count, n_jobs_max));
        switch (inter >> 10) {
        case 1: launch_down_pairwise<1>(st, dev_table, param_table, h, d, hidden, n_jobs_max, ctas_per_job); break;
        case 2: launch_down_pairwise<2>(st, dev_table, param_table, h, d, hidden, n_jobs_max, ctas_per_job); break;
        default: launch_down_pairwise<4>(st, dev_table, param_table, h, d, hidden, n_jobs_max, ctas_per_job); break;
        }
        launches += 2;
        t_last_layer_path |= S14_LAYER_PATH_F32;
    }
    if (km) cudaEventRecord(km->ev[3], st);
    if (!y) return launches;  // the caller mixes (expert-parallel combine)
    dim3 gm(ceil_div(hidden, 256), n_tokens);
    k_moe_mix<<<gm, 256, 0, st>>>(dev_table, param_table, d, y, hidden);
    if (km) cudaEventRecord(km->ev[4], st);
    launches += 1;
    *err = cudaGetLastError();
    return launches;
}

bool fp8_shared_layer_ok(int sm_count, uint32_t mode, const UmmaScratch *umma, uint32_t n_routed, uint32_t hidden, uint32_t inter) {
    return mode != S14_ACCUM_REFERENCE && umma && umma_layer_ok(sm_count, 1u, n_routed, hidden, inter) &&
           (hidden == 1024u || hidden == 2048u || hidden == 4096u) && (inter == 1024u || inter == 2048u || inter == 4096u);
}

int launch_layer_fp8_shared(cudaStream_t st, int sm_count, const JobTable &routed, const FusedRouter *router, const uint8_t *shared_page,
                            const float *x, const uint16_t *x_bf16, float *h, float *d, float *y,
                            unsigned int *counters, const UmmaScratch *umma, uint32_t hidden, uint32_t inter, cudaError_t *err,
                            BranchPost *post) {
    // The layer kernel first: see s14_fp8_expert.cu.  y may be x: it is written last.
    // at most 32 MB of the page ahead, as it takes the memory from the layer's own last copies (4096 x 4096, 50 MB: two routed experts
    // 39.7 us, so 38.1, six 51.9 and 50.1)
    const size_t page_bytes = 3u * ((size_t)hidden * inter + (size_t)(hidden >> 7) * (inter >> 7)), ahead = std::min<size_t>(page_bytes, 32u << 20);
    *err = launch_moe_layer_umma(st, sm_count, nullptr, routed, x, d, umma->handed, umma->tiles, counters, umma->status, hidden, inter, router,
                                 nullptr, umma->trace, nullptr, 1, nullptr, false, x_bf16, shared_page, ahead);
    if (*err != cudaSuccess) return 0;
    *err = launch_fp8_expert(st, sm_count, x, x_bf16, shared_page, h, umma->handed, y, post, hidden, inter);
    if (post && *err == cudaSuccess) post->done = true;
    return 3;
}

int launch_router(cudaStream_t st, const s14_router_desc &r, float *scores, float *select,
                  JobTable *table_out, const uint8_t *const *page_table, const uint8_t *shared_page,
                  uint32_t shared_kind, unsigned int *counter, cudaError_t *err, const KernelMarks *km,
                  uint32_t ep_rank, uint32_t ep_world, uint32_t shared_owner) {
    const uint32_t warps = r.n_experts * r.n_tokens;
    if (km) cudaEventRecord(km->ev[0], st);
    k_router<<<warps, 64, 0, st>>>(r.x, r.router_weight_bf16, r.bias, scores, select,
                                                r.n_experts, r.hidden, r.n_tokens, r.score_fn, r.top_k,
                                                r.route_scale, r.ids_out, r.weights_out, table_out,
                                                page_table, shared_page, shared_kind, counter, ep_rank,
                                                ep_world, shared_owner);
    *err = cudaGetLastError();
    return 1;
}

__global__ void __launch_bounds__(256)
k_stack_step(const float *__restrict__ x, const float *__restrict__ y, float *out, float *y_copy, uint32_t n,
             uint32_t residual) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = y[i];
    if (y_copy) y_copy[i] = v;
    out[i] = residual ? __fadd_rn(x[i], v) : v;
}

cudaError_t launch_stack_step(cudaStream_t st, const float *x, const float *y, float *out, float *y_copy,
                              uint32_t n, bool residual) {
    k_stack_step<<<ceil_div(n, 256), 256, 0, st>>>(x, y, out, y_copy, n, residual ? 1u : 0u);
    return cudaGetLastError();
}

cudaError_t launch_mix_slots(cudaStream_t st, const float *slots, const float *weights, uint32_t n_routed,
                             int has_shared, float *y, uint32_t hidden) {
    k_mix_slots<<<ceil_div(hidden, 256), 256, 0, st>>>(slots, weights, n_routed, has_shared, y, hidden);
    return cudaGetLastError();
}

}  // namespace s14
