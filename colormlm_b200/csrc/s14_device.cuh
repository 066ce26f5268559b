// Device helpers shared by the kernel files of the S14 MoE path.
#ifndef S14_DEVICE_CUH
#define S14_DEVICE_CUH

#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "s14_internal.h"
#include "s14_page_layout.h"

namespace s14 {

// ---------------------------------------------------------------- decode ----

// Eight E2M1 codes of one 32-bit word (low nibble first) -> four f16x2 words.
__device__ __forceinline__ void e2m1x8_to_h2x4(uint32_t w, uint32_t &h0, uint32_t &h1,
                                               uint32_t &h2, uint32_t &h3) {
    asm("{\n"
        ".reg .b8 b0, b1, b2, b3;\n"
        "mov.b32 {b0, b1, b2, b3}, %4;\n"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n"
        "}\n"
        : "=r"(h0), "=r"(h1), "=r"(h2), "=r"(h3)
        : "r"(w));
}

// Four E4M3 codes of one 32-bit word -> two f16x2 words.
__device__ __forceinline__ void e4m3x4_to_h2x2(uint32_t w, uint32_t &h0, uint32_t &h1) {
    asm("{\n"
        ".reg .b16 lo, hi;\n"
        "mov.b32 {lo, hi}, %2;\n"
        "cvt.rn.f16x2.e4m3x2 %0, lo;\n"
        "cvt.rn.f16x2.e4m3x2 %1, hi;\n"
        "}\n"
        : "=r"(h0), "=r"(h1)
        : "r"(w));
}

__device__ __forceinline__ float2 h2_to_f2(uint32_t h) {
    __half2 v;
    *reinterpret_cast<uint32_t *>(&v) = h;
    return __half22float2(v);
}

// 2^(code-127) as a double: exact for every code 0..254.
__device__ __forceinline__ double ue8m0_to_f64(uint32_t code) {
    return __hiloint2double((int)((code + 896u) << 20), 0);
}

// 2^(code-127) as a float; code 0 is the subnormal 2^-127.
__device__ __forceinline__ float ue8m0_to_f32(uint32_t code) {
    return __uint_as_float(code == 0u ? 0x00400000u : (code << 23));
}

// Weights that a kernel reads once.  ldg_stream takes the non-coherent path, which wants them unchanged from the
// kernel's start to its end: for kernels that start when what precedes them is complete.  A kernel that waits for
// it inside (launch_pdl) has ld_stream and, for what its warps share, ld_u8 and ld_f32.
__device__ __forceinline__ uint4 ldg_stream(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_stream(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_u8(const uint8_t *p) {
    uint32_t v;
    asm volatile("ld.global.u8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_f32x4(const float4 *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_f32(const float *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The sums of P values (a power of two up to 32) over a warp, each added in warp_sum's order: a lane gives away half of the values it
// holds at every step, so 16 values take 16 exchanges where warp_sum takes 5 each.  Lane l returns value l / (32 / P)'s.
template <uint32_t P>
__device__ __forceinline__ double warp_sums(double (&v)[P], uint32_t lane) {
    static_assert(P >= 1u && P <= 32u && (P & (P - 1u)) == 0u, "a power of two");
    uint32_t o = 16u;
#pragma unroll
    for (uint32_t half = P / 2u; half > 0u; half >>= 1, o >>= 1) {
        const bool upper = lane & o;
#pragma unroll
        for (uint32_t i = 0; i < half; ++i) {
            const double give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    double sum = v[0];
#pragma unroll
    for (; o > 0u; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// The reference's SwiGLU (examples/s14_vulkan_numeric.rs:1543-1556) in F32 with
// separate operations.  expf is evaluated in double and rounded once, which
// reproduces a correctly rounded expf.  The F32 quotient g / (1 + e) is taken in double and rounded
// to F32: with 53 >= 2 * 24 + 2 bits the second rounding changes nothing, so this is the correctly
// rounded F32 division; unlike the F32 division, the double one never leaves its inline path for
// operands of F32 range (the F32 one calls a subroutine whenever 1 + e is huge or infinite, which a
// strongly negative gate makes it, and that subroutine's first call in a layer cost the tensor-core
// layer kernel up to a microsecond of instruction fetch while the weights stream).
__device__ __forceinline__ float swiglu_limit_f32(float gate, float up) {
    const float g = fminf(gate, 10.0f);
    const float u = fminf(fmaxf(up, -10.0f), 10.0f);
    const float e = (float)exp(-(double)g);
    const float q = (float)((double)g / (double)__fadd_rn(1.0f, e));
    return __fmul_rn(q, u);
}

// An expert's score from its logit (the double-accumulated dot product, rounded to F32 first):
// sigmoid or sqrt(softplus), evaluated in double and rounded once.
__device__ __forceinline__ float router_score_f32(double logit_sum, uint32_t score_fn) {
    const double l = (double)(float)logit_sum;
    const double sc = (score_fn == S14_SCORE_SIGMOID) ? 1.0 / (1.0 + exp(-l)) : sqrt(l > 20.0 ? l : log1p(exp(l)));
    return (float)sc;
}

__device__ __forceinline__ const JobTable &table_of(const JobTable *dev, const JobTable &param) {
    return dev ? *dev : param;
}

// An expert page as the kernels see it.  FP8 pages are the six tensors one after the other
// (w1 | w3 | w2 | s1 | s3 | s2, weights [N, K] bytes, one UE8M0 code per 128 x 128 block).  MXFP4
// pages are read through the offset functions of s14_page_layout.h from `base`.
struct PageView {
    const uint8_t *base;
    const uint8_t *w1, *w3, *w2, *s1, *s3, *s2;  // FP8 pages only
};

__device__ __forceinline__ PageView page_view(const uint8_t *page, uint32_t kind, uint32_t hidden,
                                              uint32_t inter) {
    PageView v;
    v.base = page;
    const size_t elems = (size_t)hidden * inter;
    const size_t sb = (size_t)((inter + 127u) >> 7) * ((hidden + 127u) >> 7);
    v.w1 = page;
    v.w3 = page + elems;
    v.w2 = page + 2 * elems;
    v.s1 = page + 3 * elems;
    v.s3 = v.s1 + sb;
    v.s2 = v.s3 + sb;
    (void)kind;
    return v;
}

// The dependency calls of a kernel launched by launch_pdl: wait until what precedes the launch in the stream is complete
// and its writes are visible, then let the launch behind be set up.  In this order a launch's set-up can overlap the
// kernel directly in front of it alone: everything before that one is complete.
__device__ __forceinline__ void dependency_wait() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}
// A hint that the lines at p will be read: allowed in front of dependency_wait() even where an earlier kernel of the
// stream still writes them, because it brings them to the L2, which that kernel's stores go through, and no value
// to this kernel.
__device__ __forceinline__ void l2_hint(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The result of a launch.  A refused launch also stays behind as the thread's last error, where the next check of the
// library, or of whoever shares the runtime with it, would find it and blame another call.
inline cudaError_t launch_status(cudaError_t e) {
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
}

// A launch as a programmatic dependent of what precedes it in the stream, optionally in clusters of
// `cluster` CTAs (0: none).  But for those below the kernels launched so read nothing in front of dependency_wait(), weights and pages
// included: a caller's kernel may write those too, and one that lets its own dependents start early is not even
// complete when such a launch starts.  Behind it they use coherent loads that the compiler keeps in place (__ldcg,
// ld_stream, ld_u8, ld_f32).  A non-coherent load (__ldg, or a plain one through a const __restrict__ pointer)
// could return what the operand held before.
//
// Four kernels read in front of their wait what the launch directly in front of them does not write, and may only follow a launch that
// triggers behind its own wait, because then everything in front of that one is complete when they start: the first digits launch of a
// block call (k_block_digits or its official form, early: reads x, writes digits), behind the launch that picks the routes or a copy; k_hc_reduce with kAhead (the streams),
// behind k_hc_dots; k_fp8_expert_up (the token and its page; writes h), behind the layer kernel with a page `ahead`; the blocks' down kernel
// (k_block_pair: records and pages), behind the second digits launch.  The layer kernel
// without one copies pages, router rows and tables, which are constant during a step, in front of its wait.  k_hc_reduce, k_router and
// the layer kernel without a page ahead trigger in front of their own wait: none of the three may follow one of these directly.
//
// `shared`: bytes of shared memory an SM needs for this kernel, 1 KB per CTA included (0: not said).  A dependent launch takes
// over SMs from a kernel that is still running elsewhere, and without a word the SMs stay divided as that kernel has them:
// behind one that fills shared memory the loads of the next find hardly any L1 to be in flight in.
template <class Kernel, class... Args>
inline cudaError_t launch_dependent(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, uint32_t cluster, size_t shared, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[3];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster) {
        cudaLaunchAttribute &a = attr[cfg.numAttrs++];
        a.id = cudaLaunchAttributeClusterDimension;
        a.val.clusterDim.x = cluster;
        a.val.clusterDim.y = 1;
        a.val.clusterDim.z = 1;
    }
    if (shared) {
        constexpr size_t kMost = 228u * 1024u;   // of an SM
        cudaLaunchAttribute &a = attr[cfg.numAttrs++];
        a.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        a.val.sharedMemCarveout = (unsigned)std::min<size_t>(100u, (shared * 100u + kMost - 1u) / kMost);
    }
    return launch_status(cudaLaunchKernelEx(&cfg, kernel, args...));
}
template <class Kernel, class... Args>
inline cudaError_t launch_pdl(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, uint32_t cluster, Args... args) {
    return launch_dependent(kernel, grid, block, smem, st, cluster, 0u, args...);
}

// The CTAs of a cluster where fits(n) says whether clusters of n can run: the most of 16 and, beyond which a device or the part of it
// that the process has may refuse them, the portable 8.
template <class Fits>
inline uint32_t cluster_that_fits(Fits fits) {
    return fits(16u) ? 16u : 8u;
}

// A kernel in clusters of sixteen (beyond the portable eight): allowed once per kernel and device.
template <class Kernel>
inline cudaError_t allow_wide_clusters(Kernel kernel, bool (&done)[64]) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return e != cudaSuccess ? e : cudaErrorInvalidDevice;
    if (!done[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        done[dev] = e == cudaSuccess;
    }
    return e;
}

}  // namespace s14

#endif
