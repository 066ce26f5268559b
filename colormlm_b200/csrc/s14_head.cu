// The LM head of a decode step or a verify block: full logits of 1..8 tokens over a BF16 matrix, the greedy
// token, and the steps before it (the head's hyper-connection reduce and RMSNorm) as one launch.
// Reference: fast16/research/polaris_meridian_v1/local_s14_primitives/final_head.py:43-191,
// scheduler/s14_runner/src/runner.rs:485-508.
#include <cooperative_groups.h>

#include "s14_device.cuh"

namespace s14 {

namespace cg = cooperative_groups;

namespace {

// ---- logits -------------------------------------------------------------------------------------
//
// logits[t, v] = sum_k x[t, k] * W[v, k], W BF16, 1 GB per call at 129280 x 4096: the weight stream bounds it
// (1.06 GB / 6.55 TB/s = 162 us), so what a weight element costs on the SM has to stay below 1.5 clocks per
// 12 elements.  A register kernel does not manage that for eight tokens: it reads 32 bytes of x per weight
// element through the L1 and converts a partial sum to double per 4 products (16 conversions per clock and
// SM), 1118 us.  Here x is split once per CTA into three BF16 parts (x = h + m + l: 6, 8 and 8
// significant bits, each remainder's sign being worth one more; exact for |x| from 2^-110, below which m and l run out
// of BF16's exponents, to where h may still be rounded up, 2^127) kept in shared memory, and a warp takes
// sixteen rows of W as the A operand of mma.m16n8k16, the eight tokens' parts as B: every product is exact in
// F32.  The sums of sixteen products with h (few of their bits fall off the F32 sum) go to double every 16 elements of K;
// m and l, 2^-6 (2^-3 for BF16 values) and 2^-15 of h, are summed in F32 over 128 elements and then added (blocks of K
// that do not depend on the number of tokens).  Measured RMS error over the RMS result, N(0,1) x N(0,0.02), K = 4096
// (2048 the same within 2 %), rounding the result alone 2.54e-8: F32 x 2.94e-8, the register kernel's 4-product chains
// 4.75e-8; BF16 values 2.62e-8 and 2.65e-8 (with six bits in h 2.95e-8, four 2.68e-8).
// A lane loads 16 bytes (eight k) of each of its two rows: words 0, 1 are its k slots of a first MMA, words 2, 3
// of a second one, and x is read from shared memory in the same order, so K is only permuted.  Two warps share
// sixteen rows (the halves of K): 8080 row tiles over 148 x 8 pairs are 6.8 rounds, the last one 82 % full.  Eight
// 16-byte loads per lane are in flight (64 KB per SM), across row tiles; they need room in the L1, which shared
// memory takes away (with eight tokens' 198 KB of parts resident: 290 us).  So K is walked in `phases` of at
// most 50 KB of parts, the CTA's row tiles once per phase, their sums waiting in shared memory in between.
constexpr uint32_t kHeadThreads = 512, kHeadPairs = kHeadThreads / 64u, kHeadDepth = 4;
constexpr uint32_t kHeadPad = 64;   // a token's row of parts: the lanes of two tokens then use all banks once
constexpr uint32_t kHeadTiles = 56; // row tiles of a CTA whose sums wait between phases (1 KB each)
constexpr size_t kHeadPartBytes = 50u * 1024u;

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The BF16 parts of v: 6 significant bits, then 8, then the 8 that are left (nearest each time, so a remainder is at most
// half a unit of the part before).  A BF16 value, which two parts hold in any case, gives the first one
// three: the sums of its products lose less on their way into double.  Infinities and NaNs go into the first alone.
__device__ __forceinline__ void head_parts(float v, uint32_t (&p)[3]) {
    const uint32_t u = __float_as_uint(v);
    const bool bf16 = (u & 0xffffu) == 0u;
    const uint32_t keep = bf16 ? 0xffe00000u : 0xfffc0000u;
    uint32_t h = (u + (bf16 ? 0x00100000u : 0x00020000u)) & keep;
    if ((h & 0x7f800000u) == 0x7f800000u && isfinite(v)) h = u & keep;  // would round to infinity
    if (!isfinite(v)) {
        const __nv_bfloat16 b = __float2bfloat16_rn(v);
        p[0] = *reinterpret_cast<const uint16_t *>(&b);
        p[1] = p[2] = 0u;
        return;
    }
    const float r = __fsub_rn(v, __uint_as_float(h));  // exact
    const __nv_bfloat16 m = __float2bfloat16_rn(r), l = __float2bfloat16_rn(__fsub_rn(r, __bfloat162float(m)));
    p[0] = h >> 16;
    p[1] = *reinterpret_cast<const uint16_t *>(&m);
    p[2] = *reinterpret_cast<const uint16_t *>(&l);
}

// Sixteen rows times the tokens over 128 elements of K, as one warp takes them: four steps of 32.  A row's logit is these
// sums added in the order of K within each half of a phase, the halves added, the phases added: whichever
// kernel and shard works the row out, the bits are the same.
struct HeadBlock {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    float low[4] = {0.f, 0.f, 0.f, 0.f}, c[2][4];
    __device__ __forceinline__ void step(const uint4 &a0, const uint4 &a1, const uint4 (&b)[3]) {
#pragma unroll
        for (int e = 0; e < 4; ++e) c[0][e] = c[1][e] = 0.f;
        mma_bf16(c[0], a0.x, a1.x, a0.y, a1.y, b[0].x, b[0].y);
        mma_bf16(c[1], a0.z, a1.z, a0.w, a1.w, b[0].z, b[0].w);
#pragma unroll
        for (int part = 2; part >= 1; --part) {
            mma_bf16(low, a0.x, a1.x, a0.y, a1.y, b[part].x, b[part].y);
            mma_bf16(low, a0.z, a1.z, a0.w, a1.w, b[part].z, b[part].w);
        }
    }
    __device__ __forceinline__ void carry() {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            acc[e] += (double)c[0][e];
            acc[e] += (double)c[1][e];
        }
    }
    __device__ __forceinline__ double sum(int e) const { return acc[e] + (double)low[e]; }
};

// One row's dot product by a whole warp as k_head_logits takes it, for the sums that the parts get wrong: an infinite
// weight times a part that is zero is NaN, two parts of opposite sign make inf - inf of it, and a product near the
// largest float overflows in two parts at once.  Out of line: its callers are never there with ordinary numbers, and
// k_head_mma has no register to spare.
__device__ __noinline__ float head_row_dot(const float *x, const uint16_t *w, uint32_t hidden) {
    double acc = 0.0;
#pragma unroll 1
    for (uint32_t p = threadIdx.x & 31u; p < (hidden >> 3); p += 32u) {
        const uint4 q = ld_stream(reinterpret_cast<const uint4 *>(w) + p);
        const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
        float2 part = make_float2(0.f, 0.f);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const float2 xv = __ldcg(reinterpret_cast<const float2 *>(x + p * 8u) + i);
            part = __ffma2_rn(make_float2(__uint_as_float(wd[i] << 16), __uint_as_float(wd[i] & 0xffff0000u)), xv, part);
        }
        acc += (double)part.x + (double)part.y;
    }
    return (float)warp_sum(acc);
}

__global__ void __launch_bounds__(kHeadThreads, 1)
k_head_mma(const float *__restrict__ x, const uint16_t *__restrict__ w, float *__restrict__ out, uint32_t n_rows, uint32_t hidden,
           uint32_t out_stride, uint32_t n_tokens, uint32_t phases) {
    extern __shared__ __align__(16) uint8_t s_parts[];      // [3][n_tokens][pitch], then the tiles' sums [tile][4][32]
    __shared__ double s_half[kHeadPairs][2][4][32];          // the second warp's half of K, by tile parity
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, pair = warp >> 1, half = warp & 1u;
    const uint32_t g = lane >> 2, q = lane & 3u;
    const uint32_t span = hidden / phases;                   // of K per phase
    const uint32_t pitch = span * 2u + kHeadPad, part_bytes = n_tokens * pitch;
    const uint32_t steps = span >> 6;                        // of 32 k, of this warp's half: a multiple of four
    const uint32_t n_tiles = (n_rows + 15u) >> 4, grid = gridDim.x;
    double *const s_sum = reinterpret_cast<double *>(s_parts + 3u * part_bytes);
    // the CTA's tiles: blockIdx.x + i * grid, i < n_mine; at most kHeadTiles at a time, dealt to the pairs in turn
    const uint32_t n_mine = n_tiles > blockIdx.x ? (n_tiles - blockIdx.x + grid - 1u) / grid : 0u;
    const uint32_t batch = phases > 1u ? kHeadTiles : n_mine;

    const uint16_t *p0, *p1;
    auto rows_of = [&](uint32_t i, uint32_t phase) {
        const uint32_t t = blockIdx.x + i * grid, r0 = min(t * 16u + g, n_rows - 1u), r1 = min(t * 16u + g + 8u, n_rows - 1u);
        const uint32_t k0 = phase * span + half * (span >> 1) + q * 8u;
        p0 = w + (size_t)r0 * hidden + k0;
        p1 = w + (size_t)r1 * hidden + k0;
    };
    uint4 a0[kHeadDepth], a1[kHeadDepth];
    auto fetch = [&](uint32_t i, uint32_t k) {
        a0[i] = ld_stream(reinterpret_cast<const uint4 *>(p0 + (k + i) * 32u));
        a1[i] = ld_stream(reinterpret_cast<const uint4 *>(p1 + (k + i) * 32u));
    };
    dependency_wait();
    if (pair < n_mine) {  // in flight while x is split
        rows_of(pair, 0u);
#pragma unroll
        for (uint32_t i = 0; i < kHeadDepth; ++i) fetch(i, 0u);
    }
    const uint8_t *const sb = s_parts + (g < n_tokens ? g : 0u) * pitch + half * span + q * 16u;
    const bool has_b = g < n_tokens;
    uint32_t parity = 0;
#pragma unroll 1
    for (uint32_t base = 0; base < n_mine; base += batch) {
        const uint32_t end = min(base + batch, n_mine);
#pragma unroll 1
        for (uint32_t phase = 0; phase < phases; ++phase) {
            __syncthreads();  // the parts of the phase before are not read any more
            for (uint32_t i = tid; i < n_tokens * (span >> 1); i += kHeadThreads) {
                const uint32_t t = i / (span >> 1), k2 = i - t * (span >> 1);
                const float2 v = __ldcg(reinterpret_cast<const float2 *>(x + (size_t)t * hidden + phase * span) + k2);
                uint32_t px[3], py[3];
                head_parts(v.x, px);
                head_parts(v.y, py);
#pragma unroll
                for (uint32_t part = 0; part < 3; ++part)
                    *reinterpret_cast<uint32_t *>(s_parts + part * part_bytes + t * pitch + k2 * 4u) = px[part] | (py[part] << 16);
            }
            __syncthreads();
#pragma unroll 1
            for (uint32_t i = base + pair; i < end; i += kHeadPairs, parity ^= 1u) {
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
                // what this pair reads after this tile: its next tile, of this phase or the next, or of the next batch
                uint32_t next = i + kHeadPairs, next_phase = phase;
                if (next >= end) {
                    next = base + pair;
                    if (++next_phase == phases) next_phase = 0u, next = end + pair;
                }
                const bool more = next < n_mine;
#pragma unroll 1
                for (uint32_t s0 = 0; s0 < steps; s0 += kHeadDepth) {
                    const bool last = s0 + kHeadDepth == steps;
                    if (last && more) rows_of(next, next_phase);
                    const uint32_t k_next = last ? 0u : s0 + kHeadDepth;
                    HeadBlock blk;
#pragma unroll
                    for (uint32_t j = 0; j < kHeadDepth; ++j) {
                        uint4 b[3];
#pragma unroll
                        for (uint32_t part = 0; part < 3; ++part) {
                            b[part] = make_uint4(0u, 0u, 0u, 0u);
                            if (has_b) b[part] = *reinterpret_cast<const uint4 *>(sb + part * part_bytes + (s0 + j) * 64u);
                        }
                        blk.step(a0[j], a1[j], b);
                        if (!last || more) fetch(j, k_next);
                        blk.carry();
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[e] += blk.sum(e);
                }
                if (half == 1u) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) s_half[pair][parity][e][lane] = acc[e];
                }
                asm volatile("bar.sync %0, 64;" ::"r"(1u + pair) : "memory");
                if (half == 0u) {
                    double *const sum = s_sum + (size_t)(i - base) * 128u + lane;   // (this lane's own words)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        acc[e] += s_half[pair][parity][e][lane];
                        if (phase > 0u) acc[e] += sum[e * 32];
                        if (phase + 1u < phases) {
                            sum[e * 32] = acc[e];
                        } else {
                            // lane holds rows g, g + 8 of the tile and tokens 2 q, 2 q + 1
                            const uint32_t row = (blockIdx.x + i * grid) * 16u + g + (e >> 1) * 8u, t = 2u * q + (e & 1);
                            const bool mine = row < n_rows && t < n_tokens;
                            if (mine) out[(size_t)t * out_stride + row] = (float)acc[e];
                            // a sum that is not finite says little about the dot product (head_row_dot)
                            uint32_t redo = __ballot_sync(0xffffffffu, mine && !isfinite(acc[e]));
                            while (redo) {
                                const uint32_t src = __ffs((int)redo) - 1, t_src = 2u * (src & 3u) + (e & 1);
                                const uint32_t row_src = (blockIdx.x + i * grid) * 16u + (src >> 2) + (e >> 1) * 8u;
                                const float v = head_row_dot(x + (size_t)t_src * hidden, w + (size_t)row_src * hidden, hidden);
                                if (lane == src) out[(size_t)t * out_stride + row] = v;
                                redo &= redo - 1u;
                            }
                        }
                    }
                }
            }
        }
    }
}

// The same logits where there are at most two row tiles per SM: `wide` warps take one tile, the blocks of 128 k in turn, a
// block's loads in flight while the one before is worked on; the blocks' sums wait in shared memory and are added in
// k_head_mma's order (the same bits: a vocabulary shard may be small where another is not).  There a pair of warps walks all of
// K for a tile.  Up to a tile per SM sixteen warps share one; above that eight do, in CTAs of one tile (two CTAs per SM) or of
// two, which split x once for both.  kShared: x is split into its parts once per CTA; what does not fit in shared memory
// beside room for the loads in the L1 is split by every warp in the registers of the lanes that use it, which costs the same
// for one token as for eight.  What bounds it is the chain per block - loads, four dependent steps, the sums' way into double -
// times the blocks of a warp: more loads ahead do not help (4000 x 4096 one token 10.8 with two blocks ahead, 10.6 with one),
// more warps per tile do.  us, with eight warps to a tile always, no loads ahead and parts per CTA / now / by the register
// kernel below, which sums in another order: 64 x 4096 one token 7.8 / 5.7 / 5.6, 1000 x 7168 one token 17.4 / 9.6 / 10.9,
// four 38.8 / 18.3 / 16.2, 4000 x 4096 one token 11.9 / 10.5 / 8.8, four 24.2 / 13.3 / 23.6, eight 20.3 / 20.2 / 29.1.
constexpr uint32_t kFewSmallParts = 2048;   // tokens x hidden up to which splitting x twice on an SM costs less than sharing it
constexpr size_t kFewTwoBytes = 190u * 1024u, kFewOneBytes = 200u * 1024u;   // of shared memory: two tiles, one tile
template <bool kShared>
__global__ void __launch_bounds__(512, 1)
k_head_mma_few(const float *__restrict__ x, const uint16_t *__restrict__ w, float *__restrict__ out, uint32_t n_rows, uint32_t hidden,
               uint32_t out_stride, uint32_t n_tokens, uint32_t phases, uint32_t wide) {
    extern __shared__ __align__(16) uint8_t s_few[];   // [tile][K / 128][4][32] sums of the blocks, then the parts [3][n_tokens][pitch]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, g = lane >> 2, q = lane & 3u;
    const uint32_t n_blk = hidden >> 7, per_half = n_blk / (2u * phases);
    const uint32_t tiles = (blockDim.x >> 5) / wide, local = warp / wide, mine = warp - local * wide;   // `wide` warps to a tile
    const uint32_t pitch = hidden * 2u + kHeadPad, row0 = (blockIdx.x * tiles + local) * 16u;
    double *const s_sum = reinterpret_cast<double *>(s_few) + (size_t)local * n_blk * 128u;
    uint8_t *const s_x = s_few + (size_t)tiles * n_blk * 1024u;
    const bool has_b = g < n_tokens;
    const uint16_t *const p0 = w + (size_t)min(row0 + g, n_rows - 1u) * hidden + q * 8u;
    const uint16_t *const p1 = w + (size_t)min(row0 + g + 8u, n_rows - 1u) * hidden + q * 8u;
    const float *const xg = x + (size_t)(has_b ? g : 0u) * hidden + q * 8u;
    uint4 a0[kHeadDepth], a1[kHeadDepth];
    auto fetch = [&](uint32_t j, uint32_t b) {
        a0[j] = ld_stream(reinterpret_cast<const uint4 *>(p0 + b * 128u + j * 32u));
        a1[j] = ld_stream(reinterpret_cast<const uint4 *>(p1 + b * 128u + j * 32u));
    };
    const uint32_t end = row0 < n_rows ? n_blk : 0u;   // (the last CTA may have a tile less)
    dependency_wait();
    if (mine < end) {   // in flight while x is split
#pragma unroll
        for (uint32_t j = 0; j < kHeadDepth; ++j) fetch(j, mine);
    }
    auto parts_of = [](const float4 &lo, const float4 &hi, uint4 (&bp)[3]) {
        const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        uint32_t wd[3][4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            uint32_t px[3], py[3];
            head_parts(v[2 * i], px);
            head_parts(v[2 * i + 1], py);
#pragma unroll
            for (uint32_t part = 0; part < 3; ++part) wd[part][i] = px[part] | (py[part] << 16);
        }
#pragma unroll
        for (uint32_t part = 0; part < 3; ++part) bp[part] = make_uint4(wd[part][0], wd[part][1], wd[part][2], wd[part][3]);
    };
    if constexpr (kShared) {
        for (uint32_t i = tid; i < n_tokens * (hidden >> 3); i += blockDim.x) {
            const uint32_t t = i / (hidden >> 3), k8 = i - t * (hidden >> 3);
            const float4 *at = reinterpret_cast<const float4 *>(x + (size_t)t * hidden) + 2u * k8;
            uint4 bp[3];
            parts_of(__ldcg(at), __ldcg(at + 1), bp);
#pragma unroll
            for (uint32_t part = 0; part < 3; ++part) *reinterpret_cast<uint4 *>(s_x + (part * n_tokens + t) * pitch + k8 * 16u) = bp[part];
        }
        __syncthreads();
    }
#pragma unroll 1
    for (uint32_t b = mine; b < end; b += wide) {
        const bool more = b + wide < end;
        HeadBlock blk;
#pragma unroll
        for (uint32_t j = 0; j < kHeadDepth; ++j) {
            uint4 bp[3] = {};
            if (has_b) {
                if constexpr (kShared) {
#pragma unroll
                    for (uint32_t part = 0; part < 3; ++part)
                        bp[part] = *reinterpret_cast<const uint4 *>(s_x + (part * n_tokens + g) * pitch + b * 256u + j * 64u + q * 16u);
                } else {
                    const float4 *at = reinterpret_cast<const float4 *>(xg + b * 128u + j * 32u);
                    parts_of(__ldcg(at), __ldcg(at + 1), bp);
                }
            }
            blk.step(a0[j], a1[j], bp);
            if (more) fetch(j, b + wide);
            blk.carry();
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) s_sum[(b * 4u + e) * 32u + lane] = blk.sum(e);
    }
    __syncthreads();
    if (mine >= 4u || row0 >= n_rows) return;
    const uint32_t e = mine;   // four warps of a tile: accumulator e of every lane
    double sum = 0.0;
#pragma unroll 1
    for (uint32_t phase = 0; phase < phases; ++phase) {
        double half[2] = {0.0, 0.0};
        const double *at = s_sum + ((size_t)phase * 2u * per_half * 4u + e) * 32u + lane;
#pragma unroll 4
        for (uint32_t p = 0; p < per_half; ++p) {
            half[0] += at[p * 128u];
            half[1] += at[(per_half + p) * 128u];
        }
        const double both = half[0] + half[1];
        sum = phase ? both + sum : both;
    }
    const uint32_t row = row0 + g + (e >> 1) * 8u, t = 2u * q + (e & 1u);
    const bool ours = row < n_rows && t < n_tokens;
    if (ours) out[(size_t)t * out_stride + row] = (float)sum;
    uint32_t redo = __ballot_sync(0xffffffffu, ours && !isfinite(sum));
    while (redo) {
        const uint32_t src = __ffs((int)redo) - 1, t_src = 2u * (src & 3u) + (e & 1u);
        const float v = head_row_dot(x + (size_t)t_src * hidden, w + (size_t)(row0 + (src >> 2) + (e >> 1) * 8u) * hidden, hidden);
        if (lane == src) out[(size_t)t * out_stride + row] = v;
        redo &= redo - 1u;
    }
}

// Any hidden size that is a multiple of 8: a warp per row; 8 products in F32, carried in F64.  Up to four tokens the
// weight stream bounds it and four loads per lane pay (129280 x 4104, one token: 228 us, with one load 263; four tokens
// 541 and 598); from five on the warps that the registers of four would cost do more (eight tokens 1138 and 1066).
template <int NT>
__global__ void __launch_bounds__(256)
k_head_logits(const float *__restrict__ x, const uint16_t *__restrict__ w, float *__restrict__ out, uint32_t n_rows, uint32_t hidden,
              uint32_t out_stride) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    constexpr int kLoads = NT <= 4 ? 4 : 1;
    for (uint32_t v = warp; v < n_rows; v += n_warps) {
        const uint4 *row = reinterpret_cast<const uint4 *>(w + (size_t)v * hidden);
        double acc[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t] = 0.0;
        // 16-byte loads of the row in flight per lane (the row is read once, from HBM); the sums are taken in the order of
        // the pieces
        for (uint32_t p0 = lane; p0 < (hidden >> 3); p0 += 32u * kLoads) {
            uint4 q4[kLoads];
#pragma unroll
            for (int u = 0; u < kLoads; ++u)
                q4[u] = (p0 + 32u * u < (hidden >> 3)) ? ldg_stream(row + p0 + 32u * u) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                const uint32_t p = p0 + 32u * u;
                if (p >= (hidden >> 3)) break;
                const uint32_t wd[4] = {q4[u].x, q4[u].y, q4[u].z, q4[u].w};
                float wf[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    wf[i * 2] = __uint_as_float(wd[i] << 16);
                    wf[i * 2 + 1] = __uint_as_float(wd[i] & 0xffff0000u);
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const float4 xa = __ldg(reinterpret_cast<const float4 *>(x + (size_t)t * hidden + p * 8));
                    const float4 xb = __ldg(reinterpret_cast<const float4 *>(x + (size_t)t * hidden + p * 8 + 4));
                    float2 part = make_float2(0.f, 0.f);
                    part = __ffma2_rn(make_float2(wf[0], wf[1]), make_float2(xa.x, xa.y), part);
                    part = __ffma2_rn(make_float2(wf[2], wf[3]), make_float2(xa.z, xa.w), part);
                    part = __ffma2_rn(make_float2(wf[4], wf[5]), make_float2(xb.x, xb.y), part);
                    part = __ffma2_rn(make_float2(wf[6], wf[7]), make_float2(xb.z, xb.w), part);
                    acc[t] += (double)part.x + (double)part.y;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const double s = warp_sum(acc[t]);
            if (lane == 0) out[(size_t)t * out_stride + v] = (float)s;
        }
    }
}

// ---- greedy token -------------------------------------------------------------------------------
//
// Largest logit, lowest id on ties, -1 if there is a NaN.  One CTA reads 517 KB at the rate one SM takes in
// (13.9 us for 129 280 logits); a cluster of sixteen, or eight where sixteen are refused, shares the reading and hands its candidates over in shared
// memory, so the call still needs no scratch that calls on several streams would share.  A thread keeps its largest logit and
// that one's id; warps reduce the logit as an ordered integer, then the id of those that have it, in two operations each.
// Calls one after another, us: eight CTAs and 64-bit candidates through shuffles 3.18 (129 280 logits), 2.04 (8192); with these
// reductions 2.39, 1.81; and sixteen CTAs 2.04, 1.69 (and 1.49 for 64 logits, where the eight took 1.85).
constexpr uint32_t kArgmaxMost = 16, kArgmaxThreads = 512;

struct ArgmaxBest {
    uint32_t key, id;   // the logit as an ordered integer (all ones: a NaN was met), the lowest id that has it
};
__device__ __forceinline__ ArgmaxBest warp_best(ArgmaxBest b) {
    const uint32_t key = __reduce_max_sync(0xffffffffu, b.key);
    return {key, __reduce_min_sync(0xffffffffu, b.key == key ? b.id : 0xffffffffu)};
}

__global__ void __launch_bounds__(kArgmaxThreads)
k_greedy_argmax(const float *__restrict__ logits, uint32_t vocab, int64_t *__restrict__ result) {
    __shared__ uint2 s_warp[kArgmaxThreads / 32], s_cta[kArgmaxMost];
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();  // every CTA of the cluster runs: its shared memory may be written
    dependency_wait();
    const uint32_t n = cluster.num_blocks(), rank = cluster.block_rank(), tid = threadIdx.x, lane = tid & 31u;
    // a thread's ids rise, so the first of equal logits stays; one that met nothing has an id that loses against any
    float best = -INFINITY;
    uint32_t id = 0xffffffffu;
    bool nan = false;
    auto take = [&](float v, uint32_t i) {
        nan = nan || v != v;
        if (v > best || id == 0xffffffffu) best = v, id = i;
    };
    if ((reinterpret_cast<uintptr_t>(logits) & 15u) == 0u) {
        const uint32_t n4 = vocab >> 2;
        constexpr uint32_t kLoads = 4;   // in flight, the last round's too (129 280 logits are 3.95 loads a thread)
        for (uint32_t i0 = rank * kArgmaxThreads + tid; i0 < n4; i0 += kLoads * n * kArgmaxThreads) {
            float4 v[kLoads];
#pragma unroll
            for (uint32_t k = 0; k < kLoads; ++k)
                if (const uint32_t i = i0 + k * n * kArgmaxThreads; i < n4) v[k] = __ldcg(reinterpret_cast<const float4 *>(logits) + i);
#pragma unroll
            for (uint32_t k = 0; k < kLoads; ++k)
                if (const uint32_t i = i0 + k * n * kArgmaxThreads; i < n4)
                    take(v[k].x, 4u * i), take(v[k].y, 4u * i + 1u), take(v[k].z, 4u * i + 2u), take(v[k].w, 4u * i + 3u);
        }
        if (rank == 0u && tid < (vocab & 3u)) take(__ldcg(logits + n4 * 4u + tid), n4 * 4u + tid);
    } else {
        for (uint32_t i = rank * kArgmaxThreads + tid; i < vocab; i += n * kArgmaxThreads) take(__ldcg(logits + i), i);
    }
    const uint32_t b = __float_as_uint(__fadd_rn(best, 0.0f));  // -0 and +0 are equal
    ArgmaxBest mine = {id == 0xffffffffu ? 0u : (b & 0x80000000u) ? ~b : (b | 0x80000000u), id};
    if (nan) mine.key = 0xffffffffu;
    mine = warp_best(mine);
    if (lane == 0u) s_warp[tid >> 5] = make_uint2(mine.key, mine.id);
    __syncthreads();
    if (tid < 32u) {
        const uint2 w = tid < kArgmaxThreads / 32u ? s_warp[tid] : make_uint2(0u, 0xffffffffu);
        mine = warp_best({w.x, w.y});
        if (tid == 0u) *cluster.map_shared_rank(&s_cta[rank], 0) = make_uint2(mine.key, mine.id);
    }
    cluster.sync();
    if (rank == 0u && tid < 32u) {
        const uint2 w = tid < n ? s_cta[tid] : make_uint2(0u, 0xffffffffu);
        mine = warp_best({w.x, w.y});
        if (tid == 0u) *result = mine.key == 0xffffffffu ? -1ll : (int64_t)mine.id;
    }
}

// ---- the steps before the logits ----------------------------------------------------------------
//
// final_head.py:43-110: hyper-connection reduce of the four BF16 streams, RMSNorm, and the BF16 values as F32
// (the logits kernel's input), one launch of one cluster instead of four: the 64 KB of a token's state and
// matrix are split over eight SMs, the sums cross in shared memory.  The arithmetic is that of the operators
// s14_cmd_hc_head_reduce and s14_cmd_rms_norm: long sums in double, the rest F32 in the expressions' order,
// the reduced and the normalised vector rounded to BF16.
constexpr uint32_t kPrepCluster = 8, kPrepThreads = 256;

__device__ __forceinline__ float bf16_of(const uint16_t *p) { return __uint_as_float((uint32_t)__ldcg(p) << 16); }

__global__ void __launch_bounds__(kPrepThreads)
k_head_prep(const uint16_t *__restrict__ state, const float *__restrict__ fn, const float *__restrict__ scale,
            const float *__restrict__ base, const float *__restrict__ norm_weight, uint32_t hidden, float norm_eps, float hc_eps,
            float *__restrict__ x_out) {
    __shared__ double s_red[kPrepThreads / 32][5];
    __shared__ double s_sums[kPrepCluster][5];   // four dot products and the sum of squares of every CTA's share
    __shared__ double s_ss[kPrepCluster];
    __shared__ float s_pre[4];
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();  // every CTA of the cluster runs: its shared memory may be written
    dependency_wait();
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t n = 4u * hidden, share = n / kPrepCluster;   // a multiple of 128
    const float scale0 = __ldcg(scale), base_h = tid < 4u ? __ldcg(base + tid) : 0.0f;  // (read here: a serial chain uses them)
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (uint32_t i = tid * 4u; i < share; i += kPrepThreads * 4u) {
        const uint32_t k = rank * share + i;
        const uint2 b = __ldcg(reinterpret_cast<const uint2 *>(state + k));
        const float xs[4] = {__uint_as_float(b.x << 16), __uint_as_float(b.x & 0xffff0000u), __uint_as_float(b.y << 16),
                             __uint_as_float(b.y & 0xffff0000u)};
        float4 f[4];
#pragma unroll
        for (uint32_t m = 0; m < 4; ++m) f[m] = __ldcg(reinterpret_cast<const float4 *>(fn + (size_t)m * n + k));
#pragma unroll
        for (uint32_t m = 0; m < 4; ++m) {
            v[m] += (double)xs[0] * (double)f[m].x;
            v[m] += (double)xs[1] * (double)f[m].y;
            v[m] += (double)xs[2] * (double)f[m].z;
            v[m] += (double)xs[3] * (double)f[m].w;
        }
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) v[4] += (double)xs[e] * (double)xs[e];
    }
#pragma unroll
    for (uint32_t j = 0; j < 5; ++j) {
        v[j] = warp_sum(v[j]);
        if (lane == 0u) s_red[warp][j] = v[j];
    }
    __syncthreads();
    if (tid < 5u) {
        double s = 0.0;
#pragma unroll
        for (uint32_t wi = 0; wi < kPrepThreads / 32u; ++wi) s += s_red[wi][tid];
#pragma unroll
        for (uint32_t r = 0; r < kPrepCluster; ++r) *cluster.map_shared_rank(&s_sums[rank][tid], r) = s;
    }
    cluster.sync();
    if (tid < 4u) {
        double dot = 0.0, ss = 0.0;
#pragma unroll
        for (uint32_t r = 0; r < kPrepCluster; ++r) dot += s_sums[r][tid], ss += s_sums[r][4];
        const float rs = (float)(1.0 / sqrt((double)__fadd_rn((float)(ss / (double)n), norm_eps)));
        const float mix = __fmul_rn((float)dot, rs);
        s_pre[tid] = __fadd_rn((float)(1.0 / (1.0 + exp(-(double)__fadd_rn(__fmul_rn(mix, scale0), base_h)))), hc_eps);
    }
    __syncthreads();
    // this CTA's eighth of the hidden vector, at most four elements a thread (hidden <= 8192)
    const uint32_t part = hidden / kPrepCluster;
    float red[4];
    double ss = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t e = tid + i * kPrepThreads, d = rank * part + e;
        red[i] = 0.0f;
        if (e < part) {
            float acc = __fmul_rn(s_pre[0], bf16_of(state + d));
#pragma unroll
            for (uint32_t h = 1; h < 4; ++h) acc = __fadd_rn(acc, __fmul_rn(s_pre[h], bf16_of(state + (size_t)h * hidden + d)));
            red[i] = __bfloat162float(__float2bfloat16_rn(acc));
            ss += (double)red[i] * (double)red[i];
        }
    }
    ss = warp_sum(ss);
    __syncthreads();
    if (lane == 0u) s_red[warp][0] = ss;
    __syncthreads();
    if (tid == 0u) {
        double s = 0.0;
#pragma unroll
        for (uint32_t wi = 0; wi < kPrepThreads / 32u; ++wi) s += s_red[wi][0];
#pragma unroll
        for (uint32_t r = 0; r < kPrepCluster; ++r) *cluster.map_shared_rank(&s_ss[rank], r) = s;
    }
    cluster.sync();
    double all = 0.0;
#pragma unroll
    for (uint32_t r = 0; r < kPrepCluster; ++r) all += s_ss[r];
    const float rs = (float)(1.0 / sqrt((double)__fadd_rn((float)(all / (double)hidden), norm_eps)));
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t e = tid + i * kPrepThreads, d = rank * part + e;
        if (e < part) x_out[d] = __bfloat162float(__float2bfloat16_rn(__fmul_rn(__ldcg(norm_weight + d), __fmul_rn(red[i], rs))));
    }
}

// The largest dynamic shared memory a kernel may ask for on the current device (0: could not be set).
size_t smem_limit_of(const void *fn, size_t (&limit)[64]) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!limit[dev]) {
        cudaFuncAttributes fa;
        int optin = 0;
        if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
            return 0;
        const size_t most = (size_t)optin - fa.sharedSizeBytes;
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) return 0;
        limit[dev] = most;
    }
    return limit[dev];
}
size_t head_smem_limit() {
    static size_t limit[64] = {};
    return smem_limit_of((const void *)k_head_mma, limit);
}
template <bool kShared>
size_t few_smem_limit() {
    static size_t limit[64] = {};
    return smem_limit_of((const void *)k_head_mma_few<kShared>, limit);
}

}  // namespace

cudaError_t launch_head_logits(cudaStream_t st, int sm_count, const float *x, uint32_t n_tokens, const uint16_t *w, uint32_t n_rows,
                               uint32_t hidden, float *out, uint32_t out_stride) {
    // the tensor-core kernel: phases of K in whole groups of steps per half row, as few as keep the parts small;
    // sizes that have none take the register kernel
    // (a row's bits do not depend on how many rows a call has: a vocabulary may be dealt over ranks in shards of any size.
    // They do depend on the number of tokens, which sets the phases and, for some hidden sizes, the kernel.)
    for (uint32_t phases = 1; phases <= 8u; phases *= 2u) {
        const size_t parts = 3u * (size_t)n_tokens * (hidden / phases * 2u + kHeadPad);
        const size_t smem = parts + (phases > 1u ? kHeadTiles * 1024u : 0u);
        if (hidden % (256u * phases) != 0u || smem > head_smem_limit()) continue;
        if (parts > kHeadPartBytes && hidden % (512u * phases) == 0u && phases < 8u) continue;
        const uint32_t tiles = (n_rows + 15u) / 16u;
        if (tiles <= 2u * (uint32_t)sm_count) {
            const size_t sums = (size_t)hidden * 8u, shared = 3u * (size_t)n_tokens * (hidden * 2u + kHeadPad);
            const size_t most = few_smem_limit<true>();
            auto few = [&](auto kernel, uint32_t warps, uint32_t wide, size_t bytes) {
                const uint32_t per_cta = warps / wide, resident = 16u / warps;
                return launch_dependent(kernel, dim3((tiles + per_cta - 1u) / per_cta), dim3(warps * 32u), bytes, st, 0u, resident * (bytes + 1024u),
                                        x, w, out, n_rows, hidden, out_stride, n_tokens, phases, wide);
            };
            const bool alone = tiles <= (uint32_t)sm_count;
            // 4000 rows, us: 2048 x one token in CTAs of one tile 6.2, of two 6.7; 1024 x six 5.8 and 5.3; 4096 x five of two 14.5,
            // split in registers 20.3; 7168 x two in two rounds of one tile 22.6, of two (198 KB) 27.1
            if (!alone && n_tokens * hidden <= kFewSmallParts && sums + shared <= most) return few(k_head_mma_few<true>, 8u, 8u, sums + shared);
            if (!alone && 2u * sums + shared <= std::min(kFewTwoBytes, most)) return few(k_head_mma_few<true>, 16u, 8u, 2u * sums + shared);
            // (two rounds: 7168 x three 26.6, in registers 32.6; 4096 x six 21.3 and 20.3)
            if ((alone || n_tokens <= 4u) && sums + shared <= std::min(kFewOneBytes, most))
                return few(k_head_mma_few<true>, 16u, 16u, sums + shared);
            if (sums <= few_smem_limit<false>()) return few(k_head_mma_few<false>, alone ? 16u : 8u, alone ? 16u : 8u, sums);
        }
        const uint32_t ctas = tiles < (uint32_t)sm_count ? tiles : (uint32_t)sm_count;
        // (the division of the SM: 129280 x 4096 one token behind the layer kernel 296 us without it, 166 with it)
        return launch_dependent(k_head_mma, dim3(ctas), dim3(kHeadThreads), smem, st, 0u, smem + sizeof(double) * kHeadPairs * 256u + 1024u, x, w,
                                out, n_rows, hidden, out_stride, n_tokens, phases);
    }
    const uint32_t blocks = std::min((n_rows + 7u) / 8u, (uint32_t)sm_count * 8u);
    switch (n_tokens) {
    case 1: k_head_logits<1><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    case 2: k_head_logits<2><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    case 3: k_head_logits<3><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    case 4: k_head_logits<4><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    case 5: k_head_logits<5><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    case 6: k_head_logits<6><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    case 7: k_head_logits<7><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    default: k_head_logits<8><<<blocks, 256, 0, st>>>(x, w, out, n_rows, hidden, out_stride); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_greedy_argmax(cudaStream_t st, const float *logits, uint32_t vocab, int64_t *result) {
    // asked once per device
    static bool allowed[64] = {};
    static uint32_t size[64] = {};
    int dev = -1;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return e != cudaSuccess ? e : cudaErrorInvalidDevice;
    if (!size[dev])
        size[dev] = cluster_that_fits([&](uint32_t n) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = n;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(n);
            cfg.blockDim = dim3(kArgmaxThreads);
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int fit = 0;
            return launch_status(allow_wide_clusters(k_greedy_argmax, allowed)) == cudaSuccess &&
                   launch_status(cudaOccupancyMaxActiveClusters(&fit, k_greedy_argmax, &cfg)) == cudaSuccess && fit > 0;
        });
    return launch_pdl(k_greedy_argmax, dim3(size[dev]), dim3(kArgmaxThreads), 0, st, size[dev], logits, vocab, result);
}

cudaError_t launch_head_prep(cudaStream_t st, const uint16_t *state, const float *fn, const float *scale, const float *base,
                             const float *norm_weight, uint32_t hidden, float norm_eps, float hc_eps, float *x_out) {
    return launch_pdl(k_head_prep, dim3(kPrepCluster), dim3(kPrepThreads), 0, st, kPrepCluster, state, fn, scale, base, norm_weight,
                      hidden, norm_eps, hc_eps, x_out);
}

}  // namespace s14
