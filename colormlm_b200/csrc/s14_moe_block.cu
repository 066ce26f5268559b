// The MoE layer of a BLOCK of tokens (a verify block of up to 8 tokens, a prefill of hundreds) on
// the fifth-generation tensor cores, with the tokens grouped by expert so that an expert's page is
// streamed once for all the tokens routed to it.  Semantics: the reference's per-token layer loop
// (examples/s14_vulkan_numeric.rs:929-947) applied to every token of the block, which is all the
// reference's own prefill does (ssd_inference/src/forward.rs:544-549 walks the tokens one by one).
//
// The contraction is the one of the one-token layer kernel (s14_moe_umma.cu), widened along N:
// tcgen05.mma kind::mxf4.block_scale with A = 128 weight rows x 64 K-elements of page bytes as they
// are, and B = the sixteen balanced base-8 digit rows of EVERY token of a chunk (up to twelve tokens
// that share the expert: N = 16 * tokens; official arithmetic: six rows each, up to thirty-two tokens).
// Accumulator columns 16 t .. 16 t + 15 hold the digit shares of token t's dot products; added without loss and
// rounded once they give the dot product rounded to F32, so every token's result has the bits that the one-token kernel
// and the double-accumulating CPU restatement give for that token alone, up to ties closer than a sum in double resolves.
//
// Six launches per layer, all plain stream order (the routed calls run the router's two launches first):
//   k_block_digits   x [T, hidden] -> digit tiles (2 KB per token and 256 elements) + block exponents
//   k_block_group    routes [T, top_k] -> chunks (expert page, tokens that share it); an item index decodes to
//                    (chunk, pair of slices or row tiles) from the chunk records
//   k_block_pair     up items (chunk, two slices of 64 intermediate elements): w1 | w3 units x the chunk's token
//                    tiles; epilogue: limited SwiGLU, the hidden values of every (token, route) pair as F32
//   k_block_digits   their digit tiles (laid out by the up epilogue itself they tripled its time)
//   k_block_pair     down items (chunk, two tiles of 128 rows of w2) x the pairs' digit tiles -> the
//                    pairs' expert outputs [pair, hidden] (expert parallel: into every rank's pair buffer)
//   k_block_mix      per token the ordered mix: routes in order, shared expert last (expert parallel: after
//                    every rank's rows have arrived)
// Items are dealt round robin to the pairs of CTAs (s14_moe_pair.cu), the chunks of one expert next to each
// other, so that the second and later chunks of an expert find its units in the L2.
// With the official expert arithmetic
// (fast16/research/polaris_meridian_v1/s14_first_real_token/executor.py:712-743) the same contractions run on
// quantised inputs: k_block_digits_official quantises per 128 elements to E4M3FN values (which the digit rows hold
// exactly), the up epilogue leaves BF16 gate and up projections, the second digits launch makes the hidden values of them
// (SwiGLU, times the route's weight, BF16), the down epilogue
// and the mix round to BF16.
#include "s14_moe_block.cuh"

namespace s14 {

namespace {

// A chunk's B operand is made of groups of sixteen digit rows: one token each; in the official arithmetic,
// whose values need six digit rows, the tokens' rows follow one another.  Most groups of a chunk:
constexpr uint32_t kGrpSmall = 2;    // blocks of up to twelve tokens (of twelve 6 and 12 are 2 and 4 % faster at the size below, and not taken)
constexpr uint32_t kGrpSparse = 6;
constexpr uint32_t kGrpDense = 12;
// F32, us with 2 / 6 / 12 (256 experts of 4096 x 2048 unless said; 4 and 8 lie in between): 1 token 41.6 / 43.7 / 45.2, 4 71.9 / 75.9 / 76.2,
// 8 109.2 / 108.7 / 110.1, 12 141.5 / 138.6 / 136.4, 13 149.5 / 147.1 / 145.3, 32 248 / 236.6 / 234.8, 64 349 / 293.7 / 288.4, 128 576 / 388 / 362,
// 370 1425 / 761 / 623, 1000 3619 / 1703 / 1319.  With 6 / 12: 20 over 16 of 1024 x 512 31.1 / 34.8, 20 over 64 of 2048 x 1024 52.5 / 55.2,
// 100 over 64 of 1024 x 512 56.9 / 58.7, 60 over 128 of 1024 x 512 47.0 / 51.2, 200 over 64 of 512 x 512 68.5 / 68.0, 50 over 128 of 2048 x 1024
// 81.7 / 79.8, 370 over 256 of 1024 x 512 129.0 / 125.5, 45 over 192 of 2048 x 1536 118.8 / 117.2, 100 over 64 of 2048 x 1024 93.2 / 87.8.  So: the
// kernels for twelve pass over an expert less often, but need the registers in which the next launch's CTAs would be set up, some three
// microseconds for the call; they pay from 2^29 pairs x hidden x inter on (a page below 2^19 counted as that: an item's fixed part;
// 200 over 64 of 512 x 512 by the product alone 69.7, so 67.6), where experts have a pair on average at least
// (13 and 32 tokens over 256 lie below it, for 1 %).
constexpr uint64_t kDenseWork = 1ull << 29, kDensePage = 1ull << 19;
// Official arithmetic, 6 / 12 groups (16 / 32 tokens): the same, from 2^30 on.  60 over 16 of 512 x 512 30.2 / 32.6, 20 over 64 of 2048 x 1024 53.8 / 55.5,
// 40 over 32 of it 47.6 / 48.9, 150 over 128 of 1024 x 512 56.1 / 58.1, 45 over 192 of 2048 x 1536 116.4 / 116.2, 80 over 64 of 2048 x 1024 70.0 / 69.8,
// 370 over 256 of 1024 x 512 83.1 / 83.6, 200 over 256 of 4096 x 2048 386 / 380, 300 over 64 of 2048 x 1024 108.6 / 99.4.
constexpr uint64_t kDenseOfficial = 1ull << 30;
static_assert(kBlockNt == kGrpDense * 8u / 6u * 2u, "a chunk record holds the tokens of the official arithmetic's chunks");

// The nearest E4M3FN values (ties to even) of two numbers of magnitude 448 at most, as F32 values: the conversion there and back.
// (Rounded by shifts of the exponent, with a branch for the subnormals, the second digits launch of 1000 tokens at 4096 x 2048 took
// 70 us and takes 56, the first 24 and 18.)
__device__ __forceinline__ float2 e4m3fn_round2(float a, float b) {
    uint16_t p;
    uint32_t h;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(p) : "f"(b), "f"(a));   // (the second operand is the lower byte)
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"(p));
    return __half22float2(*reinterpret_cast<const __half2 *>(&h));
}

// The digit tiles and block exponents of n vectors of K elements, a CTA per vector.  In the official arithmetic the
// vector is first quantised as the official linears quantise their input
// (l42_real_reference/l42_reference.py:389-403): per 128 elements amax = max(|x|, 1e-4), scale =
// 2^ceil(log2(amax / 448)) (F32 quotient, the logarithm taken in double and rounded to F32), x / scale
// clipped to +-448, rounded to E4M3FN, times the scale.  The quantised values are F32 values with four
// significant bits: within a scale block, whose largest magnitude is below 2^E, all are multiples of
// 2^(E-18) (the smallest E4M3FN step is 2^-18 of the range's end), so six digit rows hold them (digit6_code_bytes) and a
// chunk has room for 32 tokens where sixteen rows each leave room for twelve.  The rows of a chunk's tokens follow one another without
// a gap, so a token's place in the 128-byte swizzle, which goes by the row modulo eight, depends on its place in its CTA's half of
// the chunk (6 i mod 8: 0, 6, 4, 2 in turn).  A tile of 768 bytes therefore exists in four forms: all four of a token's (it is in
// seven chunks), the one that its place takes of a pair's (`slots`, from k_block_group).  With eight rows, a tile of 1 KB, and 24 tokens to
// a chunk 1000 tokens made 408 chunks, so 334.
// With `slots` the vectors are the pairs' gate and up projections and the hidden values are made of them here, element by element over
// the whole chip: in the up kernel's epilogue they stood in the way of the next item (see s14_moe_pair.cu).
__global__ void __launch_bounds__(512)
k_block_digits_official(const float *__restrict__ x, uint32_t K, uint8_t *__restrict__ dig, uint8_t *__restrict__ exps, uint32_t early,
                        const uint8_t *__restrict__ slots, const float *__restrict__ weights, uint32_t top_k) {
    const uint32_t v = blockIdx.x, g = threadIdx.x;   // K / 8 threads: whole warps, K is a multiple of 256
    // early: the launch in front neither writes x nor uses what is written here (it picks the routes), and whatever is in front
    // of it is complete when this kernel starts, because it lets this one start behind its own wait (a launch that triggers in
    // front of it would make this a race); so the work runs beside it, and the wait for it comes last
    if (!early) dependency_wait();
    float xs[8];
    uint32_t place = 0u;   // the form that the pair's digit tile takes
    if (slots) {
        place = __ldcg(slots + v) & 3u;
        // the hidden values of pair v from its gates and up projections (s14_first_real_token/executor.py:712-743): the limited SwiGLU
        // in F32, times the route's weight (not for the shared expert), rounded to BF16
        const uint32_t tok = v / kPairsPerToken, pos = v - tok * kPairsPerToken;
        const uint16_t *const row = reinterpret_cast<const uint16_t *>(x) + (size_t)v * 2u * K;
        const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(row) + g), r = __ldcg(reinterpret_cast<const uint4 *>(row + K) + g);
        const float wt = pos < top_k ? __ldcg(weights + tok * top_k + pos) : 1.0f;
        const uint32_t gw[4] = {q.x, q.y, q.z, q.w}, uw[4] = {r.x, r.y, r.z, r.w};
        bool sure[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            sure[i] = swiglu_quick(__uint_as_float((i & 1) ? gw[i >> 1] & 0xFFFF0000u : gw[i >> 1] << 16),
                                   __uint_as_float((i & 1) ? uw[i >> 1] & 0xFFFF0000u : uw[i >> 1] << 16), wt, xs[i]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!sure[i])
                xs[i] = bf16_round(__fmul_rn(swiglu_once(__uint_as_float((i & 1) ? gw[i >> 1] & 0xFFFF0000u : gw[i >> 1] << 16),
                                                         __uint_as_float((i & 1) ? uw[i >> 1] & 0xFFFF0000u : uw[i >> 1] << 16)), wt));
    } else {
        const float4 p0 = __ldcg(reinterpret_cast<const float4 *>(x + (size_t)v * K) + 2u * g);
        const float4 p1 = __ldcg(reinterpret_cast<const float4 *>(x + (size_t)v * K) + 2u * g + 1u);
        xs[0] = p0.x, xs[1] = p0.y, xs[2] = p0.z, xs[3] = p0.w, xs[4] = p1.x, xs[5] = p1.y, xs[6] = p1.z, xs[7] = p1.w;
    }
    // a group of 128 elements is sixteen neighbouring threads
    float am = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) am = fmaxf(am, fabsf(xs[i]));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    am = fmaxf(am, 1e-4f);
    // (where the quotient is well above a power of two the logarithm's F32 value lies between the two integers)
    const float quot = __fdiv_rn(am, 448.0f);
    const uint32_t bits = __float_as_uint(quot);   // (normal: am is at least 1e-4)
    int e = (int)(bits >> 23) - 126;
    if ((bits & 0x7FFFFFu) < 128u) e = (int)ceilf((float)log2((double)quot));
    e = e < -126 ? -126 : (e > 126 ? 126 : e);
    const float scale = __uint_as_float((uint32_t)(127 + e) << 23), inv = __uint_as_float((uint32_t)(127 - e) << 23);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float2 q = e4m3fn_round2(fminf(fmaxf(__fmul_rn(xs[i], inv), -448.0f), 448.0f), fminf(fmaxf(__fmul_rn(xs[i + 1], inv), -448.0f), 448.0f));
        xs[i] = __fmul_rn(q.x, scale);
        xs[i + 1] = __fmul_rn(q.y, scale);
    }
    uint32_t words[6];
    digits6_of8(xs, g, words, exps + (size_t)v * (K >> 5));
    const uint32_t kb = g >> 2, forms = slots ? 1u : 4u;
    for (uint32_t i = 0; i < forms; ++i) {
        const uint32_t form = slots ? place : i;
        uint8_t *const chunk = dig + ((size_t)(v * forms + i) * (K >> 8) + (kb >> 3)) * 768u + (g & 3u) * 4u;
#pragma unroll
        for (uint32_t j = 0; j < 6; ++j)
            *reinterpret_cast<uint32_t *>(chunk + j * 128u + (((kb & 7u) ^ ((6u * form + j) & 7u)) << 4)) = words[j];
    }
    if (early) dependency_wait();
}

// F32 arithmetic.  A CTA takes vectors blockIdx.x, + gridDim.x, ... with the next one's loads in flight: with a CTA per vector, as above, a launch
// is its CTAs' latency - being started, a trip to the L2, code that is new to the SM, shuffles - times the rounds of what fits beside one
// another (45 tokens of 2048 x 1536 120.2 us for the call, so 118.8, 100 of 2048 x 1024 89.4 and 87.9).  The official form gains nothing by it:
// there the instructions count, and the loop's registers cost more (8 tokens 106.0 -> 108.5).  Kept to 40 registers (64 here) this one spills
// and gains nothing.
constexpr uint32_t kDigitThreads = 1024;   // of an SM, in CTAs of K / 8 (1536 and 2048 are as fast)
__global__ void __launch_bounds__(512)
k_block_digits(const float *__restrict__ x, uint32_t n, uint32_t K, uint8_t *__restrict__ dig, uint8_t *__restrict__ exps, uint32_t early) {
    const uint32_t g = threadIdx.x;   // K / 8 threads: whole warps, K is a multiple of 256
    if (!early) dependency_wait();   // (early: as above)
    auto row = [&](uint32_t v) { return reinterpret_cast<const float4 *>(x + (size_t)v * K) + 2u * g; };
    float4 p0 = __ldcg(row(blockIdx.x)), p1 = __ldcg(row(blockIdx.x) + 1);
#pragma unroll 1
    for (uint32_t v = blockIdx.x; v < n; v += gridDim.x) {
        const float xs[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
        if (v + gridDim.x < n) {
            p0 = __ldcg(row(v + gridDim.x));
            p1 = __ldcg(row(v + gridDim.x) + 1);
        }
        digits_of8(xs, g, dig + (size_t)v * (K >> 8) * 2048u, exps + (size_t)v * (K >> 5));
    }
    if (early) dependency_wait();
}

// Groups the block's (token, route) pairs by expert.  Group 0 is the shared expert (every token, mix
// position 6), group 1 + e the routed expert e; a group's members are cut into chunks of nt_cap (the
// shared expert's in token order, a routed expert's in the order its members arrive: every pair's
// result depends on that pair alone, so the order changes no bit of the output).  ids: [T, top_k]
// expert ids, negative = no route.  The page of a routed group is page_table[e], or, with per-route
// pages, the page of one of its members.  counts: [0] chunks, [1], [2] that times S, RT, [3] kBlockBadId if
// an id was out of range (then no chunk is made), else 0.  One CTA of 1024 threads.
__global__ void __launch_bounds__(1024)
k_block_group(const int32_t *__restrict__ ids, const uint8_t *const *__restrict__ pages,
              const uint8_t *const *__restrict__ page_table, const uint8_t *shared_page, uint32_t T, uint32_t top_k,
              uint32_t n_experts, uint32_t S, uint32_t RT, uint32_t nt_cap, uint32_t even, BlockChunk *__restrict__ chunks,
              uint32_t *__restrict__ counts, uint32_t ep_rank, uint32_t ep_world, uint32_t shared_by_token, uint8_t *__restrict__ slots) {
    constexpr uint32_t kG = S14_N_ROUTED_EXPERTS + 1;
    __shared__ uint32_t cnt[kG], fill[kG], chunk0[kG + 1], size[kG];
    __shared__ unsigned long long gpage[kG];
    __shared__ uint32_t bad;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, G = n_experts + 1u, n = T * top_k;
    dependency_wait();
    if (tid < kG) {
        cnt[tid] = 0u;
        fill[tid] = 0u;
        gpage[tid] = tid == 0u ? (unsigned long long)shared_page
                               : ((page_table && tid < G) ? __ldcg(reinterpret_cast<const unsigned long long *>(page_table + tid - 1u)) : 0ull);
    }
    if (tid == 0) bad = 0u;
    __syncthreads();
    // the thread's pairs i = tid, tid + 1024, ...; an id that makes no pair here is -1
    int32_t mine_id[S14_EXPERTS_PER_TOKEN];   // (up to 1024 tokens)
#pragma unroll
    for (uint32_t k = 0; k < S14_EXPERTS_PER_TOKEN; ++k) mine_id[k] = tid + k * 1024u < n ? __ldcg(ids + tid + k * 1024u) : -1;
#pragma unroll
    for (uint32_t k = 0; k < S14_EXPERTS_PER_TOKEN; ++k) {
        if (mine_id[k] >= (int32_t)n_experts) bad = 1u;
        if (mine_id[k] >= (int32_t)n_experts || mine_id[k] < 0 || (uint32_t)mine_id[k] % ep_world != ep_rank) mine_id[k] = -1;
        else atomicAdd(&cnt[1 + mine_id[k]], 1u);  // expert parallel: the experts this rank owns
    }
    // the shared expert's members: every token; expert parallel with the shared page on every rank: the tokens
    // t with t mod world == rank (its work is a fifth of a large block's: on one rank it would bound the scaling)
    const uint32_t sh_step = shared_by_token ? ep_world : 1u, sh_first = shared_by_token ? ep_rank : 0u;
    if (tid == 0 && shared_page) cnt[0] = T > sh_first ? (T - sh_first + sh_step - 1u) / sh_step : 0u;
    __syncthreads();
    if (tid < G) {
        // the chunks of an expert of like size, in whole multiples of `even`: what one of them costs goes with its size, and
        // neighbouring items - an expert's chunks in turn - go to neighbouring CTAs (full chunks and a rest: 370 tokens 730
        // us, so 705; 1000 official ones 1265 and 1165)
        const uint32_t n_ch = (cnt[tid] + nt_cap - 1u) / nt_cap;
        chunk0[tid] = n_ch;
        size[tid] = n_ch <= 1u ? nt_cap : ((cnt[tid] + n_ch * even - 1u) / (n_ch * even)) * even;
    }
    __syncthreads();
    if (tid < 32u) {
        // exclusive scan of the groups' chunk counts: nine groups per lane
        constexpr uint32_t kPer = (kG + 31u) / 32u;
        uint32_t mine = 0;
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t g = lane * kPer + k;
            if (g < G) mine += chunk0[g];
        }
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += v;
        }
        uint32_t c = incl - mine;
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t g = lane * kPer + k;
            if (g < G) {
                const uint32_t n_ch = chunk0[g];
                chunk0[g] = c;
                c += n_ch;
            }
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (lane == 0) {
            chunk0[G] = total;
            const uint32_t c_all = bad ? 0u : total;  // with a bad id the contraction kernels find no item, the mix writes nothing
            counts[0] = c_all;
            counts[1] = c_all * S;
            counts[2] = c_all * RT;
            counts[3] = bad ? kBlockBadId : 0u;
        }
    }
    __syncthreads();
    if (bad) return;
    // member k of group g: its chunk's record; official arithmetic: also the form its digit tile takes, which goes by the place in
    // the half of the chunk that a CTA of the pair brings
    auto place = [&](uint32_t g, uint32_t k, uint32_t pair) {
        const uint32_t c = k / size[g], t = k - c * size[g];
        chunks[chunk0[g] + c].pair[t] = pair;
        if (slots) {
            const uint32_t nt = min(size[g], cnt[g] - c * size[g]), half = (nt + 1u) >> 1;
            slots[pair] = (uint8_t)((t < half ? t : t - half) & 3u);
        }
    };
#pragma unroll
    for (uint32_t kk = 0; kk < S14_EXPERTS_PER_TOKEN; ++kk) {
        if (mine_id[kk] < 0) continue;
        const uint32_t i = tid + kk * 1024u, g = 1u + (uint32_t)mine_id[kk], t = i / top_k, m = i - t * top_k;
        const uint32_t k = atomicAdd(&fill[g], 1u);
        if (k == 0u && !page_table) gpage[g] = __ldcg(reinterpret_cast<const unsigned long long *>(pages + i));
        place(g, k, t * kPairsPerToken + m);
    }
    if (shared_page) {
        for (uint32_t k = tid; sh_first + k * sh_step < T; k += blockDim.x) {
            const uint32_t t = sh_first + k * sh_step;
            place(0u, k, t * kPairsPerToken + S14_EXPERTS_PER_TOKEN);
        }
    }
    __syncthreads();
    const uint32_t total = chunk0[G];
    for (uint32_t c = tid; c < total; c += blockDim.x) {
        // the chunk's group: the last g with chunk0[g] <= c
        uint32_t lo = 0, hi = G;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (chunk0[mid] <= c) lo = mid;
            else hi = mid;
        }
        const uint32_t g = lo, c0 = chunk0[g], nch = chunk0[g + 1u] - c0;
        BlockChunk *ch = chunks + c;
        ch->page = reinterpret_cast<const uint8_t *>(gpage[g]);
        ch->nt = c + 1u < c0 + nch ? size[g] : cnt[g] - (c - c0) * size[g];
        ch->c0 = c0;
        ch->nch = nch;
    }
}

// y[t, n]: the ordered mix of token t (examples/s14_vulkan_numeric.rs:936-946): acc = 0; acc += w * d
// over the routes in order; acc += d of the shared expert.  With `residual` the layer's input is added
// (y = x + acc, what a layer of a stack hands to the next); y may be x.  16 bytes of each
// row per thread, the seven rows' loads in flight together (one value per thread,
// row after row: 64 us for 1000 tokens of 4096, now 28).  Compiled for aligned buffers and for others: with both forms in one
// kernel the code that every warp fetches once was longer (a block of 45 tokens 148.1 us, so 147.6).
// The official arithmetic's rows are BF16 values and are stored as such: 115 MB written and read for 1000 tokens, stored as F32, now 57
// (the call, with its down kernel, 973 us power limited, now 956).  CTAs of 128 threads: 256 took 0.3 us more for a block of 8 tokens.
// The launch behind may start when the CTAs here exit, not earlier: all of them are resident at once, and while they are, the
// CTAs of the next block's router scores, which fill the FP64 pipe of an SM (where it takes all of them in double), find room on few SMs only, several on one.  Blocks one
// after another, 4096 x 2048, 64 experts, us: 200 tokens 336, so 319, official 221 and 210; 2048 x 1024, 370 tokens 212 and 203;
// 8 and 45 tokens the same.
template <bool vec, bool kOff>
__global__ void __launch_bounds__(128)
k_block_mix(const float *__restrict__ d, const int32_t *__restrict__ ids, const float *__restrict__ weights,
            uint32_t top_k, int has_shared, float *y, uint32_t hidden, const uint32_t *__restrict__ counts,
            const float *x, uint32_t residual, const unsigned long long *flags, uint32_t ep_rank, uint32_t ep_world, uint32_t ep_call,
            uint32_t wait_limit, uint32_t *status) {
    constexpr uint32_t kPer = kOff ? 8u : 4u;
    const uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) * kPer, t = blockIdx.y;   // hidden is a multiple of eight
    cudaGridDependencySynchronize();
    const uint32_t why = __ldcg(counts + 3);
    if (flags) {
        // expert parallel, exchange inside the kernels: every rank's rows of this call are in this rank's buffer
        // when its flag carries the call's number (bounded wait: about a microsecond per poll).  A rank that gave up has not
        // published its own; it waits for the others all the same, because that is what tells it that they have read
        // the buffer its next call but one writes.
        __shared__ int s_ok;
        if (threadIdx.x == 0) {
            int ok = 1;
            for (uint32_t p = 0; p < ep_world && ok; ++p) {
                if (p == ep_rank && (why & kBlockGaveUp)) continue;
                uint32_t tries = 0;
                for (;;) {
                    unsigned long long v;
                    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(flags + p) : "memory");
                    if (v >= (unsigned long long)ep_call) break;
                    if (++tries > wait_limit) {
                        ok = 0;
                        atomicExch(status, 0x5508u);
                        break;
                    }
                    __nanosleep(1000);
                }
            }
            s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) return;
    }
    if (n >= hidden) return;
    const size_t at = (size_t)t * kPairsPerToken * hidden + n;
    // (a caller's buffers may lie on any 4-byte boundary)
    auto load = [&](const float *p, float(&r)[kPer]) {
#pragma unroll
        for (uint32_t i = 0; i < kPer; i += 4u) {
            if constexpr (vec) {
                const float4 q = __ldcg(reinterpret_cast<const float4 *>(p + i));
                r[i] = q.x, r[i + 1u] = q.y, r[i + 2u] = q.z, r[i + 3u] = q.w;
            } else {
                r[i] = __ldcg(p + i), r[i + 1u] = __ldcg(p + i + 1u), r[i + 2u] = __ldcg(p + i + 2u), r[i + 3u] = __ldcg(p + i + 3u);
            }
        }
    };
    auto load_row = [&](uint32_t m, float(&r)[kPer]) {
        if constexpr (kOff) {
            const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(d) + at + (size_t)m * hidden));
            const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (uint32_t i = 0; i < kPer; ++i) r[i] = __uint_as_float((i & 1u) ? qw[(i >> 1) & 3u] & 0xFFFF0000u : qw[(i >> 1) & 3u] << 16);
        } else {
            load(d + at + (size_t)m * hidden, r);
        }
    };
    // official arithmetic: the route's weight went into the expert's hidden values; the BF16 outputs are added
    // in F32 and the sum is rounded to BF16 (moe_branch, s14_first_real_token/executor.py:716-735)
    float row[S14_EXPERTS_PER_TOKEN + 1][kPer] = {}, in[kPer] = {};
    float w[S14_EXPERTS_PER_TOKEN];
    bool there[S14_EXPERTS_PER_TOKEN];
#pragma unroll
    for (uint32_t m = 0; m < S14_EXPERTS_PER_TOKEN; ++m) {
        // (a position without a route has a row of its own all the same, with whatever is left in it: the row's load need not
        // wait for the id)
        there[m] = m < top_k && __ldcg(ids + t * top_k + m) >= 0;
        w[m] = m < top_k ? __ldcg(weights + t * top_k + m) : 0.0f;
        if (m < top_k) load_row(m, row[m]);
    }
    constexpr uint32_t kSh = S14_EXPERTS_PER_TOKEN;
    if (has_shared) load_row(kSh, row[kSh]);
    if (residual) load(x + (size_t)t * hidden + n, in);
    if (why) return;   // (behind the loads, which need not wait for it)
    float out[kPer];
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
        float acc = 0.0f;
#pragma unroll
        for (uint32_t m = 0; m < S14_EXPERTS_PER_TOKEN; ++m)
            if (there[m]) acc = __fadd_rn(acc, kOff ? row[m][i] : __fmul_rn(w[m], row[m][i]));
        if (has_shared) acc = __fadd_rn(acc, row[kSh][i]);
        if (kOff) acc = bf16_round(acc);
        out[i] = residual ? __fadd_rn(in[i], acc) : acc;
    }
    float *yt = y + (size_t)t * hidden + n;
#pragma unroll
    for (uint32_t i = 0; i < kPer; i += 4u) {
        if constexpr (vec) *reinterpret_cast<float4 *>(yt + i) = make_float4(out[i], out[i + 1u], out[i + 2u], out[i + 3u]);
        else yt[i] = out[i], yt[i + 1u] = out[i + 1u], yt[i + 2u] = out[i + 2u], yt[i + 3u] = out[i + 3u];
    }
}

cudaError_t launch_mix(cudaStream_t st, const float *pairs, const int32_t *ids, const float *weights, uint32_t n_tokens, uint32_t top_k,
                       bool has_shared, const float *x, float *y, uint32_t hidden, const uint32_t *counts, bool residual,
                       const BlockEp *ep, uint32_t *status, bool official) {
    const uintptr_t where = (uintptr_t)pairs | (uintptr_t)y | (residual ? (uintptr_t)x : 0u);   // (official: `pairs` is the block's own)
    const uint32_t per_cta = official ? 1024u : 512u;
    const auto kernel = (where & 15u) ? (official ? k_block_mix<false, true> : k_block_mix<false, false>)
                                      : (official ? k_block_mix<true, true> : k_block_mix<true, false>);
    return launch_pdl(kernel, dim3((hidden + per_cta - 1u) / per_cta, n_tokens), dim3(128), 0, st, 0u, pairs, ids, weights, top_k,
                      has_shared ? 1 : 0, y, hidden, counts, x, residual ? 1u : 0u,
                      (const unsigned long long *)(ep ? ep->flags : nullptr), ep ? ep->rank : 0u, ep ? ep->world : 1u, ep ? ep->call : 0u,
                      ep ? ep->wait_limit : 0u, status);
}

}  // namespace

bool moe_block_ok(int sm_count, uint32_t hidden, uint32_t inter, uint32_t n_experts, uint32_t top_k) {
    if (sm_count <= 0 || n_experts == 0u || n_experts > S14_N_ROUTED_EXPERTS || top_k == 0u || top_k > S14_EXPERTS_PER_TOKEN)
        return false;
    if ((hidden & 511u) || (inter & 511u) || hidden < 512u || inter < 512u || hidden > 4096u || inter > 4096u) return false;
    return pair_dynamic_limit() >= 6u * (kStageA + kGrpDense / 2u * 2048u);
}

size_t moe_block_max_chunks(uint32_t max_tokens) {
    // no more chunks than pairs (chunks of one token)
    return (size_t)max_tokens * kPairsPerToken;
}

int launch_moe_block(cudaStream_t st, int sm_count, const BlockWork &w, const float *x, float *y, const int32_t *ids,
                     const float *weights, const uint8_t *const *pages, const uint8_t *const *page_table,
                     const uint8_t *shared_page, uint32_t n_tokens, uint32_t top_k, uint32_t n_experts, uint32_t hidden,
                     uint32_t inter, uint32_t *status, cudaError_t *err, bool residual, uint32_t ep_rank,
                     uint32_t ep_world, float *pairs_out, const BlockEp *ep, bool shared_by_token, bool official) {
    // How many groups a chunk may hold: a chunk's stage has room for all of them, so short chunks make the ring deeper, and
    // long ones pass over an expert's page less often (the shared expert's extra chunks come from the L2).
    *err = cudaErrorInvalidConfiguration;
    if (official && (ep || pairs_out)) return 0;   // the official arithmetic runs on one GPU
    if (n_tokens == 0u) return 0;
    const uint32_t tpg = official ? 2u : 1u;   // tokens per group of sixteen digit rows
    const bool small = n_tokens <= 12u;
    // (a group is sixteen operand rows: one token, official arithmetic six rows a token; half of a chunk's groups are one CTA's)
    const uint64_t pairs = (uint64_t)n_tokens * top_k;
    const bool dense = pairs >= n_experts && pairs * std::max((uint64_t)hidden * inter, kDensePage) >= (official ? kDenseOfficial : kDenseWork);
    const uint32_t groups = small ? kGrpSmall : (dense ? kGrpDense : kGrpSparse);
    const uint32_t S = inter >> 6, RT = hidden >> 7, counted = small ? 1u : 2u;   // slices, row tiles; as `counts` reports them
    const uint32_t cap = official ? groups * 8u / 6u * 2u : groups;   // tokens of a chunk: 4, 16, 32, or 2, 6, 12
    // The launches are programmatic dependents of one another: a kernel's blocks, barriers and tensor memory are
    // set up while the one before runs out, and every kernel but the first digits launch (see there) waits for it before it
    // reads or writes anything.
    auto digits = [&](const float *v, uint32_t n, uint32_t K, uint8_t *dig, uint8_t *exps, bool early) {
        if (*err != cudaSuccess) return;
        const uint32_t threads = K >> 3;
        if (official)
            *err = launch_pdl(k_block_digits_official, dim3(n), dim3(threads), 0, st, 0u, v, K, dig, exps, early ? 1u : 0u,
                              early ? (const uint8_t *)nullptr : (const uint8_t *)w.slots, weights, top_k);
        else
            *err = launch_pdl(k_block_digits, dim3(std::min(n, (uint32_t)sm_count * (kDigitThreads / threads))), dim3(threads), 0, st, 0u, v, n, K, dig,
                              exps, early ? 1u : 0u);
    };
    *err = cudaSuccess;
    // (in front of it: the router's launch, or the copies of the host's routes)
    digits(x, n_tokens, hidden, w.xdig, w.xexp, true);
    if (ep_world == 0u) ep_world = 1u;
    if (*err == cudaSuccess)
        *err = launch_pdl(k_block_group, dim3(1), dim3(1024), 0, st, 0u, ids, pages, page_table, shared_page, n_tokens, top_k, n_experts,
                          S / counted, RT / counted, cap, small ? 1u : 2u * tpg, w.chunks, w.counts, ep_rank, ep_world,
                          (shared_by_token && ep_world > 1u) ? 1u : 0u, official ? w.slots : (uint8_t *)nullptr);
    if (*err != cudaSuccess) return 1;
    if (pairs_out && !ep) {
        // expert parallel: the pairs of the experts this rank owns; the others stay zero for the sum over the ranks
        *err = cudaMemsetAsync(pairs_out, 0, (size_t)n_tokens * kPairsPerToken * hidden * sizeof(float), st);
        if (*err != cudaSuccess) return 2;
    }
    GemmArgs up = {}, down = {};
    up.chunks = down.chunks = w.chunks;
    up.n_chunks = down.n_chunks = w.counts;
    up.why = down.why = w.counts + 3;
    up.hidden = down.hidden = hidden;
    up.inter = down.inter = inter;
    up.dig = w.xdig;
    up.exps = w.xexp;
    up.hval = w.hval;
    up.hval16 = reinterpret_cast<uint16_t *>(w.hval);   // (as many bytes)
    down.dig = w.hdig;
    down.exps = w.hexp;
    down.out = pairs_out ? pairs_out : w.d;
    down.out16 = reinterpret_cast<uint16_t *>(w.d);     // (half of its bytes)
    if (ep) {
        // exchange inside the kernel: the owned pairs' rows into every rank's buffer of the call's parity
        for (uint32_t p = 0; p < ep->world; ++p) {
            down.out_peer[p] = ep->pairs_peer[p];
            down.flag_peer[p] = ep->flags_peer[p];
        }
        down.ep_counter = ep->counter;
        down.ep_world = ep->world;
        down.ep_rank = ep->rank;
        down.ep_call = ep->call;
    }
    // The up kernel leaves the pairs' hidden values, and a second digits launch (which also quantises them per 128
    // elements for the official arithmetic) lays out the rows of all pairs' slots (a slot without a route holds what an
    // earlier call left, perhaps in the other arithmetic, so any bits: its rows are copied into no chunk, and the mix skips it).
    *err = launch_pair_gemm(st, sm_count, false, official, up, groups / 2u, status);
    digits(w.hval, n_tokens * kPairsPerToken, inter, w.hdig, w.hexp, false);
    if (*err == cudaSuccess) *err = launch_pair_gemm(st, sm_count, true, official, down, groups / 2u, status);
    const int launches = 5;
    if (pairs_out || *err != cudaSuccess) return launches;
    *err = launch_mix(st, w.d, ids, weights, n_tokens, top_k, shared_page != nullptr, x, y, hidden, w.counts, residual, nullptr, status,
                      official);
    return launches + 1;
}

cudaError_t launch_block_mix(cudaStream_t st, const float *pairs, const int32_t *ids, const float *weights, uint32_t n_tokens,
                             uint32_t top_k, bool has_shared, const float *x, float *y, uint32_t hidden, const uint32_t *counts,
                             const BlockEp *ep, uint32_t *status) {
    return launch_mix(st, pairs, ids, weights, n_tokens, top_k, has_shared, x, y, hidden, counts, x != nullptr, ep, status, false);
}

}  // namespace s14
