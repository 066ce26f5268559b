// The contraction kernels of the grouped block path: a PAIR of CTAs (a cluster of two, the two SMs of a TPC) works on an
// item together, tcgen05.mma.cta_group::2.  What they compute is described in s14_moe_block.cu; per item it is a chunk
// of up to twelve tokens of sixteen digit rows (official arithmetic: 32 tokens of six) times 256 rows of an expert:
// two slices of the up projection or two row tiles of w2.
//
// Each CTA brings its own 128 rows of the page (a unit of 17 KB per step of 256 k) and HALF of the chunk's digit tiles; the
// pair's tensor cores read both halves, so a step costs an SM 17 + 12 KB instead of 17 + 24, one MMA does N = 192
// columns, and the accumulators of one row tile are all an SM holds: 192 columns, which leaves room for a second set.  So an
// item's accumulators are read, added and finished while the next item's MMAs run.  The kernel before this one
// (two row tiles and twelve tokens per SM, one set of accumulators, stages of 58 KB in a ring of three, N = 96) waited for the
// epilogue between two items and for a stage's way through the memory.  370 tokens, 4096 x 2048, up / down kernel: 507 / 294
// us, then 393 / 212; 1000 tokens of the official arithmetic 1200 / 444, then 577 / 311 and 424 / 227 (steps since: see below).  Small blocks, which took one row tile
// and two tokens per SM with stages of 21 KB in a ring of eight and laid out the hidden values' digit rows in the up epilogue:
// 8 tokens 117 us for the call, now 109.  (Official blocks of two to eight tokens of smaller layers gained nothing: 4 tokens of
// 2048 x 1536 49 us for the call, now 52.)
//
// What bounds it: a step is four MMAs and two copies of the unit's scale codes.  The MMAs of a full chunk take 384 cycles (270 for the
// chunks 370 tokens have on average), a step takes 520 at full clock: an SM takes in some 50 bytes a clock then, 26 KB a step, and rings of
// six stages and of seven are as fast, so it is the stream from the L2 that the rest waits for.  With the digit rows' codes laid out in
// shared memory and copied too (six copies in the issuing warp's round, which looked at a stage only when it wanted it) a step took 600:
// 370 tokens 675 us, so 635, 1000 official ones 820 and 806 (bursts; 785 and 725, 960 and 920 power limited).  Codes written by their warps
// for one stage at a time, the unit's among them, took 900 a step: a wait costs 100 cycles, over or not.
// Beside the steps the epilogue.  Cycles of an item at full clock,
// waiting for accumulators / adding their columns / the rest: 370 tokens up 3450 / 2950 / 1900, down 900 / 3050 / 380; official ones,
// with exact sums and the SwiGLU here, up 950 / 3900 / 5500, down 540 / 4150 / 1550: there the epilogue was what bounded both
// kernels (1000 tokens 1036 us, without an epilogue 825, without three of four MMAs 1003, without the tiles' copies 1067), and fewer steps
// (six digit rows for eight) alone gave nothing.  So BF16 sums are settled by plain additions and a bound where that is possible, four
// pairs of tokens side by side, and the SwiGLU is k_block_digits_official's work: 1161 us power limited, now 992.  (The like for F32 sums, one part of the
// three exact: 370 tokens nothing, 8 tokens 115 -> 120.)  Sustained, the
// 1000 W limit lowers the clock to 1.4-1.6 GHz: 0.8 J per block of 370 tokens, 0.28 of them in the MMAs.  A pair with more items
// than a batch of records drains its pipeline between two batches (1000 official tokens: 73 items, batches of 56).
//
// Roles in a CTA of 544 threads: warps 0-7 epilogue (two warpgroups, each with every lane of tensor memory, the even and
// the odd tokens of the chunk, or its halves); warps 8-11 copy (the ring slots in turn, a lane per copy: a round of waiting, arming
// and seven copies takes 0.3-0.5 us); warps 12-15, one per quadrant of tensor memory, write the scale codes of the digit rows there, two
// stages at a time and up to six ahead; warp 16 of the first CTA issues the pair's tensor operations, that of the second
// passes on that its stage is there.  A stage's barriers: `full` in each CTA (unit and tiles; in the first CTA also that the second's
// are there), `done` in each (the commit arrives at both); `rows` in the first CTA says that both CTAs' codes of a pair of stages are
// written.  Every wait is bounded; one that runs out raises the CTA's abort flag, the status word is set, the CTA
// waits for its copies and the pair's tensor work, and the pair meets at a cluster barrier before tensor memory is freed.
#include "s14_moe_block.cuh"

namespace s14 {

namespace {

constexpr uint32_t kPGroups = 12, kPCols = 16u * kPGroups;   // accumulator columns of a chunk
constexpr uint32_t kPEpi = 256, kPProds = 4, kPProdWarp0 = kPEpi / 32u, kPCodes = 4, kPCodeWarp0 = kPProdWarp0 + kPProds;
constexpr uint32_t kPMmaWarp = kPCodeWarp0 + kPCodes, kPThreads = (kPMmaWarp + 1u) * 32u;
static_assert(kPCodeWarp0 % 4u == 0u, "a warp reaches the lanes of tensor memory that its number modulo four says");
// Most stages of the ring: with more of them small blocks ask the memory for more than it has, and some SMs get less than others (8 tokens,
// 4096 x 2048, rings of 6 / 7 / 8 / 9 / 11: 110.4 / 109.6 / 109.4 / 110.0 / 115 us, 45 tokens of 2048 x 1536 122.1 / 121.3 / 121.2 / 123.0).
constexpr uint32_t kPRingMax = 8;
// tensor memory columns: two sets of accumulators, the digit rows' scale codes of six stages, the units' of four
constexpr uint32_t kPRowSets = 3, kPRowCols = 32;    // a set: two stages, [2][2][8]
constexpr uint32_t kPUnitSets = 4, kPUnitCols = 8;   // [2][4]
constexpr uint32_t kPColRows = 2u * kPCols, kPColUnits = kPColRows + kPRowSets * kPRowCols;
static_assert(kPColUnits + kPUnitSets * kPUnitCols <= 512u, "tensor memory map");
// barriers
constexpr uint32_t kPBarFull = 0, kPBarDone = kPRingMax, kPBarRows = 2 * kPRingMax;
constexpr uint32_t kPBarAccDone = kPBarRows + kPRowSets, kPBarAccFree = kPBarAccDone + 2, kPBarFin = kPBarAccFree + 2, kPBars = kPBarFin + 1;

struct PairItem {
    unsigned long long page;
    uint32_t nt, r;             // pairs of the chunk (0x100: the expert has more chunks); pair of slices or row tiles
};

// ---- operations of a CTA pair ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the shared-memory address of the same variable in the first CTA of the pair
__device__ __forceinline__ uint32_t first_cta(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// At another CTA's barrier, and the looks at one where such arrivals hand over tensor memory: scale codes that either CTA's warps have
// stored there, read by operations that the first CTA issues, and accumulators that its operations overwrite.  The order of the tensor
// operations on either side is the two fences' (fence_before, fence_after); the barrier between them is at cluster scope and orders nothing
// else, so it is relaxed: with .release.cluster and .acquire.cluster on the codes' barriers 8 tokens of 4096 x 2048 take 180 us in place of
// 110, 370 tokens 1100 in place of 720.  (Stages are written by copies, which have landed when the barrier of their own CTA says so.)
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.b32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// (mbar_wait, see there)
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
#pragma unroll 1
    for (uint32_t i = 0; i < kSpin; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2, 1000;\n"
            "selp.b32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}
// every CTA's 512 bytes at the descriptor's place into its own tensor memory
__device__ __forceinline__ void pair_copy_scales(uint32_t tmem, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(desc) : "memory");
}
// Sixteen columns of the warp's 32 lanes of its CTA's own tensor memory; complete behind tmem_st_wait().
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&w)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "r"(w[0]),
                 "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]), "r"(w[11]),
                 "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// arrives at the barrier of both CTAs when the tensor operations issued so far are complete
__device__ __forceinline__ void pair_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
// Whether the phase is complete, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.b32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// mbar_wait_warp with a test in front, 55 cycles where a try costs 83: most waits of a full pipeline are over when they begin.
// (Not in the one-token layer kernel, whose waits are for the memory: a stack of 14 layers 348 us, with the test 360.)
__device__ __forceinline__ bool stage_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_test(bar, parity) || mbar_wait(bar, parity, abort_flag));
}
// M = 256: 128 rows in each CTA
__device__ __forceinline__ constexpr uint32_t pair_idesc(uint32_t n) {
    return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) | ((256u >> 4) << 24);
}
// The 128 threads of a warpgroup of the epilogue.
__device__ __forceinline__ bool group_all(uint32_t id, bool ok) {
    uint32_t r;
    __syncwarp();
    asm volatile(
        "{\n.reg .pred p, q;\n"
        "setp.ne.b32 p, %1, 0;\n"
        "barrier.cta.red.and.pred q, %2, 128, p;\n"
        "selp.b32 %0, 1, 0, q;\n}"
        : "=r"(r)
        : "r"((uint32_t)ok), "r"(id)
        : "memory");
    return r != 0;
}

// The sum of a token's digit shares, rounded once: in F32 operations, two columns to an operation, because FP64 ones run at a
// quarter of their rate while the tensor cores are busy (sixteen conversions and additions of 8 tokens x 128 rows: 4200
// cycles, 1600 without the MMAs).  Added to s = 1.5 * 2^(e+5), where every share is below 2^(e+1), a share leaves what does not fit
// 2^(e-18) exactly behind (t = s + v; v - (t - s)); those remainders likewise 20 bits below; what they leave is at most
// 2^(e-39) and summed as it is.  The three parts are exact but for 2^-60 of the largest share - sums in double lose 2^-50 -
// and are added with the rounding errors of their own sum.  Shares too large or too small for the constants go through double.
__device__ __forceinline__ float2 minus2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
// columns first .. first + N - 1 and the N behind them into three parts each
template <int N, int M>
__device__ __forceinline__ void digit_parts(const uint32_t (&r)[M], int first, float2 sigma, float2 sigma2, float2 &p1, float2 &p2, float2 &p3) {
    float2 s1 = sigma, s2 = sigma2;
    p3 = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const float2 v = make_float2(__uint_as_float(r[first + c]), __uint_as_float(r[first + N + c]));
        const float2 t1 = __fadd2_rn(s1, v);
        const float2 v2 = minus2(v, minus2(t1, s1));
        s1 = t1;
        const float2 t2 = __fadd2_rn(s2, v2);
        p3 = __fadd2_rn(p3, minus2(v2, minus2(t2, s2)));
        s2 = t2;
    }
    p1 = minus2(s1, sigma);
    p2 = minus2(s2, sigma2);
}
// a + b + c rounded once but for what is far below the last bit
__device__ __forceinline__ float sum3(float a, float b, float c) {
    const float t = __fadd_rn(b, c), tb = __fsub_rn(t, b), te = __fadd_rn(__fsub_rn(b, __fsub_rn(t, tb)), __fsub_rn(c, tb));
    const float s = __fadd_rn(a, t), sa = __fsub_rn(s, a), se = __fadd_rn(__fsub_rn(a, __fsub_rn(s, sa)), __fsub_rn(t, sa));
    return __fadd_rn(s, __fadd_rn(se, te));
}
// the exponent field of the largest of N shares and whether the constants made of it are in range
template <int N, int M>
__device__ __forceinline__ uint32_t share_exponent(const uint32_t (&r)[M], int first) {
    float m = 0.0f;
#pragma unroll
    for (int c = 0; c < N; ++c) m = fmaxf(m, fabsf(__uint_as_float(r[first + c])));
    return __float_as_uint(m) & 0x7F800000u;   // (a NaN beside other shares is dropped here and makes the sum one)
}
__device__ __forceinline__ bool share_in_range(uint32_t ex) { return ex - (48u << 23) < (192u << 23); }   // 2^-79 .. 2^112
__device__ __forceinline__ float2 share_sigmas(uint32_t ex) {
    return make_float2(__uint_as_float(ex + (5u << 23) + 0x400000u), __uint_as_float(ex - (15u << 23) + 0x400000u));
}
template <int N, int M>
__device__ __forceinline__ void digit_sums_f64(const uint32_t (&r)[M], int first, double &a, double &b) {
    a = b = 0.0;
#pragma unroll
    for (int c = 0; c < N; ++c) {
        a += (double)__uint_as_float(r[first + c]);
        b += (double)__uint_as_float(r[first + N + c]);
    }
}
// all sixteen columns are one token's
__device__ __forceinline__ float digit_sum(const uint32_t (&r)[16]) {
    const uint32_t ex = max(share_exponent<8>(r, 0), share_exponent<8>(r, 8));
    if (!share_in_range(ex)) {
        double hi, lo;
        digit_sums_f64<8>(r, 0, hi, lo);
        return (float)(lo + hi);
    }
    const float2 sg = share_sigmas(ex);
    float2 p1, p2, p3;
    digit_parts<8>(r, 0, make_float2(sg.x, sg.x), make_float2(sg.y, sg.y), p1, p2, p3);
    return sum3(__fadd_rn(p1.x, p1.y), __fadd_rn(p2.x, p2.y), __fadd_rn(p3.x, p3.y));   // (the first two additions are exact)
}
// official arithmetic: six columns from `first` are one token's, the next six another's: their sums as BF16
template <int M>
__device__ __forceinline__ uint32_t digit_sums_pair(const uint32_t (&r)[M], int first) {
    const uint32_t e0 = share_exponent<6>(r, first), e1 = share_exponent<6>(r, first + 6);
    if (!share_in_range(e0) || !share_in_range(e1)) {
        double a, b;
        digit_sums_f64<6>(r, first, a, b);
        return bf16_pair((float)a, (float)b);
    }
    const float2 s0 = share_sigmas(e0), s1 = share_sigmas(e1);
    float2 p1, p2, p3;
    digit_parts<6>(r, first, make_float2(s0.x, s1.x), make_float2(s0.y, s1.y), p1, p2, p3);
    return bf16_pair(sum3(p1.x, p2.x, p3.x), sum3(p1.y, p2.y, p3.y));
}

// The same by plain additions, the smallest digits first, where that settles the BF16 values: each of the five sums on the way is
// rounded once, by at most 2^-24 of it, so where 2^-23 of their magnitudes' sum to either side (which leaves room for the
// roundings here) rounds to the same BF16 value, that is the exact sum's, and its F32 rounding's.  False, and nothing in `out`, for the
// others (one in some thousand; with a bound made of the largest share every other warp had one).
template <int M>
__device__ __forceinline__ bool digit_sums_quick(const uint32_t (&r)[M], int first, uint32_t &out) {
    float2 s = make_float2(__uint_as_float(r[first]), __uint_as_float(r[first + 6]));
    float ma = 0.0f, mb = 0.0f;
#pragma unroll
    for (int c = 1; c < 6; ++c) {
        s = __fadd2_rn(s, make_float2(__uint_as_float(r[first + c]), __uint_as_float(r[first + 6 + c])));
        ma = __fadd_rn(ma, fabsf(s.x));
        mb = __fadd_rn(mb, fabsf(s.y));
    }
    const float2 lo = __ffma2_rn(make_float2(ma, mb), make_float2(-0x1p-23f, -0x1p-23f), s);
    const float2 hi = __ffma2_rn(make_float2(ma, mb), make_float2(0x1p-23f, 0x1p-23f), s);
    out = bf16_pair(lo.x, lo.y);
    return out == bf16_pair(hi.x, hi.y);
}

// Operand rows of half a chunk of nt tokens, a multiple of sixteen: those of the first (nt + 1) / 2 tokens.
template <uint32_t kRows>
__device__ __forceinline__ uint32_t half_rows(uint32_t nt) { return (((nt + 1u) >> 1) * kRows + 15u) & ~15u; }

// kTok: most tokens of a chunk: 2, 6 or 12, in the official arithmetic 4, 16 or 32.  The kernel is compiled for each: what 12 or 32
// tokens need of code in the epilogue, which every launch fetches anew, and of loads for the items' records lay in the way of small blocks (us,
// official, one form and three: 8 tokens of 512 x 512 28.4 and 23.2, of 2048 x 1024, 64 experts, 48.6 and 42.2; one token of 4096 x 2048 47.0
// and 40.3).  The forms for small chunks keep to 80 registers (said by a bound of 768 threads): with 96 the CTAs of the launch behind
// find no room beside this one's, and are set up only when it ends (8 tokens 115 us, 96 registers and one F32 form 115-120, so 109.4; of
// 2048 x 1024 49.0, 52, 45.0; one token 45.7, 46, 42.3).  So do the official up kernels of all sizes, with a few bytes spilled (us, 96 and
// 80: 60 tokens over 32 of 1024 x 512 38.8 and 37.0, 20 over 64 of 2048 x 1024 55.9 and 54.3, 600 over 64 of 4096 x 2048 398 and 387, 1000 over
// 256 763 and 750).  The official down kernels for 16 and 32 lose by it (300 over 64 of 2048 x 1024 101.2 and 103.8), and so do the F32 ones
// for twelve (100 over 64 of 2048 x 1024 87.8: up 91.2, down 88.7).
template <bool kDown, bool kOff, uint32_t kTok>
__global__ void __launch_bounds__(kTok > (kOff ? (kDown ? 4u : 32u) : 6u) ? kPThreads : 768u, 1)
k_block_pair(const __grid_constant__ GemmArgs a, uint32_t *status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr uint32_t kRows = kOff ? 6u : 16u, kTileB = kRows * 128u;   // a token's digit rows, and the bytes of its tile
    static_assert(kTok <= kPCols / 2u / kRows * 2u, "the columns of an accumulator");
    constexpr uint32_t kHalf = (kTok * kRows + 31u) / 32u;       // groups of sixteen rows that a CTA of the pair brings at most
    constexpr uint32_t kMine = kOff ? kTok / 4u : kTok / 2u;      // tokens of an epilogue thread (official: pairs of them)
    constexpr uint32_t kPBatch = kOff ? 56u : 96u;                // items decoded at a time (10 KB of static shared memory are left beside the ring)
    __shared__ __align__(8) uint64_t bars[kPBars];
    __shared__ __align__(16) PairItem s_rec[kPBatch];
    __shared__ uint32_t s_pair[kPBatch][kTok];
    __shared__ float s_x[2][kOff ? 1u : kMine][64];               // an item's gates and up projections, handed across
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const uint32_t tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31u;
    const uint32_t rank = cluster_rank(), n_pairs = gridDim.x >> 1, me = blockIdx.x >> 1;
    const uint32_t K = kDown ? a.inter : a.hidden;
    const uint32_t nu = K >> 8;                                    // units of an item
    const uint32_t ring = a.ring, stage = a.stage;
    const size_t page_off = kDown ? mxfp4_down_offset(a.hidden, a.inter) : 0u;
    const uint32_t bar0 = smem_u32(bars), ring0 = smem_u32(smem);
    auto bar = [&](uint32_t i) { return bar0 + i * 8u; };
    volatile int *const abortp = &abort_flag;

    if (tid < kPBars) {
        uint32_t count = 1u;
        if (tid < kPRingMax) count = rank == 0u ? 2u : 1u;   // the copying thread; the first CTA's: and the second CTA's stage
        else if (tid >= kPBarRows && tid < kPBarRows + kPRowSets) count = 2u * kPCodes;   // the codes' warps of both CTAs
        else if (tid >= kPBarAccFree && tid < kPBarAccFree + 2u) count = 2u * kPEpi / 32u;
        mbar_init(bar(tid), count);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid == 0) abort_flag = 0;
    if (warp == kPMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        fence_before();
    }
    __syncthreads();
    cluster_barrier();   // the other CTA's barriers are there
    fence_after();
    const uint32_t tmem = tmem_slot;
    // (the down kernel reads records and pages in front of its wait, see below)
    if constexpr (!kDown) dependency_wait();
    const uint32_t R = (kDown ? (a.hidden >> 7) : (a.inter >> 6)) / 2u;   // items per chunk
    // The pair's items are q = me, me + n_pairs, ...  The chunks of one expert follow one another and so do their items, a row
    // tile's chunks side by side (so that pairs that run at the same time share the expert's units in the L2).
    const uint32_t n_items = __ldcg(a.n_chunks) * R;
    const uint32_t n_local = n_items > me ? (n_items - me + n_pairs - 1u) / n_pairs : 0u;

    // what the roles carry from batch to batch
    uint32_t slot = 0, round = 0, gi = 0, step = 0, set = 0, phase = 0;
    bool ready = false;   // the issuing warp: the next two stages are there
    bool ok = true;
    auto next_slot = [&]() {
        if (++slot == ring) {
            slot = 0;
            ++round;
        }
    };
    const unsigned long long once = l2_policy_evict_first();
    // (without an item the down kernel would end without having waited, and what is behind it would start beside the digits launch in front)
    if constexpr (kDown) {
        if (n_local == 0u) dependency_wait();
    }

#pragma unroll 1
    for (uint32_t base = 0; base < n_local; base += kPBatch) {
        const uint32_t nb = n_local - base < kPBatch ? n_local - base : kPBatch;
        // the batch's items into shared memory: the records, then the chunks' pairs, all loads in flight together
        if (tid < nb) {
            const uint32_t q = me + (base + tid) * n_pairs;
            const BlockChunk *g = a.chunks + q / R;
            const uint32_t c0 = __ldcg(&g->c0), nch = __ldcg(&g->nch), j = q - c0 * R;
            const uint32_t r = j / nch, c = c0 + (j - r * nch);
            s_rec[tid].page = __ldcg(reinterpret_cast<const unsigned long long *>(&a.chunks[c].page));
            s_rec[tid].nt = __ldcg(&a.chunks[c].nt) | (nch > 1u ? 0x100u : 0u);
            s_rec[tid].r = r;
            s_pair[tid][0] = c;
        }
        __syncthreads();
        {
            constexpr uint32_t kLoads = (kPBatch * kTok + kPThreads - 1u) / kPThreads;
            uint32_t p[kLoads];
#pragma unroll
            for (uint32_t k = 0; k < kLoads; ++k) {
                const uint32_t i = (tid + k * kPThreads) / kTok, t = (tid + k * kPThreads) % kTok;
                if (i < nb) p[k] = __ldcg(&a.chunks[s_pair[i][0]].pair[t]);
            }
            __syncthreads();
#pragma unroll
            for (uint32_t k = 0; k < kLoads; ++k) {
                const uint32_t i = (tid + k * kPThreads) / kTok, t = (tid + k * kPThreads) % kTok;
                if (i < nb) s_pair[i][t] = p[k];
            }
        }
        __syncthreads();
        if constexpr (kDown) {
            if (base == 0u) {
                // The launch in front (the second digits launch) writes the tiles and exponents of the hidden values, but neither the
                // records nor the pages; it lets this one start behind its own wait, so what is in front of it is complete.  So the items are
                // decoded and the ring's units asked for while it runs (us: 4 tokens of 512 x 512 27.9, so 25.7, 8 of 2048 x 1024 45.0 and 44.2,
                // 8 official ones 105.8 and 103.6; 370 tokens 0.5 %).
                if (warp >= kPProdWarp0 && warp < kPProdWarp0 + kPProds && lane == 31u) {
#pragma unroll 1
                    for (uint32_t s = warp - kPProdWarp0; s < ring; s += kPProds) {
                        const uint32_t i = s / nu, u = s - i * nu;
                        if (i >= nb) break;
                        const uint32_t nt = s_rec[i].nt & 0xFFu, half = (nt + 1u) >> 1, first = rank * half;
                        const uint32_t mine = nt > first ? min(nt - first, half) : 0u, full = bar(kPBarFull + s);
                        const uint8_t *const src = reinterpret_cast<const uint8_t *>(s_rec[i].page) + page_off +
                                                   ((size_t)(s_rec[i].r * 2u + rank) * nu + u) * kUnitStride;
                        mbar_arrive_expect(full, kStageA + mine * kTileB);
                        if (s_rec[i].nt >> 8) bulk_copy(ring0 + s * stage, src, kStageA, full);
                        else bulk_copy_stream(ring0 + s * stage, src, kStageA, full, once);
                    }
                }
                __syncwarp();
                dependency_wait();
            }
        }

        if (warp >= kPProdWarp0 && warp < kPProdWarp0 + kPProds) {
            // ---- a stage: the unit of this CTA's row tile, then the digit tiles of its half of the chunk ----
#pragma unroll 1
            for (uint32_t i = 0; i < nb && ok; ++i) {
                const uint32_t multi = warp_uniform(s_rec[i].nt >> 8), nt = warp_uniform(s_rec[i].nt & 0xFFu);
                const uint32_t half = (nt + 1u) >> 1, first = rank * half;   // this CTA's tokens
                const uint32_t mine = nt > first ? min(nt - first, half) : 0u;
                // a lane's copy of every stage: lane t < mine the tile of a token, the last lane the unit
                const bool is_unit = lane == 31u;
                const uint8_t *src = reinterpret_cast<const uint8_t *>(s_rec[i].page) + page_off +
                                     (size_t)(s_rec[i].r * 2u + rank) * nu * kUnitStride;
                if (lane < mine) {
                    uint32_t vec = kDown ? s_pair[i][first + lane] : s_pair[i][first + lane] / kPairsPerToken;
                    if constexpr (kOff && !kDown) vec = vec * 4u + (lane & 3u);   // the form for this place
                    src = a.dig + (size_t)vec * nu * kTileB;
                }
                const uint32_t bytes = is_unit ? kUnitStride : kTileB, to = ring0 + (is_unit ? 0u : kStageA + lane * kTileB);
#pragma unroll 1
                for (uint32_t u = 0; u < nu; ++u, src += bytes) {
                    if ((slot & (kPProds - 1u)) == warp - kPProdWarp0) {
                        ok = !round || stage_wait(bar(kPBarDone + slot), (round - 1u) & 1u, abortp);
                        if (!ok) break;
                        const uint32_t full = bar(kPBarFull + slot), dst = to + slot * stage;
                        if (is_unit && kDown && !round) {
                            // (asked for in front of the wait)
                        } else if (is_unit) {
                            mbar_arrive_expect(full, kStageA + mine * kTileB);
                            // an expert with one chunk is read once; with more, its later chunks want the units in the L2
                            if (multi) bulk_copy(dst, src, kStageA, full);
                            else bulk_copy_stream(dst, src, kStageA, full, once);
                        } else if (lane < mine) {
                            bulk_copy(dst, src, kTileB, full);   // (bytes that land before the barrier is armed are counted all the same)
                        }
                        __syncwarp();
                    }
                    next_slot();
                }
            }
        } else if (warp == kPMmaWarp) {
            if (rank == 0u) {
                const uint32_t tm = warp_uniform(tmem);
                const uint64_t a_desc0 = smem_desc(ring0, 1, 64, 2), b_desc0 = smem_desc(ring0 + kStageA, 1, 64, 2);
                const uint64_t sa_desc0 = smem_desc(ring0 + kUnitBytes, 0, 8, 0);
#pragma unroll 1
                for (uint32_t i = 0; i < nb && ok; ++i, ++gi) {
                    const uint32_t buf = gi & 1u, nt = warp_uniform(s_rec[i].nt & 0xFFu);
                    const uint32_t n = 2u * half_rows<kRows>(nt), idesc = pair_idesc(n);
                    if (gi >= 2u) {
                        const uint32_t free = bar(kPBarAccFree + buf), parity = ((gi - 2u) >> 1) & 1u;
                        ok = __all_sync(0xffffffffu, mbar_test_cluster(free, parity) || mbar_wait_cluster(free, parity, abortp));
                    }
                    if (!ok) break;
                    fence_after();
                    const uint32_t acc = tm + buf * kPCols;
#pragma unroll 1
                    for (uint32_t ku = 0; ku < nu; ku += 2u) {
                        const uint32_t slot1 = slot + 1u == ring ? 0u : slot + 1u, round1 = slot + 1u == ring ? round + 1u : round;
                        if (!ready) {
                            ok = __all_sync(0xffffffffu, mbar_wait_cluster(bar(kPBarRows + set), phase, abortp) &&
                                                             mbar_wait(bar(kPBarFull + slot), round & 1u, abortp) &&
                                                             mbar_wait(bar(kPBarFull + slot1), round1 & 1u, abortp));
                            if (!ok) break;
                        }
                        fence_after();
                        auto issue = [&](uint32_t at_slot, uint32_t odd) {
                            const uint32_t at = at_slot * (stage >> 4), sfa = tm + kPColUnits + ((step + odd) & (kPUnitSets - 1u)) * kPUnitCols;
                            const uint32_t sfb = tm + kPColRows + set * kPRowCols + odd * (kPRowCols / 2u);
                            pair_copy_scales(sfa, sa_desc0 + at);
                            pair_copy_scales(sfa + 4u, sa_desc0 + at + (kAtomBytes >> 4));
#pragma unroll
                            for (uint32_t kk = 0; kk < 4; ++kk) {
                                const uint32_t atom = kk >> 1, sfid = (kk & 1u) * 2u;
                                pair_mma(acc, a_desc0 + at + kk * 2u, b_desc0 + at + kk * 2u, idesc | (sfid << 29) | (sfid << 4),
                                         (sfa + atom * 4u) | (sfid << 30), (sfb + atom * 8u) | (sfid << 30), (ku || odd || kk) ? 1u : 0u);
                            }
                            pair_commit(bar(kPBarDone + at_slot));
                        };
                        if (elect_one()) issue(slot, 0u);
                        __syncwarp();
                        // the next two stages are looked at while the operations run
                        const uint32_t slot2 = slot1 + 1u == ring ? 0u : slot1 + 1u, round2 = slot1 + 1u == ring ? round1 + 1u : round1;
                        const uint32_t slot3 = slot2 + 1u == ring ? 0u : slot2 + 1u, round3 = slot2 + 1u == ring ? round2 + 1u : round2;
                        const uint32_t set2 = set + 1u == kPRowSets ? 0u : set + 1u, phase2 = set + 1u == kPRowSets ? phase ^ 1u : phase;
                        const bool r0 = mbar_test_cluster(bar(kPBarRows + set2), phase2), r1 = mbar_test(bar(kPBarFull + slot2), round2 & 1u);
                        const bool r2 = mbar_test(bar(kPBarFull + slot3), round3 & 1u);
                        if (elect_one()) issue(slot1, 1u);
                        __syncwarp();
                        ready = __all_sync(0xffffffffu, r0 && r1 && r2);
                        slot = slot2;
                        round = round2;
                        set = set2;
                        phase = phase2;
                        step += 2u;
                    }
                    if (!ok) break;
                    if (elect_one()) pair_commit(bar(kPBarAccDone + buf));
                    __syncwarp();
                }
            } else {
                // ---- the second CTA's stages are there ----
#pragma unroll 1
                for (uint32_t i = 0; i < nb * nu && ok; ++i) {
                    ok = stage_wait(bar(kPBarFull + slot), round & 1u, abortp);
                    if (!ok) break;
                    if (elect_one()) mbar_arrive_remote(first_cta(bar(kPBarFull + slot)));
                    __syncwarp();
                    next_slot();
                }
            }
        } else if (warp < kPEpi / 32u) {
            // ---- epilogue: a group's sixteen columns of digit shares, added exactly and rounded once ----
            const uint32_t wg = warp >> 2, row = tid & 127u, el = row & 63u, par = row >> 6;
            const uint32_t lane_base = tmem + (((warp & 3u) * 32u) << 16);
            const uint32_t free0 = first_cta(bar(kPBarAccFree));
#pragma unroll 1
            for (uint32_t i = 0; i < nb && ok; ++i, ++gi) {
                const uint32_t buf = gi & 1u, nt = s_rec[i].nt & 0xFFu, idx = s_rec[i].r * 2u + rank;   // slice or row tile
                const uint32_t *pair = s_pair[i];
                // official: this warpgroup's half of the chunk, its first token and how many there are
                const uint32_t t0 = wg * ((nt + 1u) >> 1), n_tok = nt > t0 ? min(nt - t0, (nt + 1u) >> 1) : 0u;
                ok = group_all(1u + wg, mbar_wait(bar(kPBarAccDone + buf), (gi >> 1) & 1u, abortp));
                if (!ok) break;
                fence_after();
                // tokens wg, wg + 2, ... of the chunk; official: those of its half, two BF16 values to a register
                float v[kOff ? 1u : kMine];
                uint32_t vb[kOff ? kMine : 1u] = {};
                if constexpr (kOff && kTok == 4u) {
                    uint32_t r[16];   // two tokens' six columns each
                    tmem_ld16(lane_base + buf * kPCols + wg * half_rows<kRows>(nt), r);
                    tmem_ld_wait();
                    if (!digit_sums_quick(r, 0, vb[0]) && n_tok) vb[0] = digit_sums_pair(r, 0);
                } else if constexpr (kOff) {
                    // eight tokens' six columns each at a time
                    const uint32_t at = lane_base + buf * kPCols + wg * half_rows<kRows>(nt);
#pragma unroll
                    for (uint32_t m = 0; m < kMine; m += 4u) {
                        if (2u * m < n_tok) {   // uniform in the warpgroup
                            uint32_t r[48];     // (columns beyond the half's rows are not used)
                            tmem_ld16(at + 12u * m, *reinterpret_cast<uint32_t(*)[16]>(r));
                            tmem_ld16(at + 12u * m + 16u, *reinterpret_cast<uint32_t(*)[16]>(r + 16));
                            tmem_ld16(at + 12u * m + 32u, *reinterpret_cast<uint32_t(*)[16]>(r + 32));
                            tmem_ld_wait();
                            // (without a branch between the four, so that their chains run side by side)
                            bool sure[4];
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) sure[k] = digit_sums_quick(r, 12 * (int)k, vb[m + k]);
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k)
                                if (!sure[k] && 2u * (m + k) < n_tok) vb[m + k] = digit_sums_pair(r, 12 * (int)k);
                        }
                    }
                } else {
#pragma unroll
                    for (uint32_t m = 0; m < kMine; m += 2u) {
                        const uint32_t g = 2u * m + wg;
                        if (g < nt) {   // uniform in the warpgroup
                            uint32_t r0[16], r1[16];
                            tmem_ld16(lane_base + buf * kPCols + 16u * g, r0);
                            if (m + 1u < kMine) tmem_ld16(lane_base + buf * kPCols + 16u * (g + 2u), r1);   // (not used beyond nt)
                            tmem_ld_wait();
                            v[m] = digit_sum(r0);
                            if (m + 1u < kMine) v[m + 1u] = digit_sum(r1);
                        }
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(free0 + buf * 8u);
                if constexpr (kDown) {
                    // row idx * 128 + `row` of the pairs' expert outputs
#pragma unroll
                    for (uint32_t m = 0; m < kMine; ++m) {
#pragma unroll
                        for (uint32_t k = 0; k < (kOff ? 2u : 1u); ++k) {
                            const uint32_t t = kOff ? 2u * m + k : 2u * m + wg;
                            if (t < (kOff ? n_tok : nt)) {
                                const size_t at = (size_t)pair[kOff ? t0 + t : t] * a.hidden + idx * 128u + row;
                                if constexpr (kOff) {
                                    a.out16[at] = (uint16_t)(k ? vb[m] >> 16 : vb[m]);   // (a linear's result is BF16)
                                } else if (a.ep_world > 1u) {
#pragma unroll 1
                                    for (uint32_t p = 0; p < a.ep_world; ++p) a.out_peer[p][at] = v[m];
                                } else {
                                    a.out[at] = v[m];
                                }
                            }
                        }
                    }
                } else if constexpr (kOff) {
                    // threads 0-63 of the warpgroup hold the gates of the slice's elements, threads 64-127 their up projections: BF16
                    // values into the pair's two rows (the rest is element by element and k_block_digits_official's)
#pragma unroll
                    for (uint32_t m = 0; m < kMine; ++m) {
#pragma unroll
                        for (uint32_t k = 0; k < 2; ++k)
                            if (2u * m + k < n_tok)
                                a.hval16[((size_t)pair[t0 + 2u * m + k] * 2u + par) * a.inter + idx * 64u + el] = (uint16_t)(k ? vb[m] >> 16 : vb[m]);
                    }
                } else {
                    // threads 0-63 of the warpgroup hold the gates of the slice's elements, threads 64-127 their up
                    // projections.  Each half finishes half of the tokens and hands the other the values it lacks.
#pragma unroll
                    for (uint32_t m = 0; m < kMine; ++m)
                        if (2u * m + wg < nt && (m & 1u) != par) s_x[wg][m][el] = v[m];
                    group_all(1u + wg, true);
#pragma unroll
                    for (uint32_t m = 0; m < kMine; ++m) {
                        const uint32_t t = 2u * m + wg;
                        if (t < nt && (m & 1u) == par) {
                            const float mine = v[m], other = s_x[wg][m][el];
                            a.hval[(size_t)pair[t] * a.inter + idx * 64u + el] = par ? swiglu_pair(other, mine) : swiglu_pair(mine, other);
                        }
                    }
                }
            }
        } else {
            // ---- the scale codes of ALL digit rows of the chunk (both CTAs' tensor cores multiply with every column), into tensor
            // memory as the multiplication wants them: operand row n at lane n % 32 of every quadrant, column n / 32, a word per 128 k.
            // Digit row j < 8 of a block with exponent E has the code 127 + E - 23 + 3 j, row 8 + j the code 127 + E - 47 + 3 j,
            // official row j 127 + E - 17 + 3 j; the exponents are stored as E + 100.  Lane t loads token t's, for two stages at a time;
            // rows that belong to nobody take any. ----
            const uint32_t rows0 = tmem + kPColRows + (((warp & 3u) * 32u) << 16), full0 = first_cta(bar(kPBarRows));
            constexpr uint32_t kCols = kHalf;   // tensor memory columns of a stage per 128 k
            // column c's row of this lane: its token, and (official: where the second half's rows start differs from item to item) what is
            // added to the exponents, in the lower and the upper half of a word
            uint32_t row_of[kOff ? kCols : 1u] = {}, bias0 = 0u;
            if constexpr (!kOff) {
                const uint32_t j = lane & 15u;
                bias0 = 0x01010101u * (uint32_t)(j < 8u ? 4 + 3 * (int)j : 3 * (int)(j & 7u) - 20);
            }
            auto rows_of = [&](uint32_t nt) {
                if constexpr (kOff) {
#pragma unroll
                    for (uint32_t c = 0; c < kCols; ++c) {
                        const uint32_t n = 32u * c + lane, half = (nt + 1u) >> 1, hr = half_rows<kRows>(nt), m = n < hr ? n : n - hr, in = m / kRows;
                        row_of[c] = ((n < hr ? in : half + in) & 31u) | ((10u + 3u * (m - in * kRows)) << 16);
                    }
                }
            };
            // the scale codes of one stage's rows: exponents of its two 128 k in, words out
            auto words = [&](uint32_t lo, uint32_t hi, uint32_t (&w)[16]) {
#pragma unroll
                for (uint32_t c = 0; c < 8u; ++c) {
                    w[c] = w[8u + c] = 0u;
                    if (c < kCols) {
                        const uint32_t at = kOff ? row_of[kOff ? c : 0u] : 2u * c + (lane >> 4), bias = kOff ? (at >> 16) * 0x01010101u : bias0;
                        w[c] = __shfl_sync(0xffffffffu, lo, at & 31u) + bias;
                        w[8u + c] = __shfl_sync(0xffffffffu, hi, at & 31u) + bias;
                    }
                }
            };
            auto exps_of = [&](uint32_t i) -> const uint4 * {
                if (i >= nb || lane >= (s_rec[i].nt & 0xFFu)) return nullptr;
                const uint32_t vec = kDown ? s_pair[i][lane] : s_pair[i][lane] / kPairsPerToken;
                return reinterpret_cast<const uint4 *>(a.exps + (size_t)vec * (K >> 5));
            };
            // two units' exponents per load, four loads in flight, each in registers of its own (a queue that moves them waits
            // for the newest): the units in steps of eight, the last step of an item perhaps short
            const uint4 *now = exps_of(0);
            uint4 e[4];
            auto fetch = [&](const uint4 *p, uint32_t u) { return p && u < nu ? __ldcg(p + (u >> 1)) : make_uint4(0u, 0u, 0u, 0u); };
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) e[k] = fetch(now, 2u * k);
#pragma unroll 1
            for (uint32_t i = 0; i < nb && ok; ++i) {
                const uint4 *const then = exps_of(i + 1u);
                rows_of(s_rec[i].nt & 0xFFu);
#pragma unroll 1
                for (uint32_t u0 = 0; u0 < nu && ok; u0 += 8u) {
                    const bool more = u0 + 8u < nu;
                    const uint4 *const next = more ? now : then;
                    const uint32_t at_u = more ? u0 + 8u : 0u;
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k) {
                        if (u0 + 2u * k < nu && ok) {
                            if (step >= 2u * kPRowSets) {
                                // the set's last stage, five before this pair's first, is complete; `slot` follows it
                                if (step > 2u * kPRowSets) next_slot();
                                next_slot();
                                ok = stage_wait(bar(kPBarDone + slot), round & 1u, abortp);
                            }
                            if (ok) {
                                const uint32_t at = rows0 + set * kPRowCols;
                                uint32_t w[16];
                                words(e[k].x, e[k].y, w);
                                tmem_st16(at, w);
                                words(e[k].z, e[k].w, w);
                                tmem_st16(at + 16u, w);
                                tmem_st_wait();
                                fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive_remote(full0 + set * 8u);
                                step += 2u;
                                if (++set == kPRowSets) set = 0;
                            }
                        }
                        e[k] = fetch(next, at_u + 2u * k);
                    }
                }
                now = then;
            }
        }
        __syncwarp();
        __syncthreads();  // the records are rewritten; a role that gave up has raised the flag
        if (abort_flag) break;
    }
    if (warp == kPMmaWarp && rank == 0u) {
        // All of the pair's tensor operations are complete before either CTA frees its tensor memory or leaves, also when a role
        // has given up with stages queued: they read both CTAs' shared memory and write both CTAs' tensor memory.
        if (elect_one()) pair_commit(bar(kPBarFin));
        __syncwarp();
        mbar_drain(bar(kPBarFin), 0);
    }
    if (warp >= kPProdWarp0 && warp < kPProdWarp0 + kPProds && lane == 0) {
        // copies in flight land in this CTA's shared memory, arrivals of the tensor operations at its barriers: wait for them.  (A slot's first
        // round has no wait that could run out, so every unit asked for in front of the kernel's wait is counted in `used`.)
#pragma unroll 1
        for (uint32_t s = warp - kPProdWarp0; s < ring; s += kPProds) {
            const uint32_t used = round + (s < slot ? 1u : 0u);   // rounds of this slot
            if (used) mbar_drain(bar((abort_flag ? kPBarFull : kPBarDone) + s), (used - 1u) & 1u);
        }
    }
    fence_before();
    __syncwarp();
    __syncthreads();
    cluster_barrier();
    // the last commit also arrives in the second CTA, behind the stages' arrivals: none of them is on its way when that
    // CTA leaves (behind the cluster barrier, because the first CTA may give up a wait's length after the second)
    if (rank != 0u && warp == kPCodeWarp0) mbar_drain(bar(kPBarFin), 0);
    if (warp == kPMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
    if (tid == 0 && abort_flag) {
        atomicExch(status, 0x5507u);
        atomicOr(a.why, kBlockGaveUp);
    }
    if constexpr (kDown && !kOff) {
        if (a.ep_world > 1u) {
            // every store of this CTA to the peers' buffers, and that it gave up, is ordered before the count; the last CTA of
            // the grid publishes the call's number to every rank, or 0 where a CTA of this kernel or of the up kernel gave up
            if (warp < kPEpi / 32u) __threadfence_system();
            __syncthreads();
            if (tid == 0) {
                __threadfence_system();
                if (atomicAdd(a.ep_counter, 1u) == gridDim.x - 1u) {
                    *a.ep_counter = 0u;
                    __threadfence_system();
                    const unsigned long long word = (atomicOr(a.why, 0u) & kBlockGaveUp) ? 0ull : (unsigned long long)a.ep_call;
#pragma unroll 1
                    for (uint32_t p = 0; p < a.ep_world; ++p)
                        asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(a.flag_peer[p] + a.ep_rank), "l"(word) : "memory");
                }
            }
        }
    }
}

constexpr int kMaxDevices = 64;

}  // namespace

// The dynamic shared memory the pair kernels may ask for on the current device (set once per device).
size_t pair_dynamic_limit() {
    static size_t limit[kMaxDevices] = {};
    int dev = -1, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    if (limit[dev]) return limit[dev];
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    const void *const fns[] = {(const void *)k_block_pair<false, false, 2>,  (const void *)k_block_pair<true, false, 2>,
                               (const void *)k_block_pair<false, false, 6>,  (const void *)k_block_pair<true, false, 6>,
                               (const void *)k_block_pair<false, false, 12>, (const void *)k_block_pair<true, false, 12>,
                               (const void *)k_block_pair<false, true, 4>,   (const void *)k_block_pair<true, true, 4>,
                               (const void *)k_block_pair<false, true, 16>,  (const void *)k_block_pair<true, true, 16>,
                               (const void *)k_block_pair<false, true, 32>,  (const void *)k_block_pair<true, true, 32>};
    size_t fixed = 0;
    cudaFuncAttributes fa;
    for (const void *fn : fns) {
        if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return 0;
        fixed = std::max(fixed, fa.sharedSizeBytes);
    }
    fixed = (fixed + 1023u) & ~(size_t)1023u;   // the ring starts on a 1 KB boundary behind the static part
    if ((size_t)optin <= fixed) return 0;
    const size_t most = (size_t)optin - fixed;
    for (const void *fn : fns)
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) return 0;
    limit[dev] = most;
    return most;
}

cudaError_t launch_pair_gemm(cudaStream_t st, int sm_count, bool down, bool official, GemmArgs args, uint32_t half, uint32_t *status) {
    args.stage = kStageA + half * 2048u;
    args.ring = std::min<uint32_t>((uint32_t)(pair_dynamic_limit() / args.stage), kPRingMax);
    if (args.ring < 2u * kPRowSets || half == 0u || 2u * half > kPGroups) return cudaErrorInvalidConfiguration;
    const size_t smem = (size_t)args.ring * args.stage;
    const dim3 grid((uint32_t)sm_count & ~1u), block(kPThreads);
    auto run = [&](auto up_kernel, auto down_kernel) {
        return launch_pdl(down ? down_kernel : up_kernel, grid, block, smem, st, 2u, args, status);
    };
    if (!official && half == 1u) return run(k_block_pair<false, false, 2>, k_block_pair<true, false, 2>);
    if (!official && half <= 3u) return run(k_block_pair<false, false, 6>, k_block_pair<true, false, 6>);
    if (!official) return run(k_block_pair<false, false, 12>, k_block_pair<true, false, 12>);
    if (half == 1u) return run(k_block_pair<false, true, 4>, k_block_pair<true, true, 4>);
    if (half <= 3u) return run(k_block_pair<false, true, 16>, k_block_pair<true, true, 16>);
    return run(k_block_pair<false, true, 32>, k_block_pair<true, true, 32>);
}

}  // namespace s14
