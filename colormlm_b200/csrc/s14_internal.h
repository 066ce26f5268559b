// Internal declarations shared by the kernel file and the C-ABI file.
#ifndef S14_INTERNAL_H
#define S14_INTERNAL_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/polaris_s14_cuda.h"

namespace s14 {

// One (expert page, token) pair of a fused layer call.
struct Job {
    const uint8_t *page;
    uint32_t kind;      // S14_PAGE_MXFP4 | S14_PAGE_FP8
    uint32_t token;     // row of x / y
    float weight;       // route weight (unused for the shared expert)
    uint32_t is_shared; // added last with weight 1
    uint32_t out_index; // row of the per-job down outputs this job writes (its job id unless
                        // the caller wants route slots, as the expert-parallel exchange does)
};

constexpr uint32_t kMaxTokens = S14_MAX_BLOCK_TOKENS;
constexpr uint32_t kMaxJobs = kMaxTokens * (S14_EXPERTS_PER_TOKEN + 1);

// Jobs are stored grouped by expert page (so that a page's second reader finds it
// in L2); token_jobs lists each token's jobs in mix order (route order, shared last).
struct JobTable {
    uint32_t n_jobs;
    uint32_t n_tokens;
    uint32_t token_job_begin[kMaxTokens + 1];
    uint8_t token_jobs[kMaxJobs];
    Job jobs[kMaxJobs];
};

// Optional per-kernel timing marks of one routed layer call: events are recorded before the
// router (0), before the up phase (1), between up and down (2), before the mix (3), after it (4).
struct KernelMarks {
    cudaEvent_t ev[5];
};

struct UmmaScratch;

// Expert-parallel exchange of the tcgen05 layer kernel over peer memory.  Every rank holds an
// exchange buffer: two slot buffers [n_slots, hidden] of 8-byte words {F32 bits, step + 1} (steps
// alternate between them), then the rank's own step count (64 bytes), then one 8-byte word per
// rank: the number of steps that rank has finished.  A rank stores the down vectors of the
// experts it owns into the slot rows of EVERY rank's buffer, each value with the step's number in
// one 8-byte store (plain stores to peer memory; an aligned 8-byte store arrives whole, so the
// number validates the value beside it and no fence or flag is needed); each rank polls (bounded)
// the words it needs in its own buffer and mixes from them.  Before a rank writes the slot buffer
// of step s it waits (bounded) until every peer has finished step s - 2, the last reader of that
// buffer; a rank that owns nothing in a step is waited for in this way too.  world <= 1: no exchange.
constexpr uint32_t kMaxEpWorld = 8;
struct EpExchange {
    unsigned long long *slots[kMaxEpWorld];  // rank p's exchange buffer, as mapped on this rank
    uint32_t *step;                // this rank's step count (device memory, kept by the kernel)
    uint32_t world, rank;
    uint32_t n_slots;              // top_k (+ 1 with a shared expert)
    uint32_t wait_and_mix;         // 0: publish only (single-GPU emulation of the other ranks)
    uint32_t wait_limit;           // polls (about a microsecond each) of one word before the rank gives up
};
inline size_t ep_exchange_slot_bytes(uint32_t hidden) {
    return sizeof(unsigned long long) * 2u * (S14_EXPERTS_PER_TOKEN + 1) * hidden;
}
inline size_t ep_exchange_bytes(uint32_t hidden) {
    return ep_exchange_slot_bytes(hidden) + 64u + sizeof(unsigned long long) * kMaxEpWorld;
}

// What the router reads and writes, for a layer call that computes its own routes: the tcgen05
// layer kernel scores the experts in its first microseconds (every CTA a few of them), and every
// CTA then picks the routes from the scores; other layer kernels run k_router first.
struct FusedRouter {
    const uint16_t *weight;            // [n_experts, hidden] BF16
    const float *bias;                 // [n_experts] or NULL
    float *scores, *select;            // [n_experts] scratch: score, score + bias
    uint32_t n_experts, score_fn, top_k;
    float route_scale;
    int32_t *ids_out;                  // [top_k] or NULL
    float *weights_out;                // [top_k] or NULL
    JobTable *table_out;               // the device job table k_router fills
    const uint8_t *const *page_table;  // [n_experts] expert pages (MXFP4)
    const uint8_t *shared_page;        // or NULL
    uint32_t shared_kind;
    uint32_t ep_rank, ep_world, shared_owner;
    uint32_t has_shared;               // every layer has a shared expert (a stack's layers say where)
};

// What one layer of a decode stack brings of its own (device memory, constant during a step): the
// tcgen05 layer kernel walks an array of these in one launch, the output of a layer (plus its input,
// if the stack keeps a residual) being the next layer's token.  Router shape, score function, top_k
// and page kind are the stack's and come with FusedRouter.
struct StackLayer {
    const uint16_t *router_weight;     // [n_experts, hidden] BF16
    const float *bias;                 // [n_experts] or NULL
    const uint8_t *const *page_table;  // [n_experts] expert pages (MXFP4)
    const uint8_t *shared_page;        // MXFP4 page; NULL only if no layer of the stack has one
    int32_t *ids_out;                  // [top_k] or NULL: the layer's route
    float *weights_out;                // [top_k] or NULL
    float *y_out;                      // [hidden] or NULL: the layer's MoE output before the residual
};

cudaError_t launch_mxfp4_matvec(cudaStream_t st, uint32_t mode, int sm_count, const float *x,
                                const uint8_t *w, const uint8_t *s, float *y, uint32_t n, uint32_t k);
cudaError_t launch_fp8_matvec(cudaStream_t st, uint32_t mode, int sm_count, uint32_t scale_format,
                              uint32_t n_tokens, const float *x, const uint8_t *w, const void *s,
                              float *y, uint32_t n, uint32_t k);
cudaError_t launch_swiglu_limit(cudaStream_t st, const float *gate, const float *up, float *y,
                                uint32_t n);
cudaError_t launch_route_mix(cudaStream_t st, const float *expert, float *routed, uint32_t n,
                             float weight);
cudaError_t launch_moe_accumulate(cudaStream_t st, const float *expert, float *acc, uint32_t n,
                                  float weight);
// Which implementation the calling thread's last launch_moe_layer chose (S14_LAYER_PATH_* of the header).
uint32_t last_layer_path();
// Returns the number of kernels launched.  h: [kMaxJobs, inter], d: [kMaxJobs, hidden].
int launch_moe_layer(cudaStream_t st, uint32_t mode, int sm_count, const JobTable *dev_table,
                     const JobTable &param_table, uint32_t n_tokens, uint32_t n_jobs_max,
                     uint32_t hidden, uint32_t inter, const float *x, float *h, float *d, float *y,
                     cudaError_t *err, const KernelMarks *km = nullptr, bool all_mxfp4 = false,
                     unsigned int *counters = nullptr, const struct UmmaScratch *umma = nullptr,
                     const FusedRouter *router = nullptr, const EpExchange *ep = nullptr,
                     const uint16_t *x_bf16 = nullptr, float *x_stage = nullptr, struct BranchPost *post = nullptr);
// (x_bf16, x_stage: the token as BF16; its F32 values may be written to x_stage, which is x)
// What the executor's step does with a layer's output: rounded to BF16 (branch_out, or NULL), then hc_post over the
// post-attention state.  A path that does it in its last launch, without writing y, sets `done`.
struct BranchPost {
    uint16_t *branch_out;
    const void *residual;
    const float *post, *comb;
    void *merged;
    bool done;
};
// Whether a one-token layer with an FP8 shared page runs it by kernels of its own behind the tensor-core layer
// kernel, which runs the routed experts; the last one adds the shared expert's output to theirs.
bool fp8_shared_layer_ok(int sm_count, uint32_t mode, const struct UmmaScratch *umma, uint32_t n_routed, uint32_t hidden, uint32_t inter);
// That layer (three launches): the routed experts' jobs, or a router without the shared expert.  h: [inter], d:
// [kMaxJobs, hidden] scratch.
int launch_layer_fp8_shared(cudaStream_t st, int sm_count, const JobTable &routed, const FusedRouter *router, const uint8_t *shared_page,
                            const float *x, const uint16_t *x_bf16, float *h, float *d, float *y,
                            unsigned int *counters, const struct UmmaScratch *umma, uint32_t hidden, uint32_t inter, cudaError_t *err,
                            BranchPost *post = nullptr);
// One token through one expert of an FP8 page (s14_fp8_expert.cu): x F32, or BF16 as x_bf16; h [inter] scratch; the expert's
// output added to `routed` [hidden] (kNoSum: see there) goes to y, or through `post`.  hidden and inter 1024, 2048 or 4096; x on a 16-byte boundary,
// x_bf16 (or NULL) on an 8-byte one.
inline bool fp8_expert_takes(const uint16_t *x_bf16) { return (reinterpret_cast<uintptr_t>(x_bf16) & 7u) == 0u; }
cudaError_t launch_fp8_expert(cudaStream_t st, int sm_count, const float *x, const uint16_t *x_bf16, const uint8_t *page,
                              float *h, float *routed, float *y, const BranchPost *post, uint32_t hidden, uint32_t inter);
// Scratch of the tcgen05 layer kernel (s14_moe_umma.cu): per job the digit tile of its hidden
// values and the tile's block exponents (umma_scratch_bytes), and the device status word a
// timed-out wait sets.
struct UmmaScratch {
    uint8_t *tiles;
    uint32_t *status;
    unsigned long long *trace;  // per-CTA time marks of the last launch (profiling runs), or nullptr
    float *handed;              // [4096]: see kNoSum
};
// A layer's sums that a launch behind it goes on with (an FP8 shared expert's, the end of the executor's step) lie in `handed`,
// which holds this value wherever there is none: a NaN that no addition gives (CUDA's is 0x7fffffff).  The launch that takes a sum
// puts it back.  So what a layer kernel that gave up did not write is not taken from the call before, and the launch behind
// writes no result for it either.
constexpr uint32_t kNoSum = 0xFFFFFFFFu;
size_t umma_scratch_bytes();
size_t umma_trace_bytes(int sm_count);
uint32_t umma_trace_words();
// One token, every job an MXFP4 page, hidden and inter multiples of 512 that fit shared and tensor memory.
// Sets the kernel's shared-memory attribute for the current device on first use.
bool umma_layer_ok(int sm_count, uint32_t n_tokens, uint32_t n_jobs_max, uint32_t hidden, uint32_t inter);
// Whether the tcgen05 layer kernel can score n_experts itself (a CTA scores at most two; at most 256 CTAs).
bool umma_router_ok(int sm_count, uint32_t n_experts);
// The items CTA c of G runs, in order (see s14_moe_umma.cu); returns their number, writes at most cap.
__host__ __device__ uint32_t layer_work_list(uint32_t c, uint32_t G, uint32_t n_jobs, uint32_t S, uint32_t RT,
                                             uint32_t KU, uint32_t KD, uint32_t *items, uint32_t cap, uint32_t n_early);
// ... and where CTAs run in pairs (s14_moe_umma.cu); the number that CTA `b` of the grid has in that deal
__host__ __device__ uint32_t layer_pair_list(uint32_t c, uint32_t G, uint32_t n_jobs, uint32_t S, uint32_t RT,
                                             uint32_t KU, uint32_t KD, uint32_t *items, uint32_t cap, uint32_t n_early);
__host__ __device__ uint32_t pair_cta(uint32_t b, uint32_t G, uint32_t F);
// whether that deal shares items (otherwise the lists are layer_work_list's)
__host__ __device__ bool layer_pairs_share(uint32_t G, uint32_t n_jobs, uint32_t S, uint32_t KU, uint32_t n_early);
uint32_t layer_items_bound(uint32_t G, uint32_t n_jobs, uint32_t S, uint32_t RT, uint32_t KU, uint32_t KD);
// Both phases and the mix in one launch (y == nullptr: the expert outputs go to d, the caller mixes).
// With a router the kernel computes the routes itself and the job tables are not read.  x_bf16: the token as BF16 values (x is
// not read then), on an 8-byte boundary.  ahead: bytes that the launches behind will read, asked into the L2 when the kernel's own
// copies are under way; on a 16-byte boundary.
cudaError_t launch_moe_layer_umma(cudaStream_t st, int sm_count, const JobTable *dev, const JobTable &param,
                                  const float *x, float *d, float *y, uint8_t *tiles, unsigned int *counters,
                                  uint32_t *status, uint32_t hidden, uint32_t inter,
                                  const FusedRouter *router = nullptr, const EpExchange *ep = nullptr,
                                  unsigned long long *trace = nullptr, const StackLayer *stack = nullptr,
                                  uint32_t n_layers = 1, float *hbuf = nullptr, bool residual = false,
                                  const uint16_t *x_bf16 = nullptr, const uint8_t *ahead = nullptr, size_t ahead_bytes = 0);
int launch_router(cudaStream_t st, const s14_router_desc &r, float *scores, float *select,
                  JobTable *table_out, const uint8_t *const *page_table, const uint8_t *shared_page,
                  uint32_t shared_kind, unsigned int *counter, cudaError_t *err,
                  const KernelMarks *km = nullptr, uint32_t ep_rank = 0, uint32_t ep_world = 1,
                  uint32_t shared_owner = 0);
// out[i] = residual ? x[i] + y[i] : y[i]; y_copy (or NULL) also receives y (a stack's layers launched one by one).
cudaError_t launch_stack_step(cudaStream_t st, const float *x, const float *y, float *out, float *y_copy,
                              uint32_t n, bool residual);
cudaError_t launch_mix_slots(cudaStream_t st, const float *slots, const float *weights, uint32_t n_routed,
                             int has_shared, float *y, uint32_t hidden);
cudaError_t launch_head_logits(cudaStream_t st, int sm_count, const float *x, uint32_t n_tokens,
                               const uint16_t *w, uint32_t n_rows, uint32_t hidden, float *out,
                               uint32_t out_stride);
cudaError_t launch_greedy_argmax(cudaStream_t st, const float *logits, uint32_t vocab,
                                 int64_t *result);
// The head's reduce of a BF16 state, RMSNorm, and the BF16 result as F32 values (x_out [hidden]); hidden a multiple of
// 256 up to 8192.
cudaError_t launch_head_prep(cudaStream_t st, const uint16_t *state, const float *fn, const float *scale, const float *base,
                             const float *norm_weight, uint32_t hidden, float norm_eps, float hc_eps, float *x_out);

// ---- a block of tokens through one layer, grouped by expert (s14_moe_block.cu, s14_moe_pair.cu) ----
constexpr uint32_t kBlockNt = 32;  // most tokens of one chunk (N = 192: six digit rows per token at least)
// Up to kBlockNt (token, route) pairs that share an expert page.  The chunks of one expert follow
// one another: c0 is the first of them, nch their number.
struct BlockChunk {
    const uint8_t *page;
    uint32_t nt;               // pairs in the chunk
    uint32_t c0, nch;
    uint32_t pair[kBlockNt];   // token * 7 + position in the mix (6: the shared expert)
    uint32_t pad;
};
constexpr uint32_t kBlockBadId = 1;   // an expert id was out of range
constexpr uint32_t kBlockGaveUp = 2;  // a wait inside a contraction kernel ran out
// Bytes of a token's digit tiles per 256 elements: sixteen rows of 128, or four forms of six rows (s14_moe_block.cu).
constexpr uint32_t kXDigBytes = 4u * 6u * 128u;
// Device workspace of a block object, sized for max_tokens at creation.
struct BlockWork {
    BlockChunk *chunks;
    uint32_t *counts;          // [0] chunks, [1], [2] chunks x slices, row tiles (above twelve tokens pairs of them), [3] why the call writes
                               // no result: kBlockBadId, kBlockGaveUp (set anew by every call's grouping)
    uint8_t *xdig, *xexp;      // the tokens' digit tiles and block exponents
    uint8_t *slots;            // official arithmetic: which of the four forms of a digit tile each pair's place in its chunk takes
    uint8_t *hdig, *hexp;      // the pairs' hidden values likewise
    float *d;                  // the pairs' expert outputs [pair, hidden]; official arithmetic: BF16 values, in the first half
    float *hval;               // the pairs' hidden values [pair, inter]; official arithmetic: their gates and up projections [pair, 2, inter]
                               // as BF16 values.  (What a pair without a route has there may be the other kind's bits.)
};
// Expert-parallel exchange of the block kernels over peer memory: every rank holds two pair buffers
// [pairs, hidden] F32 (calls alternate between them) and, per buffer, one 8-byte word per rank: the number
// of the last call whose rows that rank has written there.  The down kernel stores the rows of the experts it
// owns into every rank's buffer (plain stores to peer memory) and its last CTA publishes the call's number (0 where any CTA of
// the call's contraction kernels gave up: its rows are not there);
// the mix waits (bounded) until every rank's word says this call.  A rank writes call s + 1 only after its own
// mix of call s, which waited for every rank's rows of call s; so a rank that writes into a buffer for call
// s + 2 knows that every rank has finished reading call s from it: two buffers are enough.
struct BlockEp {
    float *pairs_peer[kMaxEpWorld];               // the call's pair buffer of rank p, as mapped on this rank
    unsigned long long *flags_peer[kMaxEpWorld];  // ... its flag words [world]
    const unsigned long long *flags;              // this rank's own flag words of the call's buffer
    unsigned int *counter;                        // arrival counter of the down kernel's CTAs (zero at rest)
    uint32_t world, rank, call, wait_limit;
};
// Whether the grouped tensor-core kernels can run these sizes on the current device.
bool moe_block_ok(int sm_count, uint32_t hidden, uint32_t inter, uint32_t n_experts, uint32_t top_k);
size_t moe_block_max_chunks(uint32_t max_tokens);
// ids / weights: device [n_tokens, top_k] (a negative id: no route); pages: device [n_tokens, top_k] page of every
// route, or NULL with page_table [n_experts].  Returns the number of kernels launched.
int launch_moe_block(cudaStream_t st, int sm_count, const BlockWork &w, const float *x, float *y, const int32_t *ids,
                     const float *weights, const uint8_t *const *pages, const uint8_t *const *page_table,
                     const uint8_t *shared_page, uint32_t n_tokens, uint32_t top_k, uint32_t n_experts, uint32_t hidden,
                     uint32_t inter, uint32_t *status, cudaError_t *err, bool residual = false,
                     uint32_t ep_rank = 0, uint32_t ep_world = 1, float *pairs_out = nullptr, const BlockEp *ep = nullptr,
                     bool shared_by_token = false, bool official = false);
// With pairs_out (expert parallel: rank ep_rank of ep_world computes the experts e with e mod world == rank) the
// pairs' expert outputs [n_tokens * 7, hidden] go there, zero where another rank owns the expert, and no mix runs;
// launch_block_mix mixes such a buffer once the ranks' buffers have been added up (x: the layer's input for a residual, or NULL).
cudaError_t launch_block_mix(cudaStream_t st, const float *pairs, const int32_t *ids, const float *weights, uint32_t n_tokens,
                             uint32_t top_k, bool has_shared, const float *x, float *y, uint32_t hidden, const uint32_t *counts,
                             const BlockEp *ep = nullptr, uint32_t *status = nullptr);
// Scores and routes of many tokens (s14_router.cu).  Same arithmetic as launch_router.  hidden is a multiple of 512 up to 4096; scores, select:
// [n_tokens, n_experts] scratch, parts: [8, n_tokens, 256] (for large blocks; a block's pair outputs, of 7 x 512 values a token
// at least, have room for it and are written later); status: the context's word (0x5509: a wait inside a kernel ran out, the routes are right).  Returns
// the number of kernels launched.
int launch_router_batch(cudaStream_t st, const s14_router_desc &r, float *scores, float *select, float *parts, uint32_t *status,
                        cudaError_t *err);

// ---- the steps on either side of the MoE inside one layer (s14_glue.cu) ----
// scratch: hc_scratch_bytes(the most tokens of a call).  Returns the number of kernels launched.
size_t hc_scratch_bytes(uint32_t max_tokens, int sm_count);
int launch_hc_pre(cudaStream_t st, int sm_count, bool bf16, bool head, uint32_t n_tokens, uint32_t hidden, const void *x, const float *fn,
                  const float *scale, const float *base, float norm_eps, uint32_t iters, float hc_eps, double *scratch, void *reduced,
                  float *post, float *comb, float *pre, uint32_t *status, cudaError_t *err);
cudaError_t launch_hc_post(cudaStream_t st, int sm_count, bool bf16, uint32_t n_tokens, uint32_t hidden, const void *branch, const void *residual,
                           const float *post, const float *comb, void *merged);
cudaError_t launch_rms_norm(cudaStream_t st, int sm_count, bool bf16, uint32_t n_tokens, uint32_t hidden, const void *x, const float *w, float eps,
                            void *out);
cudaError_t launch_router_hash(cudaStream_t st, const s14_router_desc &r, const int64_t *tid2eid);
cudaError_t launch_bf16_to_f32(cudaStream_t st, const uint16_t *in, float *out, uint32_t n);
// branch = BF16 of y (to branch_out, or NULL), merged = post * branch + comb . residual: one token of BF16 streams.
cudaError_t launch_branch_post(cudaStream_t st, uint32_t hidden, float *y, uint16_t *branch_out, const void *residual,
                               const float *post, const float *comb, void *merged);

}  // namespace s14


#endif
