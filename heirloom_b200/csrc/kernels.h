// Internal entry points shared between translation units: the same kernels the C ABI exposes,
// with scratch memory passed explicitly so the step executor can plan it once.
#pragma once
#include "common.cuh"

namespace hl {

// How a GEMM's work is cut: explicit split-K (partial sums for a second kernel), or whole waves of
// tiles followed by tiles whose k blocks are dealt out evenly over the CTAs.
struct GemmPlan {
  int splits;
  int dp_tiles, sk_tiles;
  size_t splitk_bytes;   // scratch for explicit split-K partial sums
  size_t sk_slot_bytes;  // scratch for the raw accumulators of partly finished tiles
};
GemmPlan gemm_plan(const hl_gemm_desc* d, int sm_count);
// For a cross-entropy loss without stored logits: per 128 columns (n in all, `parts` is [ceil(n/128)][m]) and row the maximum times
// log2(e) and the sum of 2^(x log2(e) - that), and the row's value at its target (nothing when it is out of range).
struct GemmRowStats {
  float2* parts;
  float* target_logit;  // [m]
  const int64_t* targets;
  float2* rows;         // [m] the whole row's maximum (in the same unit) and grad_scale over its sum; null without a gradient
  float grad_scale;
};
int gemm_bf16_run(hl_ctx* ctx, const hl_gemm_desc* d, const void* a, const void* b, void* c, const float* bias,
                  const void* aux_in, void* aux_out, float* workspace, size_t workspace_bytes, unsigned* stream_flags,
                  const GemmRowStats* row_stats = nullptr);
// The product with bias of which only those are wanted; false when this shape has no such form and nothing was done.
// `unused_c`: any memory of the result's size.
bool gemm_bf16_row_stats(hl_ctx* ctx, const hl_gemm_desc* d, const void* a, const void* b, const float* bias, const GemmRowStats& stats,
                         void* unused_c, int* rc);
// The mean loss out of them, and `rows` where it is wanted.  `loss_host` may be null.
int row_stats_loss(hl_ctx* ctx, const GemmRowStats& stats, int rows, int classes, float* row_loss, float* loss_dev, float* loss_host = nullptr);
// The same product again (call it where gemm_bf16_row_stats returned true), its result turned into the loss's gradient in bf16 on
// its way out: (2^(x log2(e) - maximum) - [column is the target] * sum) * grad_scale / sum.
int gemm_bf16_loss_gradient(hl_ctx* ctx, const hl_gemm_desc* d, const void* a, const void* b, const float* bias, const GemmRowStats& stats,
                            void* dlogits);
// Products that leave most of the chip idle in 128 x 256 tiles (gemm_small.cu): how many CTAs share the contraction of one of
// its 128 x bn tiles (0: not one of them), and whether a CTA has the SM's shared memory to itself.
struct GemmSmallPlan {
  int splits, bn;
  bool deep;
};
GemmSmallPlan gemm_small_plan(const hl_gemm_desc* d, const GemmPlan& big, int device, int sm_count);
int gemm_small_run(hl_ctx* ctx, const hl_gemm_desc* d, const GemmSmallPlan& plan, const void* a, const void* b, void* c,
                   const float* bias, const void* aux_in, void* aux_out, float* row_sum = nullptr);
// The GEMM with its scratch taken from (and grown in) the context.
int gemm_bf16_ctx(hl_ctx* ctx, const hl_gemm_desc* d, const void* a, const void* b, void* c, const float* bias,
                  const void* aux_in, void* aux_out);
// The scratch that gemm_bf16_ctx would take, or false where the product also uses the context's flags or its tile counter, which only one
// stream may: the launches' shares of the counter follow one another in the order in which they were queued.
bool gemm_bf16_scratch(hl_ctx* ctx, const hl_gemm_desc* d, size_t* bytes);
// A plain product with the sums of A's rows over the contraction beside it (a weight gradient and its bias gradient), where
// that costs no launch of its own; *done tells whether it was one of those, otherwise nothing has been launched.
bool gemm_bf16_small_applies(hl_ctx* ctx, const hl_gemm_desc* d);
int gemm_bf16_row_sums(hl_ctx* ctx, const hl_gemm_desc* d, const void* a, const void* b, void* c, float* row_sum, bool* done);

// Column reductions (layer-norm parameter gradients, bias gradients) end in a fold of per-block partial rows.  A
// caller that runs several of them before anyone reads the results hands in a FoldBatch: the kernels then leave their
// partial rows in the batch's scratch and one launch (fold_batch_flush) folds all of them, in a fixed order.
struct FoldJob {
  const float* partial;  // [blocks][total]
  int blocks, total, features;
  float *o0, *o1, *o2;   // column c goes to o(c / features)[c % features]; null outputs are skipped
};
struct FoldBatch {
  static constexpr int kMaxJobs = 16;
  FoldJob jobs[kMaxJobs];
  int n = 0;
  float* scratch = nullptr;  // device memory, `capacity` floats
  size_t capacity = 0, used = 0;
};
// Room for `elems` partial sums in the batch, or null when the batch is absent or full.
float* fold_batch_reserve(FoldBatch* batch, size_t elems);
// The same, folding what the batch holds when it is full; null (the caller folds at once) when there is no batch or it is too
// small for this reduction.
int fold_batch_room(hl_ctx* ctx, FoldBatch* batch, size_t elems, float** out);
void fold_batch_add(FoldBatch* batch, const float* partial, int blocks, int total, int features, float* o0, float* o1,
                    float* o2);
int fold_batch_flush(hl_ctx* ctx, FoldBatch* batch);

// Weight gradients of several layers in one launch (gemm_group.cu): dw[n_out, n_in] = dyᵀ · x and, when db is given, its column
// sums, dy and x bf16 with one row per token.  `sums`: device memory, gemm_group_sums() floats for every product with a db.
struct WeightGradJob {
  const __nv_bfloat16 *dy, *x;
  int n_out, n_in;
  float *dw, *db;
};
constexpr int kMaxGroupJobs = 70;
int gemm_group_tiles(int n_out, int n_in);
size_t gemm_group_sums(int n_out, int n_in);
int gemm_group_run(hl_ctx* ctx, const WeightGradJob* jobs, int count, int tokens, float* sums, FoldBatch* fold);

int bias_grad_impl(hl_ctx* ctx, const void* grad_out, int dtype, float* grad_bias, int rows, int cols,
                   FoldBatch* defer = nullptr);

int layer_norm_forward_impl(hl_ctx* ctx, const void* x, int x_dtype, const float* gamma, const float* beta, void* y,
                            int y_dtype, float* mean, float* rstd, int rows, int features, float eps);
int layer_norm_backward_impl(hl_ctx* ctx, const void* x, int x_dtype, const float* gamma, const float* dy,
                             const float* mean, const float* rstd, const float* residual_grad, float* dx_f32,
                             void* dx_bf16, float* dgamma, float* dbeta, float* dx_colsum, int rows, int features,
                             FoldBatch* defer = nullptr);
bool layer_norm_fast_applicable(int x_dtype, int y_dtype, int features, const void* x, const void* y);
int layer_norm_forward_fast(hl_ctx* ctx, const void* x, const float* gamma, const float* beta, void* y, float* mean,
                            float* rstd, int rows, int features, float eps);
int layer_norm_backward_fast(hl_ctx* ctx, const void* x, const float* gamma, const float* dy, const float* mean,
                             const float* rstd, const float* residual, float* dx_f32, void* dx_bf16, float* dgamma,
                             float* dbeta, float* dx_colsum, int rows, int features, FoldBatch* defer = nullptr);
bool colsum_fast_applicable(int dtype, int cols, const void* g);
int colsum_fast(hl_ctx* ctx, const void* g, int dtype, float* out, int rows, int cols, FoldBatch* defer = nullptr);
int cross_entropy_impl(hl_ctx* ctx, const float* logits, long long ld, const int64_t* targets, int rows, int classes,
                       float grad_scale, float* loss_dev, float* row_loss, void* dlogits, int dlogits_dtype,
                       long long ld_dlogits, float* loss_host = nullptr);

int flash_attention_forward_impl(hl_ctx* ctx, const void* q, const void* k, const void* v, long long ld_qkv, void* out,
                                 long long ld_out, float* lse, int batch, int time, int n_heads, int head_dim);
size_t flash_attention_backward_scratch_bytes(int batch, int time, int n_heads, int head_dim);
int flash_attention_backward_impl(hl_ctx* ctx, const void* q, const void* k, const void* v, long long ld_qkv,
                                  const void* out, long long ld_out, const void* dout, long long ld_dout,
                                  const float* lse, void* dq, void* dk, void* dv, long long ld_dqkv, int batch, int time,
                                  int n_heads, int head_dim, void* scratch, size_t scratch_bytes);

// One f32 product with f64 sums, out[i,j] = epilogue(sum_k A[i,k] * B[k,j]), element strides throughout (ref_f32.cu).  The
// product is rounded to f32, then the bias is added and rounded, then the epilogue acts, each step rounded as when it
// was an op of its own.
enum { F64_STORE = 0, F64_ACCUMULATE = 1 /* out += */, F64_GELU = 2 /* aux_out = gelu(out) */,
       F64_RESIDUAL = 3 /* out = aux_in + y */, F64_DGELU = 4 /* out = y * gelu'(aux_in) */ };
struct F64Gemm {
  const float *a, *b;
  float* out;
  long long a_row, a_col, b_row, b_col, o_row, o_col;
  int m, n, k;
  int epilogue;
  const float* bias;    // [n] or null
  const float* aux_in;  // laid out as out
  float* aux_out;
  float* row_sum;       // [m] or null: sum_k A[i,k]
};
// One or two independent products in one launch.
int f64_gemm_run(hl_ctx* ctx, const F64Gemm* problems, int count);

// Causal attention with f64 sums on f32 or bf16 rows with strides; `probs` [B,H,T,T] f32 is written by the forward.  The
// backward reads it for f32 operands and forms it again for bf16 ones.
int attention_f64_forward(hl_ctx* ctx, const void* q, const void* k, const void* v, int dtype, long long ld_qkv, void* out,
                          long long ld_out, float* probs, int batch, int time, int channels, int n_heads);
int attention_f64_backward(hl_ctx* ctx, const void* q, const void* k, const void* v, int dtype, long long ld_qkv, float* probs,
                           const void* dout, long long ld_dout, void* dq, void* dk, void* dv, long long ld_dqkv, int batch,
                           int time, int channels, int n_heads);

// One-token steps (decode.cu).  out[n] = epilogue(W[n,k] · x + bias), with a layer norm of x first when gamma is given.
enum { GV_STORE = 0, GV_GELU = 1, GV_RESIDUAL = 2 };
struct DecodeGemv {
  const void* x;
  int x_dtype;
  const void* w;
  int w_dtype;
  const float* bias;
  void* out;
  int out_dtype;
  int n, k;
  int epilogue;
  const float *gamma, *beta;
  const void* residual;      // of the output's type
  const long long* out_row;  // device: which row of `out` (row stride ld_out) is written; null: row 0
  long long ld_out;
};
int decode_gemv(hl_ctx* ctx, const DecodeGemv& g);
size_t decode_attention_smem(int dtype, int head_dim, int context);
// `settled`: the rows below the position were written before this sequence of launches began.
int decode_attention(hl_ctx* ctx, const void* qkv, int dtype, long long ld, const long long* pos, void* out, int channels,
                     int n_heads, int context, bool settled);
// The last maximum of a row of logits and the sum of exponentials below it, without taking the row to the host.  `parts` has
// room for greedy_parts(vocab) entries.
struct GreedyPart {
  double sum;  // of e^(x - max)
  float max;
  int index;   // of the last maximum, -1 when a value is not finite
};
inline int greedy_parts(int vocab) { return (vocab + 2047) / 2048; }
int decode_greedy(hl_ctx* ctx, const float* logits, int vocab, GreedyPart* parts, GreedyPart* out);
// Whether every one of n floats is finite; host function.
bool all_finite_f32(const float* x, size_t n);
int decode_embed(hl_ctx* ctx, const float* table, const float* positions, const long long* state, void* out, int dtype, int dim);

// The same in two kernels a block (decode_block.cu).  A row of the residual stream that no kernel has written yet: base + bias + the
// sum of `parts` rows, or what base holds (n = 0), or the embedding of the state's token (n = 0, base null).  The kernel that takes
// it also writes it to `keep`, where given.  Rows and `keep` are of the model's type, parts f32 on the bf16 route and f64 on the f32 one.
struct DecodeRow {
  const void* base;
  const void* parts;  // [n][d]
  int n;
  const float* bias;
  const float *table, *positions;
  const long long* state;
  void* keep;
};
struct DecodeBlock {
  int dtype, d, heads, hidden, context;
  const long long* state;  // device: position, token
  DecodeRow x;
  bool window;             // the q/k/v rows, this position's as well, come from the predecessor: x.base is only the residual
  const float *ln1_gamma, *ln1_beta;
  const void* wqkv;        // [3 d][d]
  const float* bqkv;
  void* qkv;               // rows of 3 d, those below the position settled before this sequence of launches began unless `window`
  const void* wo;
  const float* bo;
  const float *ln2_gamma, *ln2_beta;
  const void *w1, *w2;
  const float *b1, *b2;
  void *attention_parts, *feed_forward_parts;  // decode_block_parts_bytes each
};
bool decode_block_applies(int dtype, int d, int heads, int hidden, int context);
size_t decode_block_parts_bytes(int d);
// *after: the row behind the block's attention, behind its feed-forward (`x` needs a `keep`).
int decode_attention_block(hl_ctx* ctx, const DecodeBlock& b, DecodeRow* after);
int decode_feed_forward(hl_ctx* ctx, const DecodeBlock& b, const DecodeRow& x, DecodeRow* after);
// Writes the row to its `keep`.
int decode_row(hl_ctx* ctx, const DecodeRow& r, int dtype, int d);
// Final layer norm and head.
int decode_head_row(hl_ctx* ctx, const DecodeRow& x, int dtype, const float* gamma, const float* beta, const void* w, const float* bias,
                    float* out, int n, int d);

// bf16 pieces of f32 values (elementwise.cu): piece number id[j] of row r goes to out + r * ld + j * piece, for j < n; all multiples
// of 8 elements.  Pieces as split8_bf16 forms them.
struct PieceDest {
  __nv_bfloat16* out;
  long long ld, piece;
  int n, id[3];
};
// One below the other, [pieces * rows][cols], or side by side, rows of `ld` elements; the pieces in the order given.
inline PieceDest pieces_stacked(__nv_bfloat16* out, long long rows, int cols, int n, int i0, int i1, int i2 = 0) {
  return PieceDest{out, cols, rows * cols, n, {i0, i1, i2}};
}
inline PieceDest pieces_beside(__nv_bfloat16* out, long long ld, int cols, int n, int i0, int i1, int i2 = 0) {
  return PieceDest{out, ld, cols, n, {i0, i1, i2}};
}
// src [rows][cols], read once.  `b` may be empty (n = 0).  cols a multiple of 8, everything on 16 bytes.
int split_pieces(hl_ctx* ctx, const float* src, long long rows, int cols, const PieceDest& a, const PieceDest& b = PieceDest{});
// gate = gelu(gpre), mv = weighted * gate and mv's pieces; and backward: dweighted = dmv * gate, dgpre = gelu'(gpre) dmv weighted and
// its pieces.  Rounded to f32 after every operation, gelu in f64, as the single ops round.
int memory_gate_forward(hl_ctx* ctx, const float* gpre, const float* weighted, float* gate, float* mv, long long rows, int cols, const PieceDest& a);
int memory_gate_backward(hl_ctx* ctx, const float* dmv, const float* gate, const float* weighted, const float* gpre, float* dweighted, float* dgpre,
                         long long rows, int cols, const PieceDest& a, const PieceDest& b);

// Half-key gradients of the product-key form on the tensor cores (memory_keys.cu): *partial is where in the scratch the sums
// [shares][2][side][half] end up, one per share of the tokens.  Shares: 0 where this form does not apply.  The scratch's first word is
// zero before the call.
struct KeyGradient {
  const int64_t* idx;         // [tokens][top_k]
  const float* query;         // [tokens][2 * half], row stride ld_query
  long long ld_query;
  const float* grad_scores;   // [tokens][top_k]
  int tokens, top_k, side, half, slots;
};
int key_gradient_shares(const hl_ctx* ctx, const KeyGradient& k);
size_t key_gradient_bytes(const KeyGradient& k, int shares);
int key_gradient_run(hl_ctx* ctx, const KeyGradient& k, int shares, void* scratch, float** partial);

// hl_product_key_topk_from_side_scores whose choices go to rows *kept_row and on of `kept` as well (null: nowhere else).
int product_key_topk_impl(hl_ctx* ctx, const float* left_scores, const float* right_scores, int64_t* out, int tokens, int side, int top_k,
                          int beam, int64_t* kept, const long long* kept_row);

// Side scores and hl_product_key_topk_from_side_scores in one, with the selections of those two, for queries with rows of key_dim: the scores
// that can be selected are formed exactly, the others on the tensor cores.  `pieces` (product_key_pieces_bytes) come from the tables by
// product_key_pieces; query_pieces: tokens * 2 * key_dim; the approximate scores: tokens * side each; all on 16 bytes.
bool product_key_lookup_takes(int side, int key_dim, int beam);
size_t product_key_pieces_bytes(int side, int key_dim);
int product_key_pieces(hl_ctx* ctx, const float* left_keys, const float* right_keys, int side, int key_dim, void* pieces);
int product_key_lookup(hl_ctx* ctx, const float* query, const float* left_keys, const float* right_keys, const void* pieces,
                       __nv_bfloat16* query_pieces, float* left_approx, float* right_approx, int64_t* out, int tokens, int side, int key_dim,
                       int top_k, int beam);
// hl_memory_weighted_value_backward in two: the (token, slot) events sorted by row, which needs the indices alone, and the rest.  `keys`
// and `events` lie in value_sort_bytes, half each; rows that do not exist report themselves and zero their grad_weights (may be null).
bool value_events_ordered(long long n, int rows, int dim);
size_t value_sort_bytes(long long n);
size_t value_order_scratch_bytes(long long n);
int value_sort(hl_ctx* ctx, const int64_t* indices, long long n, int rows, int* keys, int* events, void* scratch, float* grad_weights);
int weighted_value_backward_ordered(hl_ctx* ctx, const int* keys, const int* events, const float* weights, const float* values,
                                    const float* grad_out, float* grad_weights, float* grad_values, long long n, int top_k, int rows, int dim);

struct AdamPlan;
int adam_plan_create(hl_ctx* ctx, const hl_adamw_tensor* tensors, int count, AdamPlan** out);
void adam_plan_destroy(AdamPlan* plan);
// hl_sum_squares_f32 whose result goes to pinned host memory as well.
int sum_squares_impl(hl_ctx* ctx, const float* x, size_t n, float* out_dev, float* out_host);
// Clipping by the global norm on the device: hp's clip_scale times min(1, limit / norm), norm the square root of *sum_sq times
// scale * scale.  Nothing is updated when that sum is not a finite non-negative number.
struct AdamClip {
  const float* sum_sq;  // device, null: no clipping
  double scale, limit;
};
int adam_plan_step(hl_ctx* ctx, AdamPlan* plan, const hl_adamw_params* hp, const AdamClip& clip = AdamClip{nullptr, 0.0, 0.0});
int adam_plan_step_range(hl_ctx* ctx, AdamPlan* plan, const hl_adamw_params* hp, int first, int count,
                         const AdamClip& clip = AdamClip{nullptr, 0.0, 0.0});
int adam_plan_chunk_elements(const AdamPlan* plan);
int adam_plan_chunk_count(const AdamPlan* plan);

extern "C" int hl_memory_copy_indices(hl_ctx* ctx, int64_t* host, const int64_t* dev, long long count);

// NCCL (loaded at run time); see nccl_ddp.cu.
int nccl_allreduce_sum_f32(hl_ctx* ctx, float* buf, size_t count, cudaStream_t stream);
int nccl_allreduce_max_u8(hl_ctx* ctx, unsigned char* buf, size_t count, cudaStream_t stream);
int mark_rows_on(hl_ctx* ctx, cudaStream_t stream, const int64_t* selected_rows, long long n_selected, const unsigned char* row_mask,
                 unsigned char* flags, int rows);
int mask_to_indices_on(hl_ctx* ctx, cudaStream_t stream, const unsigned char* mask, int rows, int64_t* out, int* count_dev);
int move_rows_on(hl_ctx* ctx, cudaStream_t stream, const float* src, const int64_t* idx, const int* count_dev, int n_max, int dim,
                 float* dst, bool scatter);
bool nccl_active(const hl_ctx* ctx);
int nccl_world(const hl_ctx* ctx);

}  // namespace hl
