// Training-step executor for the dense pre-LayerNorm decoder LM: forward, backward, bucketed
// gradient all-reduce overlapped with backward, and the fused AdamW update, on preplanned
// arenas.  It reproduces the reference's AMP-bf16 dataflow
//   MemoryTransformerLm::forward_amp_bf16 / loss_amp_bf16 (src/memory_transformer.rs:1636-1670),
//   block (src/memory_transformer.rs:1153-1172), attention (src/nn.rs:718-788),
//   feed-forward (src/nn.rs:873-884), Linear (src/nn.rs:338-450),
//   backward operand rounding (src/tensor/autograd.rs:593-851),
//   AdamW::step_mut (src/nn.rs:2156-2220) and the data-parallel exchange
//   AdamW::all_reduce_cuda_gradients_nccl (src/nn.rs:2083-2138)
// with every bf16 round trip of that path realised as "store the activation in bf16".
//
// Parameters live in one flat f32 arena (plus f32 gradients, AdamW moments and a bf16 shadow
// used as GEMM operands), ordered by the time their gradient becomes final in backward
// (lm_head first, embeddings last) so that fixed-size buckets of the gradient arena can be
// all-reduced on the collective stream while backward is still running.
#include <cmath>
#include <limits>
#include <cstring>
#include <string>
#include <vector>

#include "kernels.h"

namespace hl {
namespace {

constexpr size_t kAlignElems = 64;
inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct Slot {
  std::string name;
  size_t offset, numel;
  int rank;
  long long shape[2];
};

struct LayerOffsets {
  size_t w2, b2, w1, b1, ln2g, ln2b, wo, bo, wqkv, bqkv, ln1g, ln1b;
  // memory feed-forward blocks use these instead of w1/b1/w2/b2
  bool is_memory = false;
  size_t wq_m = 0, bq_m = 0, wg_m = 0, bg_m = 0, wout_m = 0, bout_m = 0;
  // bias of the projection that writes the block output (fc2 or the memory out_proj)
  size_t out_bias() const { return is_memory ? bout_m : b2; }
};

// Per memory layer: everything the backward needs (all f32, as in the reference the memory
// feed-forward runs in f32 also under AMP, src/memory_transformer.rs:787-789).
struct MemoryActs {
  float *query = nullptr, *weights = nullptr, *weighted = nullptr, *gpre = nullptr, *gate = nullptr, *mv = nullptr;
  int64_t* idx = nullptr;
  int *sorted_rows = nullptr, *sorted_events = nullptr;  // the selections in row order (value_sort); null: the backward pass sorts them
  __nv_bfloat16* mv_b = nullptr;  // amp route: [N, 2*value_dim] = [hi | lo] pieces of mv
  // amp route: the three projection weights as bf16 pieces along the contraction (hl_split_bf16_f32),
  // rebuilt from the f32 parameters at the start of every forward pass
  __nv_bfloat16 *wq3 = nullptr, *wg3 = nullptr, *wout3 = nullptr;
};

// A model's launch sequences as graphs.  A sequence that comes up a second time with the same sizes, scratch arena and GEMM
// settings is captured and from then on replayed: a small model's step is some sixty launches (and as many tensor maps) of
// 2 to 4 us of host time each for kernels of 2 to 5 us.  Everything a sequence reads and writes has a fixed address.
struct GraphKey {
  int kind, batch, context;
  const void* workspace;
  size_t workspace_bytes;
  unsigned long long wait_limit_ns;
  unsigned faults;
  char pairs, dynamic;  // first characters of the GEMM's environment settings
  bool operator==(const GraphKey& o) const {
    return kind == o.kind && batch == o.batch && context == o.context && workspace == o.workspace &&
           workspace_bytes == o.workspace_bytes && wait_limit_ns == o.wait_limit_ns && faults == o.faults && pairs == o.pairs &&
           dynamic == o.dynamic;
  }
};
enum { GRAPH_STEP = 0, GRAPH_LOSS = 1, GRAPH_WINDOW = 2, GRAPH_DECODE = 3, GRAPH_DECODE_GREEDY = 4,
       GRAPH_WINDOW_TO_HOST = 5 };
struct GraphEntry {
  GraphKey key{};
  cudaGraphExec_t exec = nullptr;  // null until the sequence has run once plainly
  bool plain = false;              // it could not be captured
  Counters counts{};               // what a replay adds to the context's counters
  unsigned long long used = 0;
};
struct GraphCache {
  std::vector<GraphEntry> entries;
  unsigned long long clock = 0;
  void clear() {
    for (GraphEntry& e : entries)
      if (e.exec) cudaGraphExecDestroy(e.exec);
    entries.clear();
  }
};
constexpr size_t kMaxGraphs = 6;

struct LayerActs {
  __nv_bfloat16 *a, *qkv, *o, *r, *c, *h, *g;
  __nv_bfloat16 *dy, *dh, *dr, *dqkv;  // bf16 gradients of the block output, h, r and qkv; shared by the layers unless forked
  float *lse, *mean1, *rstd1, *mean2, *rstd2;
};

}  // namespace
}  // namespace hl

using namespace hl;

struct hl_decoder {
  hl_ctx* ctx = nullptr;
  hl_decoder_config cfg{};
  int N = 0;
  // parameter arenas
  size_t arena = 0;
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16* shadow = nullptr;
  std::vector<Slot> slots;  // state-dict order
  size_t off_head_w = 0, off_head_b = 0, off_lnf_g = 0, off_lnf_b = 0, off_pos = 0, off_tok = 0;
  std::vector<LayerOffsets> lo;
  // activations
  uint8_t* act_arena = nullptr;
  size_t act_bytes = 0;
  std::vector<__nv_bfloat16*> x;  // x[l] is the input of block l; x[L] the final residual stream
  std::vector<LayerActs> la;
  __nv_bfloat16 *z = nullptr, *dlogits = nullptr, *dob = nullptr, *dxb0 = nullptr;
  // head sizes other than 64 and 128 on the bf16 route: attention runs through the f32 kernels, whose probabilities share
  // one buffer
  bool flash_ok = true;
  float* fa_probs = nullptr;
  float *logits = nullptr, *meanf = nullptr, *rstdf = nullptr, *dx0 = nullptr, *dx1 = nullptr, *dtmp = nullptr;
  int64_t *tokens = nullptr, *targets = nullptr;
  // Weight gradients beside the backward's chain of input gradients (they depend on it, nothing depends on them): on a second
  // stream, reading operands that every layer has its own copy of.
  bool lean = false;  // neither of the two below: no copies of operands
  bool fork_ok = false;
  cudaStream_t side_stream = nullptr;
  cudaEvent_t fork_event = nullptr, join_event = nullptr;
  cudaEvent_t zero_event = nullptr;  // the scattered gradients have been zeroed there
  cudaEvent_t sort_event = nullptr;  // the selections that the forward pass has left so far are in row order
  void* sort_scratch = nullptr;      // of those sorts, one at a time
  bool lookup = false;               // buffers for product_key_lookup are there (looks_up: whether a pass takes it)
  void* key_pieces = nullptr;        // of the half keys, made at the start of every pass
  __nv_bfloat16* query_pieces = nullptr;
  bool sorted = false;               // this pass sorts them there
  // a scratch arena for what runs there, in place of the context's
  void* side_arena = nullptr;
  size_t side_arena_bytes = 0;
  bool zeroed = false;
  // ... or, where the products fill the chip, collected for `group_layers` layers (0: not) and run by one launch.
  int group_layers = 0;
  std::vector<WeightGradJob> wgrads;
  float* group_sums = nullptr;
  bool forked = false;  // work has been queued on the side stream since the last join
  FoldBatch fold;  // column reductions of one block's backward, folded by one launch before its buckets are flushed
  float* loss_dev = nullptr;
  float* loss_host = nullptr;  // pinned
  float* norm_dev = nullptr;
  double* norm_dev64 = nullptr;  // f64 sum of squares over active sparse rows
  float* norm_host = nullptr;  // pinned
  // optimizer
  bool has_opt = false;
  hl_adamw_config opt{};
  long long step = 0;
  AdamPlan* plan = nullptr;
  // data-parallel buckets over the gradient arena
  size_t bucket_elems = 6553600;  // 25 MiB of f32
  size_t next_bucket = 0, n_buckets = 0;
  std::vector<cudaEvent_t> bucket_ready;
  std::vector<cudaEvent_t> bucket_done;  // recorded on the collective stream after each bucket's all-reduce
  bool comm_pending = false;             // the compute stream has not yet waited for this step's collectives
  cudaEvent_t comm_done = nullptr;
  // row-union exchanges: which rows the ranks touched is known long before their gradients are (the token ids when the
  // step starts, the selected slots when forward ends), so the union and its size are formed then, on the collective
  // stream, and the host finds the size ready when it queues the exchange itself at the end of backward
  cudaEvent_t rows_known = nullptr, tok_count_ready = nullptr, val_count_ready = nullptr;
  bool tok_prepared = false, val_prepared = false;
  // while per-kernel timing is on: events around every wait of the compute stream for the collective stream, so that
  // the time the step spends exposed to the gradient exchange can be read back (hl_decoder_comm_exposed_ms)
  std::vector<cudaEvent_t> wait_begin, wait_end;
  size_t waits_recorded = 0;
  unsigned long long launches_last_step = 0;
  // product-key memory (shared tables, MemoryTransformerLm with memory layers)
  bool has_memory = false;
  hl_memory_config mem{};
  int side = 0;
  size_t off_kl = 0, off_kr = 0, off_val = 0;
  size_t tables_end = 0;  // first arena element after the value table
  AdamPlan *plan_tables = nullptr, *plan_no_values = nullptr;  // the memory tables alone; everything but the value table
  std::vector<MemoryActs> ma;  // indexed by layer; empty entries for dense layers
  float *m_ls = nullptr, *m_rs = nullptr, *m_scores = nullptr, *m_dmv = nullptr, *m_dweighted = nullptr, *m_dgate = nullptr,
        *m_dgpre = nullptr, *m_dw = nullptr, *m_dscores = nullptr, *m_dq = nullptr;
  // amp route, backward of the three memory projections at f32 accuracy: bf16 pieces of the f32 operands, side by
  // side along the columns where the contraction runs along a row, one below the other where it runs down the rows
  __nv_bfloat16 *p_dx_side = nullptr, *p_dx_rows = nullptr, *p_mv_rows = nullptr, *p_dg_rows = nullptr, *p_dq_rows = nullptr,
                *p_dc_side = nullptr, *p_wout_rows = nullptr, *p_wc_rows = nullptr;
  unsigned char* m_row_flags = nullptr;
  unsigned char *smft_value_mask = nullptr, *smft_left_mask = nullptr, *smft_right_mask = nullptr;  // [slots], [side], [side]
  bool smft_on = false;  // the sparse-rows step filters its rows through the three masks
  float* m_packed = nullptr;         // gradient rows of the union, packed for the all-reduce (own allocation)
  size_t packed_rows_cap = 0;        // rows it holds
  // data-parallel exchange of the token-embedding gradient as the union of the rows any rank's batch touched
  bool sparse_tok_exchange = true;
  unsigned char* tok_flags = nullptr;  // [vocab]
  int64_t* tok_union_rows = nullptr;   // [vocab]
  int* tok_union_count = nullptr;
  int* tok_union_count_host = nullptr;  // pinned
  float* tok_packed = nullptr;
  size_t tok_packed_cap = 0;
  int64_t* m_union_rows = nullptr;   // rows of the value table selected by any rank this step
  int* m_union_count = nullptr;      // device count of them
  int* m_union_count_host = nullptr; // pinned mirror
  int union_n = -1;                  // rows in the union after the last exchange, -1 before any
  int64_t* decode_idx = nullptr;  // selections of a one-token step
  int64_t *m_sel_all = nullptr, *m_sel_left = nullptr, *m_sel_right = nullptr;  // concatenated selections of all memory blocks
  // f32 route (reference f32 semantics: f32 tensors, f64 accumulation inside every op)
  struct F32Layer {
    float *a, *qkv, *probs, *o, *r, *c, *h, *g;
    float *dy, *dr, *dqkv, *dwide;  // gradients of the block output, r, qkv and h; shared by the layers unless forked
  };
  // generation: how many positions of sequence 0 have their keys and values in the activation buffers (0: none) and the
  // state of the next one-token step
  int cached = 0;
  long long* decode_state = nullptr;       // device: position, token
  void* row_parts[2] = {};                 // device: what clusters add to the row, of attention and of the feed-forward
  bool head_twice = false;                 // this pass left the head's row sums instead of its logits
  float* row_logits = nullptr;             // where the logits of a single row go; null: m->logits
  GreedyPart* greedy = nullptr;            // device: the blocks' parts
  long long* decode_state_host = nullptr;  // pinned
  GreedyPart* greedy_host = nullptr;       // pinned
  float* logits_host = nullptr;            // pinned, [vocab], allocated on first use
  GraphCache graphs;
  std::vector<float*> xf;  // residual stream per block input, f32
  std::vector<F32Layer> lf;
  float *zf = nullptr, *dlogits_f = nullptr, *d_a = nullptr, *d_c = nullptr;
};

namespace hl {
namespace {

// Lays the parameters out in gradient-completion order and records the name -> slice map in
// the reference's state-dict order (src/memory_transformer.rs:2098-2117).
void plan_parameters(hl_decoder* m) {
  const hl_decoder_config& c = m->cfg;
  const long long d = c.d_model, F = c.d_ff, V = c.vocab, T = c.context;
  size_t cur = 0;
  std::vector<Slot> tmp;
  auto add = [&](const std::string& name, size_t numel, int rank, long long s0, long long s1) {
    const size_t off = cur;
    cur = align_up(cur + numel, kAlignElems);
    tmp.push_back(Slot{name, off, numel, rank, {s0, s1}});
    return off;
  };
  m->off_head_w = add("lm_head.weight", (size_t)V * d, 2, V, d);
  m->off_head_b = add("lm_head.bias", (size_t)V, 1, V, 0);
  m->off_lnf_g = add("ln_f.weight", (size_t)d, 1, d, 0);
  m->off_lnf_b = add("ln_f.bias", (size_t)d, 1, d, 0);
  m->lo.resize(c.n_layers);
  for (int l = c.n_layers - 1; l >= 0; --l) {
    const std::string b = "block." + std::to_string(l) + ".";
    LayerOffsets& o = m->lo[l];
    o.is_memory = false;
    for (int i = 0; m->has_memory && i < m->mem.n_memory_layers; ++i) o.is_memory |= m->mem.memory_layers[i] == l;
    if (o.is_memory) {
      const long long kd = m->mem.key_dim, vd = m->mem.value_dim;
      const std::string f = b + "feed_forward.memory.";
      o.wout_m = add(f + "out_proj.weight", (size_t)d * vd, 2, d, vd);
      o.bout_m = add(f + "out_proj.bias", (size_t)d, 1, d, 0);
      o.wg_m = add(f + "gate_proj.weight", (size_t)vd * d, 2, vd, d);
      o.bg_m = add(f + "gate_proj.bias", (size_t)vd, 1, vd, 0);
      o.wq_m = add(f + "query_proj.weight", (size_t)kd * d, 2, kd, d);
      o.bq_m = add(f + "query_proj.bias", (size_t)kd, 1, kd, 0);
      o.w2 = o.b2 = o.w1 = o.b1 = 0;
    } else {
    o.w2 = add(b + "feed_forward.dense.fc2.weight", (size_t)d * F, 2, d, F);
    o.b2 = add(b + "feed_forward.dense.fc2.bias", (size_t)d, 1, d, 0);
    o.w1 = add(b + "feed_forward.dense.fc1.weight", (size_t)F * d, 2, F, d);
    o.b1 = add(b + "feed_forward.dense.fc1.bias", (size_t)F, 1, F, 0);
    }
    o.ln2g = add(b + "ln2.weight", (size_t)d, 1, d, 0);
    o.ln2b = add(b + "ln2.bias", (size_t)d, 1, d, 0);
    o.wo = add(b + "attention.out_proj.weight", (size_t)d * d, 2, d, d);
    o.bo = add(b + "attention.out_proj.bias", (size_t)d, 1, d, 0);
    // q, k, v are three reference Linears stored back to back so one [3d, d] GEMM serves them
    o.wqkv = cur;
    add(b + "attention.q_proj.weight", (size_t)d * d, 2, d, d);
    cur = o.wqkv + (size_t)d * d;
    add(b + "attention.k_proj.weight", (size_t)d * d, 2, d, d);
    cur = o.wqkv + 2 * (size_t)d * d;
    add(b + "attention.v_proj.weight", (size_t)d * d, 2, d, d);
    o.bqkv = cur;
    add(b + "attention.q_proj.bias", (size_t)d, 1, d, 0);
    cur = o.bqkv + d;
    add(b + "attention.k_proj.bias", (size_t)d, 1, d, 0);
    cur = o.bqkv + 2 * d;
    add(b + "attention.v_proj.bias", (size_t)d, 1, d, 0);
    o.ln1g = add(b + "ln1.weight", (size_t)d, 1, d, 0);
    o.ln1b = add(b + "ln1.bias", (size_t)d, 1, d, 0);
  }
  if (m->has_memory) {
    const long long half = m->mem.key_dim / 2;
    m->off_kl = add("shared_memory.product_key_left", (size_t)m->side * half, 2, m->side, half);
    m->off_kr = add("shared_memory.product_key_right", (size_t)m->side * half, 2, m->side, half);
    m->off_val = add("shared_memory.value", (size_t)m->mem.slots * m->mem.value_dim, 2, m->mem.slots, m->mem.value_dim);
    m->tables_end = cur;
  }
  m->off_pos = add("position_embedding.weight", (size_t)T * d, 2, T, d);
  m->off_tok = add("token_embedding.weight", (size_t)V * d, 2, V, d);
  m->arena = cur;
  // state-dict order
  auto find = [&](const std::string& n) -> Slot {
    for (const Slot& s : tmp) if (s.name == n) return s;
    return Slot{};
  };
  m->slots.push_back(find("token_embedding.weight"));
  m->slots.push_back(find("position_embedding.weight"));
  if (m->has_memory)
    for (const char* n : {"shared_memory.product_key_left", "shared_memory.product_key_right", "shared_memory.value"})
      m->slots.push_back(find(n));
  for (int l = 0; l < c.n_layers; ++l) {
    const std::string b = "block." + std::to_string(l) + ".";
    for (const char* n : {"ln1.weight", "ln1.bias", "attention.q_proj.weight", "attention.q_proj.bias",
                          "attention.k_proj.weight", "attention.k_proj.bias", "attention.v_proj.weight",
                          "attention.v_proj.bias", "attention.out_proj.weight", "attention.out_proj.bias", "ln2.weight",
                          "ln2.bias"})
      m->slots.push_back(find(b + n));
    if (m->lo[l].is_memory) {
      for (const char* n : {"feed_forward.memory.query_proj.weight", "feed_forward.memory.query_proj.bias",
                            "feed_forward.memory.gate_proj.weight", "feed_forward.memory.gate_proj.bias",
                            "feed_forward.memory.out_proj.weight", "feed_forward.memory.out_proj.bias"})
        m->slots.push_back(find(b + n));
    } else {
      for (const char* n : {"feed_forward.dense.fc1.weight", "feed_forward.dense.fc1.bias", "feed_forward.dense.fc2.weight",
                            "feed_forward.dense.fc2.bias"})
        m->slots.push_back(find(b + n));
    }
  }
  for (const char* n : {"ln_f.weight", "ln_f.bias", "lm_head.weight", "lm_head.bias"}) m->slots.push_back(find(n));
}

template <typename T>
T* carve(uint8_t*& cursor, size_t count) {
  T* p = reinterpret_cast<T*>(cursor);
  cursor += align_up(count * sizeof(T), 256);
  return p;
}

hl_gemm_desc product(int M, int N, int K, int al, long long lda, int bl, long long ldb, int a_k_period, int b_k_period) {
  hl_gemm_desc d{};
  d.m = M; d.n = N; d.k = K;
  d.a_layout = al; d.b_layout = bl;
  d.lda = lda; d.ldb = ldb; d.ldc = N;
  d.out_dtype = HL_F32;
  d.a_k_period = a_k_period; d.b_k_period = b_k_period;
  return d;
}
// The weight gradients of a memory block's three projections (amp route).
hl_gemm_desc out_gradient(const hl_decoder* m) {
  return product(m->cfg.d_model, m->mem.value_dim, 3 * m->N, HL_MN_MAJOR, m->cfg.d_model, HL_MN_MAJOR, m->mem.value_dim, 2 * m->N, 0);
}
hl_gemm_desc in_gradient(const hl_decoder* m, int width) {
  return product(width, m->cfg.d_model, 3 * m->N, HL_MN_MAJOR, width, HL_MN_MAJOR, m->cfg.d_model, 0, m->N);
}
KeyGradient key_gradient(const hl_decoder* m) {
  KeyGradient k{};
  k.ld_query = m->mem.key_dim;
  k.tokens = m->N; k.top_k = m->mem.top_k; k.side = m->side; k.half = m->mem.key_dim / 2; k.slots = m->mem.slots;
  return k;
}
// Scratch for what a memory block's backward pass puts on the side stream.
size_t memory_side_bytes(const hl_decoder* m) {
  size_t most = 0, bytes = 0;
  if (m->cfg.precision == HL_PRECISION_AMP_BF16)
    for (const hl_gemm_desc& d : {out_gradient(m), in_gradient(m, m->mem.value_dim), in_gradient(m, m->mem.key_dim)})
      if (gemm_bf16_scratch(m->ctx, &d, &bytes)) most = std::max(most, bytes);
  const KeyGradient k = key_gradient(m);
  if (const int shares = key_gradient_shares(m->ctx, k)) most = std::max(most, key_gradient_bytes(k, shares));
  return most;
}

// Whether a pass selects by the lookup.  Exact scores of all keys cost tokens * side * key_dim products, sides in tiles of 128, and no less than one
// tile's walk along the keys, which few tokens feel; the lookup costs three products of the pieces, a pass over all approximate scores and
// top_k exact products a side.  us a block and pass, lookup less all keys (two blocks of a two-layer model, top_k 4 / 32):
//     tokens            1024        2048        4096        8192       16384
//     side 512, 512    -56 / -50   -61 / -50   -65 / -43   -99 / -60  -222 / -149
//     side 256, 256    -29 / -31   -25 / -25   -18 / -9    -19 / +6    -14 / +29
//     side 128, 512    -22 / -27   -55 / -43   -43 / -18   -20 / +19    -7 / +67
//     side 128, 128     -7 / -3    -11 / -8     -6 / +2     +2 / +18   +12 / +40
//     side 32, 64                                +5 / +1     +7 / +12   +18 / +20
// Below 2^24 products it is the launches that count (256 tokens, sides of 128 and keys of 256: -1 / +5).  It is the pass's own tokens that count: a prompt
// may be far shorter than the model's batch.
constexpr size_t kLookupProducts = size_t(1) << 24;  // tokens * side * key_dim
bool looks_up(const hl_decoder* m) {
  const double n = m->N, side = m->side, kd = m->mem.key_dim, k = m->mem.top_k;
  return m->lookup && n * side * kd >= (double)kLookupProducts &&
         (1.0 + 1.6 * (4096.0 / n) * (4096.0 / n)) * std::max(side, 128.0) * kd > 16000.0 + (100.0 + 4.0 * k) * kd + 60.0 * side;
}

// Buffers of the memory feed-forward blocks; appended to either route's arena.
void plan_memory_buffers(hl_decoder* m, uint8_t*& cur) {
  m->tok_flags = carve<unsigned char>(cur, (size_t)m->cfg.vocab);
  m->tok_union_rows = carve<int64_t>(cur, (size_t)m->cfg.vocab);
  m->tok_union_count = carve<int>(cur, 4);
  if (!m->has_memory) return;
  const size_t N = (size_t)m->N, kd = m->mem.key_dim, vd = m->mem.value_dim, k = m->mem.top_k, d = m->cfg.d_model;
  m->ma.assign(m->cfg.n_layers, MemoryActs{});
  for (int l = 0; l < m->cfg.n_layers; ++l) {
    if (!m->lo[l].is_memory) continue;
    MemoryActs& a = m->ma[l];
    a.query = carve<float>(cur, N * kd);
    a.weights = carve<float>(cur, N * k);
    a.weighted = carve<float>(cur, N * vd);
    a.gpre = carve<float>(cur, N * vd);
    a.gate = carve<float>(cur, N * vd);
    a.mv = carve<float>(cur, N * vd);
    a.idx = carve<int64_t>(cur, N * k);
    a.mv_b = carve<__nv_bfloat16>(cur, N * 2 * vd);
    a.wq3 = carve<__nv_bfloat16>(cur, kd * 3 * d);
    a.wg3 = carve<__nv_bfloat16>(cur, vd * 3 * d);
    a.wout3 = carve<__nv_bfloat16>(cur, d * 3 * vd);
    a.sorted_rows = a.sorted_events = nullptr;
    if (!m->lean && value_events_ordered((long long)(N * k), m->mem.slots, (int)vd)) {
      a.sorted_rows = reinterpret_cast<int*>(carve<uint8_t>(cur, value_sort_bytes((long long)(N * k))));
      a.sorted_events = a.sorted_rows + value_sort_bytes((long long)(N * k)) / 2 / sizeof(int);
    }
  }
  m->sort_scratch = m->lean ? nullptr : carve<uint8_t>(cur, value_order_scratch_bytes((long long)(N * k)));
  m->side_arena_bytes = m->lean ? 0 : memory_side_bytes(m);
  m->side_arena = m->side_arena_bytes ? carve<uint8_t>(cur, m->side_arena_bytes) : nullptr;
  m->m_ls = carve<float>(cur, N * m->side);
  m->m_rs = carve<float>(cur, N * m->side);
  m->m_scores = carve<float>(cur, N * k);
  m->m_dmv = carve<float>(cur, N * vd);
  m->m_dweighted = carve<float>(cur, N * vd);
  m->m_dgpre = carve<float>(cur, N * vd);
  m->m_dw = carve<float>(cur, N * k);
  m->m_dscores = carve<float>(cur, N * k);
  m->m_dq = carve<float>(cur, N * kd);
  m->lookup = !m->lean && N * m->side * kd >= kLookupProducts && product_key_lookup_takes(m->side, (int)kd, (int)k);
  if (m->cfg.precision == HL_PRECISION_AMP_BF16) {
    m->p_dx_side = carve<__nv_bfloat16>(cur, N * 2 * d);
    m->p_dx_rows = carve<__nv_bfloat16>(cur, 2 * N * d);
    m->p_mv_rows = carve<__nv_bfloat16>(cur, 3 * N * vd);
    m->p_dg_rows = carve<__nv_bfloat16>(cur, 3 * N * vd);
    m->p_dc_side = carve<__nv_bfloat16>(cur, N * 2 * (vd + kd));
    m->p_dq_rows = carve<__nv_bfloat16>(cur, 3 * N * kd);
    m->p_wout_rows = carve<__nv_bfloat16>(cur, 3 * d * vd);
    m->p_wc_rows = carve<__nv_bfloat16>(cur, 3 * (vd + kd) * d);
    m->query_pieces = m->p_dc_side;  // (the backward pass comes later)
  } else {
    m->m_dgate = carve<float>(cur, N * vd);
    if (m->lookup) m->query_pieces = carve<__nv_bfloat16>(cur, N * 2 * kd);
  }
  if (m->lookup) m->key_pieces = carve<uint8_t>(cur, product_key_pieces_bytes(m->side, (int)kd));
  m->m_row_flags = carve<unsigned char>(cur, (size_t)m->mem.slots);
  m->smft_value_mask = carve<unsigned char>(cur, (size_t)m->mem.slots);
  m->smft_left_mask = carve<unsigned char>(cur, (size_t)m->side);
  m->smft_right_mask = carve<unsigned char>(cur, (size_t)m->side);
  m->m_union_rows = carve<int64_t>(cur, (size_t)m->mem.slots);
  m->m_union_count = carve<int>(cur, 4);
  // room for this rank's selections of every memory block, or for the union of all ranks' (at most every slot)
  const size_t all = std::max(N * k * (size_t)m->mem.n_memory_layers, (size_t)m->mem.slots);
  m->m_sel_all = carve<int64_t>(cur, all);
  m->m_sel_left = carve<int64_t>(cur, all);
  m->m_sel_right = carve<int64_t>(cur, all);
  m->decode_idx = carve<int64_t>(cur, k);
}

// Operand copies of a step whose weight gradients may run beside the chain of input gradients: what a model of a few
// thousand tokens needs.  Above it the products fill the chip and the copies would be gigabytes.
constexpr size_t kForkBytes = size_t(256) << 20;

// Weight gradients of how many layers one launch takes (0: each for itself).  As many as leave the fewest waves of tiles over the
// whole backward pass (the head's product goes with the first group), the fewest layers among those: each has its own copy of
// the gradients that the products read, which kGroupBytes bounds.
constexpr size_t kGroupBytes = size_t(1) << 30;
int plan_group_layers(const hl_decoder* m) {
  const hl_decoder_config& c = m->cfg;
  const int d = c.d_model, F = c.d_ff, L = c.n_layers, pairs = std::max(1, m->ctx->sm_count / 2);
  if (d % 8 != 0 || F % 8 != 0 || c.vocab % 8 != 0) return 0;
  const size_t per_layer = (size_t)m->N * (F + 5 * d) * 2;
  const int most = (int)std::min<size_t>({(size_t)L, std::max<size_t>(1, kGroupBytes / per_layer), (size_t)(kMaxGroupJobs - 1) / 4});
  const int attention = gemm_group_tiles(3 * d, d) + gemm_group_tiles(d, d), ffn = gemm_group_tiles(F, d) + gemm_group_tiles(d, F);
  int best = 0, best_waves = 0;
  for (int g = 1; g <= most; ++g) {
    int waves = 0;
    for (int top = L; top > 0; top -= g) {
      int tiles = top == L ? gemm_group_tiles(c.vocab, d) : 0;
      for (int l = std::max(0, top - g); l < top; ++l) tiles += attention + (m->lo[l].is_memory ? 0 : ffn);
      waves += ceil_div(tiles, pairs);
    }
    if (best == 0 || waves < best_waves) { best = g; best_waves = waves; }
  }
  return best;
}

int plan_activations(hl_decoder* m, bool measure_only, size_t* bytes_out) {
  const hl_decoder_config& c = m->cfg;
  const size_t N = (size_t)m->N, d = c.d_model, F = c.d_ff, V = c.vocab, L = c.n_layers;
  uint8_t* cur = measure_only ? nullptr : m->act_arena;
  uint8_t* base = cur;
  m->x.resize(L + 1);
  m->la.resize(L);
  for (size_t l = 0; l <= L; ++l) m->x[l] = carve<__nv_bfloat16>(cur, N * d);
  for (size_t l = 0; l < L; ++l) {
    LayerActs& a = m->la[l];
    a.a = carve<__nv_bfloat16>(cur, N * d);
    a.qkv = carve<__nv_bfloat16>(cur, N * 3 * d);
    a.o = carve<__nv_bfloat16>(cur, N * d);
    a.r = carve<__nv_bfloat16>(cur, N * d);
    a.c = carve<__nv_bfloat16>(cur, N * d);
    a.h = carve<__nv_bfloat16>(cur, N * F);
    a.g = carve<__nv_bfloat16>(cur, N * F);
    a.lse = carve<float>(cur, N * c.n_heads);
    a.mean1 = carve<float>(cur, N);
    a.rstd1 = carve<float>(cur, N);
    a.mean2 = carve<float>(cur, N);
    a.rstd2 = carve<float>(cur, N);
  }
  m->z = carve<__nv_bfloat16>(cur, N * d);
  m->meanf = carve<float>(cur, N);
  m->rstdf = carve<float>(cur, N);
  m->logits = carve<float>(cur, N * V);
  m->dlogits = carve<__nv_bfloat16>(cur, N * V);
  m->dx0 = carve<float>(cur, N * d);
  m->dx1 = carve<float>(cur, N * d);
  m->dtmp = carve<float>(cur, N * d);
  m->dob = carve<__nv_bfloat16>(cur, N * d);
  m->dxb0 = carve<__nv_bfloat16>(cur, N * d);  // gradient of the embeddings' sum: written like a block output's, read by nobody
  m->fork_ok = !m->lean && N * (F + 5 * d) * 2 * L <= kForkBytes;
  m->group_layers = m->lean || m->fork_ok ? 0 : plan_group_layers(m);
  {
    // one set of gradients per layer, per layer of a group, or for all; a group's last layer writes the next one's dy already
    const size_t sets = m->fork_ok ? L : std::max(1, m->group_layers), dy_sets = m->fork_ok ? L : std::min(L, sets + (m->group_layers > 0));
    for (size_t i = 0; i < L; ++i) {  // the order of the backward pass
      LayerActs& a = m->la[L - 1 - i];
      a.dy = i < dy_sets ? carve<__nv_bfloat16>(cur, N * d) : m->la[L - 1 - i % dy_sets].dy;
      if (i >= sets) {
        const LayerActs& first = m->la[L - 1 - i % sets];
        a.dh = first.dh; a.dr = first.dr; a.dqkv = first.dqkv;
        continue;
      }
      a.dh = carve<__nv_bfloat16>(cur, N * F);
      a.dr = carve<__nv_bfloat16>(cur, N * d);
      a.dqkv = carve<__nv_bfloat16>(cur, N * 3 * d);
    }
  }
  if (m->group_layers > 0)  // biases of the head, of fc1 and of qkv
    m->group_sums = carve<float>(cur, gemm_group_sums(V, d) + m->group_layers * (gemm_group_sums(F, d) + gemm_group_sums(3 * d, d)));
  if (!m->flash_ok) {
    m->fa_probs = carve<float>(cur, (size_t)c.batch * c.n_heads * c.context * c.context);
  }
  plan_memory_buffers(m, cur);
  {
    // partial rows of the column reductions: two layer norms (at most 2 CTAs per SM, three sums each) and the bias
    // column sums (at most 64 slabs) of one block, or the head's
    const size_t sm = (size_t)m->ctx->sm_count;
    const size_t ln = 2 * sm * 3 * d + 64;
    const size_t wide = m->has_memory ? std::max(F, (size_t)(m->mem.key_dim + m->mem.value_dim)) : F;
    const size_t layer = 2 * ln + 64 * (wide + 3 * d) + 4 * 64;
    const size_t head = ln + 64 * V + 2 * 64;
    m->fold.capacity = std::max(4 * layer, head);  // several layers' reductions wait for one fold
    m->fold.scratch = carve<float>(cur, m->fold.capacity);
    m->fold.n = 0;
    m->fold.used = 0;
  }
  m->tokens = carve<int64_t>(cur, N);
  m->targets = carve<int64_t>(cur, N);
  m->decode_state = carve<long long>(cur, 2);
  m->row_parts[0] = carve<uint8_t>(cur, decode_block_parts_bytes(c.d_model));
  m->row_parts[1] = carve<uint8_t>(cur, decode_block_parts_bytes(c.d_model));
  m->greedy = carve<GreedyPart>(cur, greedy_parts(c.vocab));
  m->loss_dev = carve<float>(cur, 4);
  m->norm_dev = carve<float>(cur, 4);
  m->norm_dev64 = carve<double>(cur, 2);
  *bytes_out = (size_t)(cur - base);
  return HL_OK;
}

int plan_activations_f32(hl_decoder* m, bool measure_only, size_t* bytes_out) {
  const hl_decoder_config& c = m->cfg;
  const size_t N = (size_t)m->N, d = c.d_model, F = c.d_ff, V = c.vocab, L = c.n_layers;
  const size_t BHTT = (size_t)c.batch * c.n_heads * c.context * c.context;
  uint8_t* cur = measure_only ? nullptr : m->act_arena;
  uint8_t* base = cur;
  m->xf.resize(L + 1);
  m->lf.resize(L);
  for (size_t l = 0; l <= L; ++l) m->xf[l] = carve<float>(cur, N * d);
  for (size_t l = 0; l < L; ++l) {
    hl_decoder::F32Layer& a = m->lf[l];
    a.a = carve<float>(cur, N * d);
    a.qkv = carve<float>(cur, N * 3 * d);
    a.probs = carve<float>(cur, BHTT);
    a.o = carve<float>(cur, N * d);
    a.r = carve<float>(cur, N * d);
    a.c = carve<float>(cur, N * d);
    a.h = carve<float>(cur, N * F);
    a.g = carve<float>(cur, N * F);
  }
  m->zf = carve<float>(cur, N * d);
  m->logits = carve<float>(cur, N * V);
  m->dlogits_f = carve<float>(cur, N * V);
  m->d_a = carve<float>(cur, N * d);
  m->d_c = carve<float>(cur, N * d);
  m->fork_ok = !m->lean && !m->has_memory && N * (F + 5 * d) * sizeof(float) * L <= kForkBytes;  // (memory blocks share theirs)
  for (size_t l = 0; l < L; ++l) {
    hl_decoder::F32Layer& a = m->lf[l];
    if (l > 0 && !m->fork_ok) {
      a.dy = m->lf[0].dy; a.dr = m->lf[0].dr; a.dqkv = m->lf[0].dqkv; a.dwide = m->lf[0].dwide;
      continue;
    }
    a.dy = m->fork_ok ? carve<float>(cur, N * d) : m->d_a;
    a.dr = carve<float>(cur, N * d);
    a.dqkv = carve<float>(cur, N * 3 * d);
    a.dwide = carve<float>(cur, N * F);
  }
  plan_memory_buffers(m, cur);
  // partial rows of a full batch of layer norms' parameter gradients (at most two CTAs per SM, two sums each)
  m->fold.capacity = (size_t)FoldBatch::kMaxJobs * (2 * (size_t)m->ctx->sm_count * 2 * d + 64);
  m->fold.scratch = carve<float>(cur, m->fold.capacity);
  m->fold.n = 0;
  m->fold.used = 0;
  m->tokens = carve<int64_t>(cur, N);
  m->targets = carve<int64_t>(cur, N);
  m->decode_state = carve<long long>(cur, 2);
  m->row_parts[0] = carve<uint8_t>(cur, decode_block_parts_bytes(c.d_model));
  m->row_parts[1] = carve<uint8_t>(cur, decode_block_parts_bytes(c.d_model));
  m->greedy = carve<GreedyPart>(cur, greedy_parts(c.vocab));
  m->loss_dev = carve<float>(cur, 4);
  m->norm_dev = carve<float>(cur, 4);
  m->norm_dev64 = carve<double>(cur, 2);
  *bytes_out = (size_t)(cur - base);
  return HL_OK;
}

struct Gemm {
  hl_decoder* m;
  int run(int M, int N, int K, const void* a, long long lda, int al, const void* b, long long ldb, int bl, void* c,
          long long ldc, int out_dtype, int epi = HL_EPI_NONE, const float* bias = nullptr, const void* aux_in = nullptr,
          long long ld_aux_in = 0, void* aux_out = nullptr, long long ld_aux_out = 0, int a_k_period = 0,
          int b_k_period = 0) const {
    hl_gemm_desc d{};
    d.m = M; d.n = N; d.k = K;
    d.a_k_period = a_k_period;
    d.b_k_period = b_k_period;
    d.a_layout = al; d.b_layout = bl;
    d.lda = lda; d.ldb = ldb; d.ldc = ldc;
    d.epilogue = epi; d.out_dtype = out_dtype; d.split_k = 0;
    d.ld_aux_in = ld_aux_in; d.ld_aux_out = ld_aux_out;
    return gemm_bf16_ctx(m->ctx, &d, a, b, c, bias, aux_in, aux_out);
  }
};

#define HL_TRY(expr)            \
  do {                          \
    int _rc = (expr);           \
    if (_rc != HL_OK) return _rc; \
  } while (0)

// While one of these lives, launches of the context go to the side stream, which first waits for everything queued on the
// compute stream so far.
struct SideStream {
  hl_decoder* m;
  cudaStream_t main;
  int rc = HL_OK;
  explicit SideStream(hl_decoder* model) : m(model), main(model->ctx->stream) {
    cudaError_t e = cudaEventRecord(m->fork_event, main);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(m->side_stream, m->fork_event, 0);
    if (e != cudaSuccess) rc = fail_cuda(e, "fork to the side stream");
    m->ctx->stream = m->side_stream;
    m->forked = true;
  }
  ~SideStream() { m->ctx->stream = main; }
};

// The same with a scratch arena of its own.
struct SideWork : SideStream {
  explicit SideWork(hl_decoder* model) : SideStream(model) { swap(); }
  ~SideWork() { swap(); }
 private:
  void swap() {
    std::swap(m->ctx->workspace, m->side_arena);
    std::swap(m->ctx->workspace_bytes, m->side_arena_bytes);
  }
};

int join_side(hl_decoder* m) {
  if (!m->forked) return HL_OK;
  m->forked = false;
  HL_CUDA(cudaEventRecord(m->join_event, m->side_stream));
  HL_CUDA(cudaStreamWaitEvent(m->ctx->stream, m->join_event, 0));
  return HL_OK;
}

int zero_memory_table_grads(hl_decoder* m) {
  if (!m->has_memory) return HL_OK;
  const size_t count = m->off_val + (size_t)m->mem.slots * m->mem.value_dim - m->off_kl;
  HL_CUDA(cudaMemsetAsync(m->grads + m->off_kl, 0, sizeof(float) * count, m->ctx->stream));
  return HL_OK;
}

bool beside(const hl_decoder* m) { return m->side_stream && !nccl_active(m->ctx) && !m->ctx->profiler; }

// Gradients that are sums over scattered rows (embeddings, memory tables) start at zero: zeroed beside the forward pass, which
// does not look at them, so that 20 MB or 540 MB of them do not stand between two kernels of the backward pass.
int zero_tables(hl_decoder* m) {
  HL_TRY(zero_memory_table_grads(m));
  HL_CUDA(cudaMemsetAsync(m->grads + m->off_pos, 0, sizeof(float) * (m->arena - m->off_pos), m->ctx->stream));
  return HL_OK;
}
int zero_tables_beside(hl_decoder* m) {
  m->zeroed = beside(m);
  if (!m->zeroed) return HL_OK;
  SideStream side(m);
  HL_TRY(side.rc);
  HL_TRY(zero_tables(m));
  HL_CUDA(cudaEventRecord(m->zero_event, m->ctx->stream));
  return HL_OK;
}
// Before the first of those gradients is added to.
int tables_are_zero(hl_decoder* m) {
  if (!m->zeroed) return zero_tables(m);
  HL_CUDA(cudaStreamWaitEvent(m->ctx->stream, m->zero_event, 0));
  return HL_OK;
}

// Collected weight gradients are not final when their layer is done, so not while buckets of them are being exchanged.
bool grouping(const hl_decoder* m) { return m->group_layers > 0 && !nccl_active(m->ctx); }
int run_weight_gradients(hl_decoder* m) {
  const int rc = gemm_group_run(m->ctx, m->wgrads.data(), (int)m->wgrads.size(), m->N, m->group_sums, &m->fold);
  m->wgrads.clear();
  return rc;
}

// dw[n_out, n_in] = dyᵀ · x and, when asked for, db = column sums of dy (both bf16, one row per token)
int weight_gradient(hl_decoder* m, const __nv_bfloat16* dy, int n_out, const __nv_bfloat16* x, int n_in, float* dw, float* db) {
  hl_gemm_desc d{};
  d.m = n_out; d.n = n_in; d.k = m->N;
  d.a_layout = HL_MN_MAJOR; d.b_layout = HL_MN_MAJOR;
  d.lda = n_out; d.ldb = n_in; d.ldc = n_in;
  d.epilogue = HL_EPI_NONE; d.out_dtype = HL_F32;
  if (grouping(m)) {
    m->wgrads.push_back(WeightGradJob{dy, x, n_out, n_in, dw, db});
    return HL_OK;
  }
  bool done = false;
  if (gemm_bf16_small_applies(m->ctx, &d)) {
    // no scratch arena on this path, so it may run on either stream
    if (m->fork_ok && !nccl_active(m->ctx) && !m->ctx->profiler) {
      SideStream side(m);
      HL_TRY(side.rc);
      return gemm_bf16_row_sums(m->ctx, &d, dy, x, dw, db, &done);
    }
    return gemm_bf16_row_sums(m->ctx, &d, dy, x, dw, db, &done);
  }
  HL_TRY(gemm_bf16_ctx(m->ctx, &d, dy, x, dw, nullptr, nullptr, nullptr));
  return db ? bias_grad_impl(m->ctx, dy, HL_BF16, db, m->N, n_out, &m->fold) : HL_OK;
}

// ---- memory feed-forward core (both routes): lookup, re-scoring, softmax, weighted value -----------
// query [N, key_dim] f32 is already in ma[l].query (MemoryFeedForward::forward_named,
// src/memory_transformer.rs:742-781).
// In a one-token step the block's selections of the window stay, with this position's in the position's row, as a full-window
// pass would leave them: they are read by others.
int memory_core_forward(hl_decoder* m, int l, bool one_token = false) {
  hl_ctx* ctx = m->ctx;
  MemoryActs& a = m->ma[l];
  int64_t* idx = one_token ? m->decode_idx : a.idx;
  const float* P = m->params;
  const int N = m->N, kd = m->mem.key_dim, vd = m->mem.value_dim, k = m->mem.top_k, side = m->side;
  const int beam = std::min(side, std::max(k, (int)ceil(sqrt((double)k))));  // product_key_beam, :2014-2016
  if (!one_token && looks_up(m)) {
    HL_TRY(product_key_lookup(ctx, a.query, P + m->off_kl, P + m->off_kr, m->key_pieces, m->query_pieces, m->m_ls, m->m_rs, idx, N, side, kd, k, beam));
  } else {
    ProfileScope prof(ctx, HL_PROF_OTHER, 2.0 * (double)N * side * 4.0);
    HL_TRY(hl_product_key_side_scores_f32(ctx, a.query, kd, P + m->off_kl, P + m->off_kr, m->m_ls, m->m_rs, N, side, kd));
    HL_TRY(product_key_topk_impl(ctx, m->m_ls, m->m_rs, idx, N, side, k, beam, one_token ? a.idx : nullptr, m->decode_state));
  }
  // timed as one family ("other" in the per-kernel profile); work = table rows gathered, in bytes
  ProfileScope prof(ctx, HL_PROF_OTHER, (double)N * k * (double)(kd + vd) * 4.0);
  if (m->sorted && a.sorted_rows) {  // for the backward pass, beside what follows
    SideStream beside(m);
    HL_TRY(beside.rc);
    HL_TRY(value_sort(ctx, idx, (long long)N * k, m->mem.slots, a.sorted_rows, a.sorted_events, m->sort_scratch, nullptr));
    HL_CUDA(cudaEventRecord(m->sort_event, ctx->stream));
  }
  HL_TRY(hl_memory_selected_scores_forward(ctx, idx, a.query, kd, P + m->off_kl, P + m->off_kr, m->m_scores, N, k, side, kd,
                                           m->mem.slots));
  HL_TRY(hl_softmax_rows_f32(ctx, m->m_scores, a.weights, N, k));
  return hl_memory_weighted_value_forward(ctx, idx, a.weights, P + m->off_val, a.weighted, N, k, m->mem.slots, vd);
}

// What every memory block's lookup of a pass reads of the tables, which all of them share.
int prepare_lookups(hl_decoder* m) {
  if (!looks_up(m)) return HL_OK;
  return product_key_pieces(m->ctx, m->params + m->off_kl, m->params + m->off_kr, m->side, m->mem.key_dim, m->key_pieces);
}

// dweighted -> m_dq (gradient of the query) and the table gradients (added into the arena).
int memory_core_backward(hl_decoder* m, int l, const float* dweighted) {
  hl_ctx* ctx = m->ctx;
  MemoryActs& a = m->ma[l];
  const float* P = m->params;
  float* G = m->grads;
  const int N = m->N, kd = m->mem.key_dim, vd = m->mem.value_dim, k = m->mem.top_k, side = m->side;
  ProfileScope prof(ctx, HL_PROF_OTHER, (double)N * k * (double)(kd + 3 * vd) * 4.0);
  if (m->sorted && a.sorted_rows) {
    HL_CUDA(cudaStreamWaitEvent(ctx->stream, m->sort_event, 0));
    HL_TRY(weighted_value_backward_ordered(ctx, a.sorted_rows, a.sorted_events, a.weights, P + m->off_val, dweighted, m->m_dw, G + m->off_val,
                                           (long long)N * k, k, m->mem.slots, vd));
  } else {
    HL_TRY(hl_memory_weighted_value_backward(ctx, a.idx, a.weights, P + m->off_val, dweighted, m->m_dw, G + m->off_val, N, k,
                                             m->mem.slots, vd));
  }
  HL_TRY(hl_softmax_rows_backward_f32(ctx, a.weights, m->m_dw, m->m_dscores, N, k));
  auto scores_backward = [&](float* dq, float* dl, float* dr) {
    return hl_memory_selected_scores_backward(ctx, a.idx, a.query, kd, P + m->off_kl, P + m->off_kr, m->m_dscores, dq, kd, dl, dr, N, k, side, kd,
                                              m->mem.slots);
  };
  const KeyGradient keys = key_gradient(m);
  const int shares = beside(m) ? key_gradient_shares(ctx, keys) : 0;
  if (shares == 0 || key_gradient_bytes(keys, shares) > m->side_arena_bytes) return scores_backward(m->m_dq, G + m->off_kl, G + m->off_kr);
  {  // nothing in the backward pass waits for the tables' gradients
    SideWork side_work(m);
    HL_TRY(side_work.rc);
    HL_TRY(scores_backward(nullptr, G + m->off_kl, G + m->off_kr));
  }
  return scores_backward(m->m_dq, nullptr, nullptr);
}

// A product on the side stream where its scratch is there, else where everything is.
int run_beside(hl_decoder* m, const hl_gemm_desc& d, const __nv_bfloat16* a, const __nv_bfloat16* b, float* c) {
  size_t bytes = 0;
  if (!beside(m) || !gemm_bf16_scratch(m->ctx, &d, &bytes) || bytes > m->side_arena_bytes)
    return gemm_bf16_ctx(m->ctx, &d, a, b, c, nullptr, nullptr, nullptr);
  SideWork side(m);
  HL_TRY(side.rc);
  return gemm_bf16_ctx(m->ctx, &d, a, b, c, nullptr, nullptr, nullptr);
}

// Final layer norm and head of one row of the residual stream: the logits in row 0 of m->logits.
int decode_head(hl_decoder* m, const void* x, int dtype) {
  DecodeGemv g{};
  g.x = x; g.x_dtype = dtype;
  g.gamma = m->params + m->off_lnf_g; g.beta = m->params + m->off_lnf_b;
  g.w = dtype == HL_BF16 ? (const void*)(m->shadow + m->off_head_w) : (const void*)(m->params + m->off_head_w);
  g.w_dtype = dtype;
  g.bias = m->params + m->off_head_b;
  g.out = m->row_logits ? m->row_logits : m->logits; g.out_dtype = HL_F32;
  g.n = m->cfg.vocab; g.k = m->cfg.d_model;
  return decode_gemv(m->ctx, g);
}

// A matrix-vector product of one row, in the model's precision, behind a layer norm when one is given.
DecodeGemv row_gemv(const hl_decoder* m, const void* x, size_t w, size_t b, void* out, int n, int k, int epilogue, const void* residual,
                    size_t ln_g, size_t ln_b) {
  const bool amp = m->cfg.precision == HL_PRECISION_AMP_BF16;
  DecodeGemv g{};
  g.x = x; g.x_dtype = amp ? HL_BF16 : HL_F32;
  g.w = amp ? (const void*)(m->shadow + w) : (const void*)(m->params + w);
  g.w_dtype = g.x_dtype;
  g.bias = m->params + b;
  g.out = out; g.out_dtype = g.x_dtype;
  g.n = n; g.k = k; g.epilogue = epilogue; g.residual = residual;
  if (ln_g) { g.gamma = m->params + ln_g; g.beta = m->params + ln_b; }
  return g;
}

// Block l for the row whose position stands in m->decode_state, in the two kernels of decode_block.cu.  `x`: its input row; with
// `window` the block's q/k/v rows are there.  Returns the row behind the block, or behind its attention in front of a memory block.
bool row_block_fused(const hl_decoder* m) {
  const hl_decoder_config& c = m->cfg;
  return decode_block_applies(c.precision == HL_PRECISION_AMP_BF16 ? HL_BF16 : HL_F32, c.d_model, c.n_heads, c.d_ff, c.context);
}
int row_block_fused(hl_decoder* m, int l, const DecodeRow& x, bool window, DecodeRow* after) {
  const hl_decoder_config& c = m->cfg;
  const LayerOffsets& o = m->lo[l];
  const bool amp = c.precision == HL_PRECISION_AMP_BF16;
  const float* P = m->params;
  auto weight = [&](size_t w) { return amp ? (const void*)(m->shadow + w) : (const void*)(P + w); };
  DecodeBlock b{};
  b.dtype = amp ? HL_BF16 : HL_F32;
  b.d = c.d_model; b.heads = c.n_heads; b.hidden = c.d_ff; b.context = c.context;
  b.state = m->decode_state;
  b.x = x;
  b.x.keep = window ? nullptr : amp ? (void*)m->x[l] : (void*)m->xf[l];
  b.window = window;
  b.ln1_gamma = P + o.ln1g; b.ln1_beta = P + o.ln1b;
  b.wqkv = weight(o.wqkv); b.bqkv = P + o.bqkv;
  b.qkv = amp ? (void*)m->la[l].qkv : (void*)m->lf[l].qkv;
  b.wo = weight(o.wo); b.bo = P + o.bo;
  b.attention_parts = m->row_parts[0]; b.feed_forward_parts = m->row_parts[1];
  DecodeRow r{};
  HL_TRY(decode_attention_block(m->ctx, b, &r));
  r.keep = amp ? (void*)m->la[l].r : (void*)m->lf[l].r;
  if (o.is_memory) { *after = r; return HL_OK; }
  b.ln2_gamma = P + o.ln2g; b.ln2_beta = P + o.ln2b;
  b.w1 = weight(o.w1); b.b1 = P + o.b1;
  b.w2 = weight(o.w2); b.b2 = P + o.b2;
  return decode_feed_forward(m->ctx, b, r, after);
}
int row_head(hl_decoder* m, const DecodeRow& x) {
  const bool amp = m->cfg.precision == HL_PRECISION_AMP_BF16;
  return decode_head_row(m->ctx, x, amp ? HL_BF16 : HL_F32, m->params + m->off_lnf_g, m->params + m->off_lnf_b,
                         amp ? (const void*)(m->shadow + m->off_head_w) : (const void*)(m->params + m->off_head_w), m->params + m->off_head_b,
                         m->row_logits ? m->row_logits : m->logits, m->cfg.vocab, m->cfg.d_model);
}

// Attention and feed-forward of block l for the row whose position stands in m->decode_state, `x` being its input row; the
// result goes to row 0 of the block's output.  The block's q/k/v rows are there, `settled`: but for this row, since before
// the sequence of launches began.
int row_block(hl_decoder* m, int l, const void* x, bool settled) {
  hl_ctx* ctx = m->ctx;
  const hl_decoder_config& c = m->cfg;
  const LayerOffsets& o = m->lo[l];
  const int d = c.d_model, F = c.d_ff;
  const bool amp = c.precision == HL_PRECISION_AMP_BF16;
  void *next, *qkv, *att, *r, *g;
  if (amp) { next = m->x[l + 1]; qkv = m->la[l].qkv; att = m->la[l].o; r = m->la[l].r; g = m->la[l].g; }
  else { next = m->xf[l + 1]; qkv = m->lf[l].qkv; att = m->lf[l].o; r = m->lf[l].r; g = m->lf[l].g; }
  HL_TRY(decode_attention(ctx, qkv, amp ? HL_BF16 : HL_F32, 3 * d, m->decode_state, att, d, c.n_heads, c.context, settled));
  HL_TRY(decode_gemv(ctx, row_gemv(m, att, o.wo, o.bo, r, d, d, GV_RESIDUAL, x, 0, 0)));
  if (o.is_memory) return HL_OK;
  HL_TRY(decode_gemv(ctx, row_gemv(m, r, o.w1, o.b1, g, F, d, GV_GELU, nullptr, o.ln2g, o.ln2b)));
  return decode_gemv(ctx, row_gemv(m, g, o.w2, o.b2, next, d, F, GV_RESIDUAL, r, 0, 0));
}

bool decode_applicable(const hl_decoder* m) {
  const hl_decoder_config& c = m->cfg;
  const int dt = c.precision == HL_PRECISION_AMP_BF16 ? HL_BF16 : HL_F32;
  return decode_attention_smem(dt, c.d_model / c.n_heads, c.context) <= 48 * 1024;
}
// The last block of a pass that wants its last position only: behind the q/k/v product nothing but that row is worked on (a
// window of 500 of the GPT-sized model: 24 us less, 64 rows of four f32 blocks: 26).  Memory blocks keep all rows: their routing
// is read by others.
bool last_block_by_row(const hl_decoder* m, int l) {
  return l == m->cfg.n_layers - 1 && !m->lo[l].is_memory && decode_applicable(m);
}

// The head's product as gemm_bf16_row_stats takes it; its results lie in the logits' buffer.
struct HeadStats {
  hl_gemm_desc desc{};
  GemmRowStats stats{};
  float* row_loss;
  bool fits;
  HeadStats(const hl_decoder* m, bool gradient) {
    const size_t N = (size_t)m->N, V = (size_t)m->cfg.vocab, parts = (size_t)ceil_div(m->cfg.vocab, 128) * N;
    desc.m = m->N; desc.n = m->cfg.vocab; desc.k = m->cfg.d_model;
    desc.a_layout = desc.b_layout = HL_K_MAJOR;
    desc.lda = desc.ldb = m->cfg.d_model; desc.ldc = m->cfg.vocab;
    desc.epilogue = HL_EPI_BIAS; desc.out_dtype = HL_F32;
    stats.parts = reinterpret_cast<float2*>(m->logits);
    stats.rows = gradient ? stats.parts + parts : nullptr;
    stats.target_logit = m->logits + 2 * (parts + N);
    stats.targets = m->targets;
    stats.grad_scale = 1.0f / (float)m->N;
    row_loss = stats.target_logit + N;
    fits = 2 * parts + 4 * N <= N * V;
  }
};
// Whether a training step forms the logits twice, for the row sums and for their gradient, instead of storing them in f32 for the
// loss kernel to read and turn into the gradient: 2 d flop an element (d is at most 1024 here) against eight bytes.  Bound by the
// tensor core then instead of by the copy rate.  Step of a one-block model, stored / twice, us, in turn in one process (quartiles 1 to
// 3 % apart where the power cap acts): d 512, 4096 x 32000 780 / 729, 1024 x 32000 315 / 303; d 768, 16384 x 50304 5293 / 4895,
// 2048 x 32000 562 / 551; d 1024, 16384 x 32000 4655 / 4316, 1024 x 32000 431 / 428.  In the benchmark step, whose other products
// draw on the same power, 17280 / 17260.
// Below 1024 rows the logits stay in L2 and the second product's start costs what it saves: d 768, 512 x 32000 277 / 286.  With few
// columns they stay there too, and the wider rows are, the more the product costs: d 960, 1024 x 8000 264 / 270, 2048 x 2000 271 / 275,
// d 832, 1024 x 8000 242 / 245; from 48 MB of logits or 4096 rows on even those gain (d 960, 1536 x 8000 316 / 315, 4096 x 2000
// 409 / 388), and at d 512 all do (1024 x 8000 187 / 183), up to d 768 as many as lose (2048 x 2000 224 / 227 and 240 / 240).
constexpr int kHeadTwiceRows = 1024, kHeadTwiceManyRows = 4096, kHeadTwiceWide = 768;
constexpr long long kHeadTwiceLogits = 12000000;
bool head_twice_pays(const hl_decoder* m) {
  return m->N >= kHeadTwiceRows &&
         (m->N >= kHeadTwiceManyRows || m->cfg.d_model <= kHeadTwiceWide || (long long)m->N * m->cfg.vocab >= kHeadTwiceLogits);
}

// What a forward pass is for: logits and activations for the backward pass, the logits of the last position alone (they go to
// row 0 of m->logits), or the mean loss alone (to m->loss_dev).
enum class Forward { all, last_position, loss };
int forward(hl_decoder* m, Forward what = Forward::all) {
  hl_ctx* ctx = m->ctx;
  struct Only {  // no backward pass follows
    hl_ctx* c;
    ~Only() { c->forward_only = false; }
  } only{ctx};
  ctx->forward_only = what != Forward::all;
  const hl_decoder_config& c = m->cfg;
  const int N = m->N, d = c.d_model, F = c.d_ff, V = c.vocab, B = c.batch, T = c.context, H = c.n_heads;
  const Gemm g{m};
  const float* P = m->params;
  const __nv_bfloat16* W = m->shadow;
  if (!m->comm_pending) ctx->reserve_sms = 0;  // nothing of the gradient exchange is in flight during a forward pass
  HL_TRY(hl_embedding_forward(ctx, P + m->off_tok, V, m->tokens, P + m->off_pos, T, m->x[0], HL_BF16, N, d));
  HL_TRY(prepare_lookups(m));
  for (int l = 0; l < c.n_layers; ++l) {
    const LayerOffsets& o = m->lo[l];
    LayerActs& a = m->la[l];
    HL_TRY(layer_norm_forward_impl(ctx, m->x[l], HL_BF16, P + o.ln1g, P + o.ln1b, a.a, HL_BF16, a.mean1, a.rstd1, N, d, 1e-5f));
    HL_TRY(g.run(N, 3 * d, d, a.a, d, HL_K_MAJOR, W + o.wqkv, d, HL_K_MAJOR, a.qkv, 3 * d, HL_BF16, HL_EPI_BIAS, P + o.bqkv));
    if (what == Forward::last_position && last_block_by_row(m, l)) {
      if (row_block_fused(m)) {
        DecodeRow x{}, after{};
        x.base = m->x[l] + (size_t)(N - 1) * d;
        HL_TRY(row_block_fused(m, l, x, true, &after));
        return row_head(m, after);
      }
      HL_TRY(row_block(m, l, m->x[l] + (size_t)(N - 1) * d, false));
      return decode_head(m, m->x[l + 1], HL_BF16);
    }
    if (m->flash_ok) HL_TRY(flash_attention_forward_impl(ctx, a.qkv, a.qkv + d, a.qkv + 2 * d, 3 * d, a.o, d, a.lse, B, T, H, d / H));
    // head sizes other than 64 and 128: the f64 kernels read the bf16 rows (widened exactly) and round to bf16 where the flash route
    // stores bf16; the backward pass forms the probabilities again
    else HL_TRY(attention_f64_forward(ctx, a.qkv, a.qkv + d, a.qkv + 2 * d, HL_BF16, 3 * d, a.o, d, m->fa_probs, B, T, d, H));
    HL_TRY(g.run(N, d, d, a.o, d, HL_K_MAJOR, W + o.wo, d, HL_K_MAJOR, a.r, d, HL_BF16, HL_EPI_BIAS_RESIDUAL, P + o.bo,
                 m->x[l], d));
    HL_TRY(layer_norm_forward_impl(ctx, a.r, HL_BF16, P + o.ln2g, P + o.ln2b, a.c, HL_BF16, a.mean2, a.rstd2, N, d, 1e-5f));
    if (o.is_memory) {
      // The reference keeps the memory feed-forward in f32 under AMP (src/memory_transformer.rs:787-789).  Its three
      // projections still run on the tensor cores here, at f32 accuracy: the block input is bf16-exact, so
      // x*W = x*W_hi + x*W_mid + x*W_lo with exact products and one f32 accumulation (a contraction of 3*d against
      // the weight's three bf16 pieces, the input read three times); out_proj takes the f32 mv as hi + lo pieces and
      // drops only the lo*lo term (2^-16 relative, far below the bf16 rounding of the block output that follows).
      // The query decides the routing, so it has to be this accurate; lookup, scores, softmax, gather and gate are f32.
      MemoryActs& ma = m->ma[l];
      const int kd = m->mem.key_dim, vd = m->mem.value_dim;
      HL_TRY(hl_split_bf16_f32(ctx, P + o.wq_m, ma.wq3, kd, d, HL_SPLIT_HI_MID_LO));
      HL_TRY(hl_split_bf16_f32(ctx, P + o.wg_m, ma.wg3, vd, d, HL_SPLIT_HI_MID_LO));
      HL_TRY(hl_split_bf16_f32(ctx, P + o.wout_m, ma.wout3, d, vd, HL_SPLIT_HI_HI_LO));
      HL_TRY(g.run(N, kd, 3 * d, a.c, d, HL_K_MAJOR, ma.wq3, 3 * d, HL_K_MAJOR, ma.query, kd, HL_F32, HL_EPI_BIAS, P + o.bq_m,
                   nullptr, 0, nullptr, 0, d));
      HL_TRY(memory_core_forward(m, l));
      HL_TRY(g.run(N, vd, 3 * d, a.c, d, HL_K_MAJOR, ma.wg3, 3 * d, HL_K_MAJOR, ma.gpre, vd, HL_F32, HL_EPI_BIAS, P + o.bg_m,
                   nullptr, 0, nullptr, 0, d));
      HL_TRY(memory_gate_forward(ctx, ma.gpre, ma.weighted, ma.gate, ma.mv, N, vd, pieces_beside(ma.mv_b, 2 * vd, vd, 2, 0, 1)));
      HL_TRY(g.run(N, d, 3 * vd, ma.mv_b, 2 * vd, HL_K_MAJOR, ma.wout3, 3 * vd, HL_K_MAJOR, m->x[l + 1], d, HL_BF16,
                   HL_EPI_BIAS_RESIDUAL, P + o.bout_m, a.r, d, nullptr, 0, 2 * vd));
      continue;
    }
    HL_TRY(g.run(N, F, d, a.c, d, HL_K_MAJOR, W + o.w1, d, HL_K_MAJOR, a.h, F, HL_BF16, HL_EPI_BIAS_GELU, P + o.b1, nullptr,
                 0, a.g, F));
    HL_TRY(g.run(N, d, F, a.g, F, HL_K_MAJOR, W + o.w2, F, HL_K_MAJOR, m->x[l + 1], d, HL_BF16, HL_EPI_BIAS_RESIDUAL,
                 P + o.b2, a.r, d));
  }
  if (what == Forward::last_position) return decode_head(m, m->x[c.n_layers] + (size_t)(N - 1) * d, HL_BF16);
  HL_TRY(layer_norm_forward_impl(ctx, m->x[c.n_layers], HL_BF16, P + m->off_lnf_g, P + m->off_lnf_b, m->z, HL_BF16, m->meanf,
                                 m->rstdf, N, d, 1e-5f));
  m->head_twice = false;
  if (what == Forward::loss || head_twice_pays(m)) {
    // maxima and sums of the logits without the logits, in the buffer that would hold them
    const HeadStats h(m, what == Forward::all);
    int rc = HL_OK;
    if (h.fits && gemm_bf16_row_stats(ctx, &h.desc, m->z, W + m->off_head_w, P + m->off_head_b, h.stats, m->logits, &rc)) {
      HL_TRY(rc);
      m->head_twice = what == Forward::all;  // the backward pass takes the loss, and forms the logits again for its gradient
      return m->head_twice ? HL_OK : row_stats_loss(ctx, h.stats, N, V, h.row_loss, m->loss_dev);
    }
  }
  HL_TRY(g.run(N, V, d, m->z, d, HL_K_MAJOR, W + m->off_head_w, d, HL_K_MAJOR, m->logits, V, HL_F32, HL_EPI_BIAS,
               P + m->off_head_b));
  if (what == Forward::loss)
    return cross_entropy_impl(ctx, m->logits, V, m->targets, N, V, 1.0f, m->loss_dev, nullptr, nullptr, HL_BF16, V);
  return HL_OK;
}

// Bucket b covers gradient-arena elements [b*bucket, min((b+1)*bucket, arena)); it may be reduced
// once every gradient below its end is final.  Pure host arithmetic, shared with hl_ddp_ready_buckets.
inline void bucket_range(size_t arena, size_t bucket, size_t b, size_t* start, size_t* end) {
  *start = b * bucket;
  *end = std::min(*start + bucket, arena);
}

// Queue the all-reduce of every bucket whose gradients are final.
int flush_buckets(hl_decoder* m, size_t done_elems) {
  if (!nccl_active(m->ctx)) return HL_OK;
  while (m->next_bucket < m->n_buckets) {
    size_t start, end;
    bucket_range(m->arena, m->bucket_elems, m->next_bucket, &start, &end);
    if (end > done_elems) break;
    HL_CUDA(cudaEventRecord(m->bucket_ready[m->next_bucket], m->ctx->stream));
    HL_CUDA(cudaStreamWaitEvent(m->ctx->comm_stream, m->bucket_ready[m->next_bucket], 0));
    // The value table and the token-embedding table travel as the union of the rows that carry a gradient
    // (exchange_rows), not densely: their ranges are cut out of the bucket (value table first, token table last).
    size_t cut_lo[2], cut_hi[2];
    int cuts = 0;
    if (m->has_memory) { cut_lo[cuts] = m->off_val; cut_hi[cuts] = m->off_val + (size_t)m->mem.slots * m->mem.value_dim; ++cuts; }
    if (m->sparse_tok_exchange) { cut_lo[cuts] = m->off_tok; cut_hi[cuts] = m->off_tok + (size_t)m->cfg.vocab * m->cfg.d_model; ++cuts; }
    size_t at = start;
    for (int c = 0; c <= cuts && at < end; ++c) {
      const size_t stop = c < cuts ? std::min(end, std::max(at, cut_lo[c])) : end;
      if (at < stop) HL_TRY(nccl_allreduce_sum_f32(m->ctx, m->grads + at, stop - at, m->ctx->comm_stream));
      at = c < cuts ? std::max(stop, std::min(end, cut_hi[c])) : end;
    }
    HL_CUDA(cudaEventRecord(m->bucket_done[m->next_bucket], m->ctx->comm_stream));
    m->next_bucket += 1;
    m->ctx->reserve_sms = m->ctx->comm_sms;  // collectives are in flight from here to the optimizer's last wait
  }
  return HL_OK;
}

// Data-parallel exchange of a table gradient of which only some rows are non-zero: every rank marks the rows it
// touched, the masks are combined with a byte-wise maximum, the union's gradient rows are packed, summed over the
// ranks and put back (src/bin/heirloom/runtime.rs:4171-4214).  Rows outside the union have zero gradient on every
// rank.  Runs on the collective stream in two halves: the union of the rows when they are known, the exchange of the
// gradient rows after the dense buckets; the host reads the union's size between the two, long after it was written.
struct RowExchange {
  float* grad;            // [rows, dim] in the gradient arena
  int rows, dim;
  unsigned char* flags;   // [rows], zero on entry and on return
  int64_t* union_rows;    // [rows]
  int* count_dev;
  int* count_host;        // pinned
  float** packed;         // own allocation, grown on demand
  size_t* packed_cap;     // rows it holds
  size_t max_events;      // rows all ranks together can touch at most
};

// First half, queued as soon as the touched rows are known: x.flags holds this rank's marks; the union over the ranks, its
// row list and its size (copied to pinned host memory) follow on the collective stream, `ready` after them.
int prepare_rows(hl_decoder* m, const RowExchange& x, cudaEvent_t ready) {
  hl_ctx* ctx = m->ctx;
  cudaStream_t cs = ctx->comm_stream;
  HL_TRY(nccl_allreduce_max_u8(ctx, x.flags, (size_t)x.rows, cs));
  HL_TRY(mask_to_indices_on(ctx, cs, x.flags, x.rows, x.union_rows, x.count_dev));
  HL_CUDA(cudaMemcpyAsync(x.count_host, x.count_dev, sizeof(int), cudaMemcpyDeviceToHost, cs));
  HL_CUDA(cudaMemsetAsync(x.flags, 0, (size_t)x.rows, cs));
  HL_CUDA(cudaEventRecord(ready, cs));
  return HL_OK;
}

// Second half, once the gradient rows are final: pack the union's rows, sum them over the ranks, put them back.  The
// host reads the size here; the device passed `ready` long ago unless the caller queued both halves back to back.
int finish_rows(hl_decoder* m, const RowExchange& x, cudaEvent_t ready, int* union_n) {
  hl_ctx* ctx = m->ctx;
  cudaStream_t cs = ctx->comm_stream;
  HL_CUDA(cudaEventSynchronize(ready));
  const int n = *x.count_host;
  HL_REQUIRE(n >= 0 && n <= x.rows, "hl_decoder: row union out of range");
  *union_n = n;
  if (n > 0) {
    // The packed rows live in a buffer of their own: the context's scratch arena belongs to the compute stream,
    // which keeps running (and may regrow the arena) while this exchange is in flight on the collective stream.
    if ((size_t)n > *x.packed_cap) {
      const size_t cap = std::max((size_t)n, std::min((size_t)x.rows, x.max_events));
      if (*x.packed) {
        HL_CUDA(cudaStreamSynchronize(cs));  // an earlier step's exchange may still be reading the old buffer
        HL_CUDA(cudaFree(*x.packed));
        *x.packed = nullptr;
        *x.packed_cap = 0;
      }
      HL_CUDA(cudaMalloc(reinterpret_cast<void**>(x.packed), sizeof(float) * cap * x.dim));
      *x.packed_cap = cap;
      ctx->counters.allocations += 1;
      ctx->counters.allocated_bytes += sizeof(float) * cap * x.dim;
    }
    HL_TRY(move_rows_on(ctx, cs, x.grad, x.union_rows, nullptr, n, x.dim, *x.packed, false));
    HL_TRY(nccl_allreduce_sum_f32(ctx, *x.packed, (size_t)n * x.dim, cs));
    HL_TRY(move_rows_on(ctx, cs, *x.packed, x.union_rows, nullptr, n, x.dim, x.grad, true));
  }
  return HL_OK;
}

// The value table: rows = the slots the memory blocks selected.
RowExchange value_rows(hl_decoder* m) {
  const size_t per_layer = (size_t)m->N * m->mem.top_k;
  return RowExchange{m->grads + m->off_val, m->mem.slots, m->mem.value_dim, m->m_row_flags, m->m_union_rows, m->m_union_count,
                     m->m_union_count_host, &m->m_packed, &m->packed_rows_cap,
                     (size_t)nccl_world(m->ctx) * per_layer * (size_t)m->mem.n_memory_layers};
}

// Queued after forward: the selections of every memory block are on the device.
int prepare_value_rows(hl_decoder* m) {
  if (!m->has_memory || !nccl_active(m->ctx)) return HL_OK;
  hl_ctx* ctx = m->ctx;
  cudaStream_t cs = ctx->comm_stream;
  const size_t per_layer = (size_t)m->N * m->mem.top_k;
  const int slots = m->mem.slots;
  HL_CUDA(cudaEventRecord(m->rows_known, ctx->stream));
  HL_CUDA(cudaStreamWaitEvent(cs, m->rows_known, 0));
  HL_CUDA(cudaMemsetAsync(m->m_row_flags, 0, (size_t)slots, cs));
  for (int l = 0; l < m->cfg.n_layers; ++l)
    if (m->lo[l].is_memory) HL_TRY(mark_rows_on(ctx, cs, m->ma[l].idx, (long long)per_layer, nullptr, m->m_row_flags, slots));
  HL_TRY(prepare_rows(m, value_rows(m), m->val_count_ready));
  m->val_prepared = true;
  return HL_OK;
}

int exchange_value_rows(hl_decoder* m) {
  if (!m->has_memory || !nccl_active(m->ctx)) return HL_OK;
  if (!m->val_prepared) HL_TRY(prepare_value_rows(m));
  m->val_prepared = false;
  return finish_rows(m, value_rows(m), m->val_count_ready, &m->union_n);
}

// The token-embedding table: rows = the token ids of the batch.  At a Zipf-distributed batch of 16 Ki tokens over a
// vocabulary of 50 Ki this is a small share of the 154 MB table, and it is the gradient that becomes final last in
// backward, i.e. the exchange nothing is left to hide behind.
RowExchange token_rows(hl_decoder* m) {
  return RowExchange{m->grads + m->off_tok, m->cfg.vocab, m->cfg.d_model, m->tok_flags, m->tok_union_rows, m->tok_union_count,
                     m->tok_union_count_host, &m->tok_packed, &m->tok_packed_cap, (size_t)nccl_world(m->ctx) * (size_t)m->N};
}

// Queued as soon as the step's token ids are on the device.
int prepare_token_rows(hl_decoder* m) {
  if (!m->sparse_tok_exchange || !nccl_active(m->ctx)) return HL_OK;
  hl_ctx* ctx = m->ctx;
  cudaStream_t cs = ctx->comm_stream;
  const int V = m->cfg.vocab;
  HL_CUDA(cudaEventRecord(m->rows_known, ctx->stream));
  HL_CUDA(cudaStreamWaitEvent(cs, m->rows_known, 0));
  HL_CUDA(cudaMemsetAsync(m->tok_flags, 0, (size_t)V, cs));
  HL_TRY(mark_rows_on(ctx, cs, m->tokens, (long long)m->N, nullptr, m->tok_flags, V));
  HL_TRY(prepare_rows(m, token_rows(m), m->tok_count_ready));
  m->tok_prepared = true;
  return HL_OK;
}

int exchange_token_rows(hl_decoder* m) {
  if (!m->sparse_tok_exchange || !nccl_active(m->ctx)) return HL_OK;
  if (!m->tok_prepared) HL_TRY(prepare_token_rows(m));
  m->tok_prepared = false;
  int n = 0;
  return finish_rows(m, token_rows(m), m->tok_count_ready, &n);
}

int backward(hl_decoder* m) {
  hl_ctx* ctx = m->ctx;
  const hl_decoder_config& c = m->cfg;
  const int N = m->N, d = c.d_model, F = c.d_ff, V = c.vocab, B = c.batch, T = c.context, H = c.n_heads;
  const Gemm g{m};
  const float* P = m->params;
  const __nv_bfloat16* W = m->shadow;
  float* G = m->grads;
  m->next_bucket = 0;
  m->wgrads.clear();
  if (m->comm_pending) {  // a previous step's collectives were never consumed: finish them before its gradients are overwritten
    HL_CUDA(cudaStreamWaitEvent(m->ctx->stream, m->comm_done, 0));
    m->comm_pending = false;
  }
  // loss and dlogits = (softmax - onehot)/N in bf16, the operand precision of the next GEMMs
  if (m->head_twice) {
    const HeadStats h(m, true);
    HL_TRY(row_stats_loss(ctx, h.stats, N, V, h.row_loss, m->loss_dev, m->loss_host));
    HL_TRY(gemm_bf16_loss_gradient(ctx, &h.desc, m->z, W + m->off_head_w, P + m->off_head_b, h.stats, m->dlogits));
  } else {
    HL_TRY(cross_entropy_impl(ctx, m->logits, V, m->targets, N, V, 1.0f, m->loss_dev, nullptr, m->dlogits, HL_BF16, V, m->loss_host));
  }
  if (m->has_memory) HL_TRY(tables_are_zero(m));
  FoldBatch* fb = &m->fold;
  fb->n = 0;
  fb->used = 0;
  // Everything up to arena element `done` has been written, the column reductions in the batch apart: they are folded one
  // launch per full batch, unless a bucket of the gradient exchange is waiting for them.
  auto finished = [&](size_t done) -> int {
    if (nccl_active(ctx) || done == m->arena) HL_TRY(fold_batch_flush(ctx, fb));
    return flush_buckets(m, done);
  };
  // lm_head.  Its bias gradient, where it is a pass of its own over the logits' gradient, runs beside the two products.
  const hl_gemm_desc head_gradient = product(V, d, N, HL_MN_MAJOR, V, HL_MN_MAJOR, d, 0, 0);
  const bool bias_apart = beside(m) && !grouping(m) && !gemm_bf16_small_applies(ctx, &head_gradient);
  if (bias_apart) {
    SideStream side(m);
    HL_TRY(side.rc);
    HL_TRY(bias_grad_impl(ctx, m->dlogits, HL_BF16, G + m->off_head_b, N, V, fb));
  }
  HL_TRY(weight_gradient(m, m->dlogits, V, m->z, d, G + m->off_head_w, bias_apart ? nullptr : G + m->off_head_b));
  HL_TRY(g.run(N, d, V, m->dlogits, V, HL_K_MAJOR, W + m->off_head_w, d, HL_MN_MAJOR, m->dtmp, d, HL_F32));
  if (bias_apart) HL_TRY(join_side(m));  // its partial sums are folded with the others'
  float* dx = m->dx0;
  float* dx_next = m->dx1;
  // every layer-norm backward also returns the column sums of the gradient it writes: the bias
  // gradient of the projection that produced that residual-stream value (fc2 or out_proj)
  HL_TRY(layer_norm_backward_impl(ctx, m->x[c.n_layers], HL_BF16, P + m->off_lnf_g, m->dtmp, m->meanf, m->rstdf, nullptr, dx,
                                  m->la[c.n_layers - 1].dy, G + m->off_lnf_g, G + m->off_lnf_b, G + m->lo[c.n_layers - 1].out_bias(),
                                  N, d, fb));
  HL_TRY(finished(m->off_lnf_b + d));
  for (int l = c.n_layers - 1; l >= 0; --l) {
    const LayerOffsets& o = m->lo[l];
    LayerActs& a = m->la[l];
    if (o.is_memory) {
      // y = r + out_proj(weighted * gelu(gate_proj(c))), weighted from the lookup on query_proj(c)
      MemoryActs& ma = m->ma[l];
      const int kd = m->mem.key_dim, vd = m->mem.value_dim;
      // The reference runs these three projections in f32 also backward (src/memory_transformer.rs:787-789).  Here
      // every product stays on the tensor cores with its f32 operands as bf16 pieces: hi*hi + lo*hi + hi*lo in one
      // f32 accumulation (the dropped lo*lo term is 2^-16 relative), or hi + mid + lo (exact) against the block input,
      // which is bf16-exact.  `side`: pieces along the columns, for operands contracted along their rows' direction;
      // `rows`: pieces one below the other, for operands contracted down their rows.  The gradients of the two projections
      // that read c are one product over both: hi*lo and lo*hi of the two, 2^-8 of the rest, come first and hi*hi after them, since the
      // tensor core's additions truncate what it has added up so far (error against f64 of 16384 x 512 over 2 x 512: 4.5e-6, of it 4.4e-6
      // the dropped lo*lo; a projection after the other with hi*hi first 6.2e-6, two products added up 5.1e-6).
      HL_TRY(join_side(m));  // the block's buffers are those of the one above
      const int ROWS = HL_SPLIT_STACK_ROWS;
      const float* dy = dx;  // dL/dy of this block, f32
      // out_proj: dW = dy^T mv, dmv = dy W
      HL_TRY(split_pieces(ctx, dy, N, d, pieces_stacked(m->p_dx_rows, N, d, 2, 0, 1), pieces_beside(m->p_dx_side, 2 * d, d, 2, 0, 1)));
      HL_TRY(hl_split_bf16_f32(ctx, ma.mv, m->p_mv_rows, N, vd, HL_SPLIT_HI_HI_LO | ROWS));
      HL_TRY(run_beside(m, out_gradient(m), m->p_dx_rows, m->p_mv_rows, G + o.wout_m));
      HL_TRY(hl_split_bf16_f32(ctx, P + o.wout_m, m->p_wout_rows, d, vd, HL_SPLIT_HI_HI_LO | ROWS));
      HL_TRY(g.run(N, vd, 3 * d, m->p_dx_side, 2 * d, HL_K_MAJOR, m->p_wout_rows, vd, HL_MN_MAJOR, m->m_dmv, vd, HL_F32,
                   HL_EPI_NONE, nullptr, nullptr, 0, nullptr, 0, 2 * d));
      // gate_proj: dW = dgpre^T c (c is bf16-exact: three exact pieces of dgpre, c read three times)
      const int both = vd + kd;
      HL_TRY(memory_gate_backward(ctx, m->m_dmv, ma.gate, ma.weighted, ma.gpre, m->m_dweighted, m->m_dgpre, N, vd,
                                  pieces_stacked(m->p_dg_rows, N, vd, 3, 0, 1, 2), PieceDest{m->p_dc_side, 2 * both, both, 2, {0, 1}}));
      HL_TRY(run_beside(m, in_gradient(m, vd), m->p_dg_rows, a.c, G + o.wg_m));
      HL_TRY(bias_grad_impl(ctx, m->m_dgpre, HL_F32, G + o.bg_m, N, vd, fb));
      HL_TRY(memory_core_backward(m, l, m->m_dweighted));
      // query_proj: dW = dq^T c
      HL_TRY(split_pieces(ctx, m->m_dq, N, kd, pieces_stacked(m->p_dq_rows, N, kd, 3, 0, 1, 2),
                          PieceDest{m->p_dc_side + vd, 2 * both, both, 2, {0, 1}}));
      HL_TRY(run_beside(m, in_gradient(m, kd), m->p_dq_rows, a.c, G + o.wq_m));
      HL_TRY(bias_grad_impl(ctx, m->m_dq, HL_F32, G + o.bq_m, N, kd, fb));
      // dc = dgpre Wg + dq Wq
      HL_TRY(split_pieces(ctx, P + o.wg_m, vd, d, PieceDest{m->p_wc_rows, d, (long long)both * d, 3, {1, 0, 0}}));
      HL_TRY(split_pieces(ctx, P + o.wq_m, kd, d, PieceDest{m->p_wc_rows + (size_t)vd * d, d, (long long)both * d, 3, {1, 0, 0}}));
      HL_TRY(g.run(N, d, 3 * both, m->p_dc_side, 2 * both, HL_K_MAJOR, m->p_wc_rows, d, HL_MN_MAJOR, m->dtmp, d, HL_F32, HL_EPI_NONE,
                   nullptr, nullptr, 0, nullptr, 0, 2 * both));
    } else {
    // y = r + fc2(gelu(fc1(c)));   dx is dL/dy (f32), a.dy its bf16 operand copy
    HL_TRY(weight_gradient(m, a.dy, d, a.g, F, G + o.w2, nullptr));
    HL_TRY(g.run(N, F, d, a.dy, d, HL_K_MAJOR, W + o.w2, F, HL_MN_MAJOR, a.dh, F, HL_BF16, HL_EPI_DGELU, nullptr, a.h, F));
    HL_TRY(weight_gradient(m, a.dh, F, a.c, d, G + o.w1, G + o.b1));
    HL_TRY(g.run(N, d, F, a.dh, F, HL_K_MAJOR, W + o.w1, d, HL_MN_MAJOR, m->dtmp, d, HL_F32));
    }
    // dr = dx + LN2'(dc)
    HL_TRY(layer_norm_backward_impl(ctx, a.r, HL_BF16, P + o.ln2g, m->dtmp, a.mean2, a.rstd2, dx, dx_next, a.dr,
                                    G + o.ln2g, G + o.ln2b, G + o.bo, N, d, fb));
    std::swap(dx, dx_next);  // dx is now dL/dr
    HL_TRY(weight_gradient(m, a.dr, d, a.o, d, G + o.wo, nullptr));
    HL_TRY(g.run(N, d, d, a.dr, d, HL_K_MAJOR, W + o.wo, d, HL_MN_MAJOR, m->dob, d, HL_BF16));
    if (m->flash_ok) {
      const size_t need = flash_attention_backward_scratch_bytes(B, T, H, d / H);
      if (need > ctx->workspace_bytes) HL_TRY(ensure_workspace(ctx, need));
      HL_TRY(flash_attention_backward_impl(ctx, a.qkv, a.qkv + d, a.qkv + 2 * d, 3 * d, a.o, d, m->dob, d, a.lse, a.dqkv,
                                           a.dqkv + d, a.dqkv + 2 * d, 3 * d, B, T, H, d / H, ctx->workspace,
                                           ctx->workspace_bytes));
    } else {
      HL_TRY(attention_f64_backward(ctx, a.qkv, a.qkv + d, a.qkv + 2 * d, HL_BF16, 3 * d, m->fa_probs, m->dob, d, a.dqkv,
                                    a.dqkv + d, a.dqkv + 2 * d, 3 * d, B, T, d, H));
    }
    HL_TRY(weight_gradient(m, a.dqkv, 3 * d, a.a, d, G + o.wqkv, G + o.bqkv));
    HL_TRY(g.run(N, d, 3 * d, a.dqkv, 3 * d, HL_K_MAJOR, W + o.wqkv, d, HL_MN_MAJOR, m->dtmp, d, HL_F32));
    // dx_in = dr + LN1'(da)
    HL_TRY(layer_norm_backward_impl(ctx, m->x[l], HL_BF16, P + o.ln1g, m->dtmp, a.mean1, a.rstd1, dx, dx_next, l > 0 ? m->la[l - 1].dy : m->dxb0,
                                    G + o.ln1g, G + o.ln1b, l > 0 ? G + m->lo[l - 1].out_bias() : nullptr, N, d, fb));
    std::swap(dx, dx_next);
    if (grouping(m) && (l == 0 || (c.n_layers - l) % m->group_layers == 0)) HL_TRY(run_weight_gradients(m));
    HL_TRY(finished(o.ln1b + d));
  }
  // embeddings: scatter-add into zeroed tables, the last column sums folded beside them
  if (!m->has_memory) HL_TRY(tables_are_zero(m));
  if (beside(m)) {
    SideStream side(m);
    HL_TRY(side.rc);
    HL_TRY(fold_batch_flush(ctx, fb));
  }
  HL_TRY(hl_embedding_backward(ctx, dx, m->tokens, G + m->off_tok, V, G + m->off_pos, T, N, d));
  HL_TRY(join_side(m));
  HL_TRY(finished(m->arena));
  if (nccl_active(ctx)) {
    if (m->has_memory || m->sparse_tok_exchange) {
      // the row exchanges read gradients the compute stream is still producing
      HL_CUDA(cudaEventRecord(m->comm_done, ctx->stream));
      HL_CUDA(cudaStreamWaitEvent(ctx->comm_stream, m->comm_done, 0));
      HL_TRY(exchange_token_rows(m));
      HL_TRY(exchange_value_rows(m));
    }
    // The compute stream waits for the collectives only when something reads the averaged gradients:
    // the optimizer takes them bucket group by bucket group, every other reader waits for all of them.
    HL_CUDA(cudaEventRecord(m->comm_done, ctx->comm_stream));
    m->comm_pending = true;
  }
  return HL_OK;
}

// ---- f32 route ---------------------------------------------------------------------------------
// Op by op what the reference's f32 path does (MemoryTransformerLm::forward / loss,
// src/memory_transformer.rs:2069-2081, :1604-1610; Linear = matmul(weight.transpose()) then
// add(bias), src/nn.rs:454-475), every op rounding its f32 result from an f64 accumulation.
// x · Wᵀ + b; the epilogue may add a residual (aux_in) or leave gelu of the result in aux_out
F64Gemm linear_f32(const float* x, const float* w, const float* b, float* y, int rows, int in, int out, int epilogue = F64_STORE,
                   const float* aux_in = nullptr, float* aux_out = nullptr) {
  F64Gemm g{};
  g.a = x; g.a_row = in; g.a_col = 1;
  g.b = w; g.b_row = 1; g.b_col = in;
  g.out = y; g.o_row = out; g.o_col = 1;
  g.m = rows; g.n = out; g.k = in;
  g.bias = b; g.epilogue = epilogue; g.aux_in = aux_in; g.aux_out = aux_out;
  return g;
}

// dx = dy · W (times gelu'(aux_in), or added to what is there), dw = dyᵀ · x and db, in one launch
int linear_backward_f32(hl_decoder* m, const float* x, const float* w, const float* dy, float* dx, float* dw, float* db, int rows,
                        int in, int out, int epilogue = F64_STORE, const float* aux_in = nullptr) {
  F64Gemm g[2] = {};
  g[0].a = dy; g[0].a_row = out; g[0].a_col = 1;
  g[0].b = w; g[0].b_row = in; g[0].b_col = 1;
  g[0].out = dx; g[0].o_row = in; g[0].o_col = 1;
  g[0].m = rows; g[0].n = in; g[0].k = out;
  g[0].epilogue = epilogue; g[0].aux_in = aux_in;
  g[1].a = dy; g[1].a_row = 1; g[1].a_col = out;
  g[1].b = x; g[1].b_row = in; g[1].b_col = 1;
  g[1].out = dw; g[1].o_row = in; g[1].o_col = 1;
  g[1].m = out; g[1].n = in; g[1].k = rows;
  g[1].row_sum = db;
  if (m->fork_ok && beside(m)) {  // the weight gradient beside whatever follows on the chain
    HL_TRY(f64_gemm_run(m->ctx, g, 1));
    SideStream side(m);
    HL_TRY(side.rc);
    return f64_gemm_run(m->ctx, g + 1, 1);
  }
  return f64_gemm_run(m->ctx, g, 2);
}

int forward_f32_gemm(hl_decoder* m, const F64Gemm& g) { return f64_gemm_run(m->ctx, &g, 1); }

int forward_f32(hl_decoder* m, bool last_only = false) {
  hl_ctx* ctx = m->ctx;
  const hl_decoder_config& c = m->cfg;
  const int N = m->N, d = c.d_model, F = c.d_ff, V = c.vocab, B = c.batch, T = c.context, H = c.n_heads;
  const float* P = m->params;
  HL_TRY(hl_embedding_forward(ctx, P + m->off_tok, V, m->tokens, P + m->off_pos, T, m->xf[0], HL_F32, N, d));
  HL_TRY(prepare_lookups(m));
  for (int l = 0; l < c.n_layers; ++l) {
    const LayerOffsets& o = m->lo[l];
    hl_decoder::F32Layer& a = m->lf[l];
    HL_TRY(layer_norm_forward_impl(ctx, m->xf[l], HL_F32, P + o.ln1g, P + o.ln1b, a.a, HL_F32, nullptr, nullptr, N, d, 1e-5f));
    HL_TRY(forward_f32_gemm(m, linear_f32(a.a, P + o.wqkv, P + o.bqkv, a.qkv, N, d, 3 * d)));
    if (last_only && last_block_by_row(m, l)) {
      if (row_block_fused(m)) {
        DecodeRow x{}, after{};
        x.base = m->xf[l] + (size_t)(N - 1) * d;
        HL_TRY(row_block_fused(m, l, x, true, &after));
        return row_head(m, after);
      }
      HL_TRY(row_block(m, l, m->xf[l] + (size_t)(N - 1) * d, false));
      return decode_head(m, m->xf[l + 1], HL_F32);
    }
    HL_TRY(attention_f64_forward(ctx, a.qkv, a.qkv + d, a.qkv + 2 * d, HL_F32, 3 * d, a.o, d, a.probs, B, T, d, H));
    HL_TRY(forward_f32_gemm(m, linear_f32(a.o, P + o.wo, P + o.bo, a.r, N, d, d, F64_RESIDUAL, m->xf[l])));
    HL_TRY(layer_norm_forward_impl(ctx, a.r, HL_F32, P + o.ln2g, P + o.ln2b, a.c, HL_F32, nullptr, nullptr, N, d, 1e-5f));
    if (o.is_memory) {
      MemoryActs& ma = m->ma[l];
      const int kd = m->mem.key_dim, vd = m->mem.value_dim;
      HL_TRY(forward_f32_gemm(m, linear_f32(a.c, P + o.wq_m, P + o.bq_m, ma.query, N, d, kd)));
      HL_TRY(memory_core_forward(m, l));
      HL_TRY(forward_f32_gemm(m, linear_f32(a.c, P + o.wg_m, P + o.bg_m, ma.gpre, N, d, vd, F64_GELU, nullptr, ma.gate)));
      HL_TRY(hl_binary_f32(ctx, HL_MUL, ma.weighted, ma.gate, ma.mv, (size_t)N * vd));
      HL_TRY(forward_f32_gemm(m, linear_f32(ma.mv, P + o.wout_m, P + o.bout_m, m->xf[l + 1], N, vd, d, F64_RESIDUAL, a.r)));
    } else {
      HL_TRY(forward_f32_gemm(m, linear_f32(a.c, P + o.w1, P + o.b1, a.h, N, d, F, F64_GELU, nullptr, a.g)));
      HL_TRY(forward_f32_gemm(m, linear_f32(a.g, P + o.w2, P + o.b2, m->xf[l + 1], N, F, d, F64_RESIDUAL, a.r)));
    }
  }
  if (last_only) return decode_head(m, m->xf[c.n_layers] + (size_t)(N - 1) * d, HL_F32);
  HL_TRY(layer_norm_forward_impl(ctx, m->xf[c.n_layers], HL_F32, P + m->off_lnf_g, P + m->off_lnf_b, m->zf, HL_F32, nullptr,
                                 nullptr, N, d, 1e-5f));
  return forward_f32_gemm(m, linear_f32(m->zf, P + m->off_head_w, P + m->off_head_b, m->logits, N, d, V));
}

int backward_f32(hl_decoder* m) {
  hl_ctx* ctx = m->ctx;
  const hl_decoder_config& c = m->cfg;
  const int N = m->N, d = c.d_model, F = c.d_ff, V = c.vocab, B = c.batch, T = c.context, H = c.n_heads;
  const float* P = m->params;
  float* G = m->grads;
  m->next_bucket = 0;
  if (m->comm_pending) {  // a previous step's collectives were never consumed: finish them before its gradients are overwritten
    HL_CUDA(cudaStreamWaitEvent(m->ctx->stream, m->comm_done, 0));
    m->comm_pending = false;
  }
  FoldBatch* fb = &m->fold;
  fb->n = 0;
  fb->used = 0;
  // Everything up to arena element `done` has been written, the layer norms' parameter gradients apart, which are folded
  // by one launch per full batch unless a bucket of the gradient exchange is waiting for them.
  auto finished = [&](size_t done) -> int {
    if (nccl_active(ctx) || done == m->arena) HL_TRY(fold_batch_flush(ctx, fb));
    return flush_buckets(m, done);
  };
  HL_TRY(cross_entropy_impl(ctx, m->logits, V, m->targets, N, V, 1.0f, m->loss_dev, nullptr, m->dlogits_f, HL_F32, V, m->loss_host));
  if (m->has_memory) HL_TRY(tables_are_zero(m));
  float* dx = m->lf[c.n_layers - 1].dy;  // gradient of the residual stream
  HL_TRY(linear_backward_f32(m, m->zf, P + m->off_head_w, m->dlogits_f, m->d_c, G + m->off_head_w, G + m->off_head_b, N, d, V));
  HL_TRY(layer_norm_backward_impl(ctx, m->xf[c.n_layers], HL_F32, P + m->off_lnf_g, m->d_c, nullptr, nullptr, nullptr, dx,
                                  nullptr, G + m->off_lnf_g, G + m->off_lnf_b, nullptr, N, d, fb));
  HL_TRY(finished(m->off_lnf_b + d));
  for (int l = c.n_layers - 1; l >= 0; --l) {
    const LayerOffsets& o = m->lo[l];
    hl_decoder::F32Layer& a = m->lf[l];
    if (o.is_memory) {
      MemoryActs& ma = m->ma[l];
      const int kd = m->mem.key_dim, vd = m->mem.value_dim;
      const size_t nv = (size_t)N * vd;
      HL_TRY(linear_backward_f32(m, ma.mv, P + o.wout_m, dx, m->m_dmv, G + o.wout_m, G + o.bout_m, N, vd, d));
      HL_TRY(hl_binary_f32(ctx, HL_MUL, m->m_dmv, ma.gate, m->m_dweighted, nv));
      HL_TRY(hl_binary_f32(ctx, HL_MUL, m->m_dmv, ma.weighted, m->m_dgate, nv));
      HL_TRY(hl_gelu_backward(ctx, ma.gpre, m->m_dgate, m->m_dgpre, HL_F32, nv));
      HL_TRY(linear_backward_f32(m, a.c, P + o.wg_m, m->m_dgpre, m->d_c, G + o.wg_m, G + o.bg_m, N, d, vd));
      HL_TRY(join_side(m));  // its buffers are those of the block above
      HL_TRY(memory_core_backward(m, l, m->m_dweighted));
      // the query path's input gradient is added to the gate path's
      HL_TRY(linear_backward_f32(m, a.c, P + o.wq_m, m->m_dq, m->d_c, G + o.wq_m, G + o.bq_m, N, d, kd, F64_ACCUMULATE));
    } else {
      // y = r + fc2(gelu(fc1(ln2 r)))
      HL_TRY(linear_backward_f32(m, a.g, P + o.w2, dx, a.dwide, G + o.w2, G + o.b2, N, F, d, F64_DGELU, a.h));
      HL_TRY(linear_backward_f32(m, a.c, P + o.w1, a.dwide, m->d_c, G + o.w1, G + o.b1, N, d, F));
    }
    HL_TRY(layer_norm_backward_impl(ctx, a.r, HL_F32, P + o.ln2g, m->d_c, nullptr, nullptr, dx, a.dr, nullptr, G + o.ln2g,
                                    G + o.ln2b, nullptr, N, d, fb));
    dx = a.dr;
    // r = x + out_proj(attention(q, k, v))
    HL_TRY(linear_backward_f32(m, a.o, P + o.wo, dx, m->d_c, G + o.wo, G + o.bo, N, d, d));
    HL_TRY(attention_f64_backward(ctx, a.qkv, a.qkv + d, a.qkv + 2 * d, HL_F32, 3 * d, a.probs, m->d_c, d, a.dqkv,
                                  a.dqkv + d, a.dqkv + 2 * d, 3 * d, B, T, d, H));
    HL_TRY(linear_backward_f32(m, a.a, P + o.wqkv, a.dqkv, m->d_c, G + o.wqkv, G + o.bqkv, N, d, 3 * d));
    float* dx_next = l > 0 ? m->lf[l - 1].dy : m->d_a;
    HL_TRY(layer_norm_backward_impl(ctx, m->xf[l], HL_F32, P + o.ln1g, m->d_c, nullptr, nullptr, dx, dx_next, nullptr,
                                    G + o.ln1g, G + o.ln1b, nullptr, N, d, fb));
    dx = dx_next;
    HL_TRY(finished(o.ln1b + d));
  }
  if (!m->has_memory) HL_TRY(tables_are_zero(m));
  if (beside(m)) {
    SideStream side(m);
    HL_TRY(side.rc);
    HL_TRY(fold_batch_flush(ctx, fb));
  }
  HL_TRY(hl_embedding_backward(ctx, dx, m->tokens, G + m->off_tok, V, G + m->off_pos, T, N, d));
  HL_TRY(join_side(m));
  HL_TRY(finished(m->arena));
  if (nccl_active(ctx)) {
    if (m->has_memory || m->sparse_tok_exchange) {
      // the row exchanges read gradients the compute stream is still producing
      HL_CUDA(cudaEventRecord(m->comm_done, ctx->stream));
      HL_CUDA(cudaStreamWaitEvent(ctx->comm_stream, m->comm_done, 0));
      HL_TRY(exchange_token_rows(m));
      HL_TRY(exchange_value_rows(m));
    }
    // The compute stream waits for the collectives only when something reads the averaged gradients:
    // the optimizer takes them bucket group by bucket group, every other reader waits for all of them.
    HL_CUDA(cudaEventRecord(m->comm_done, ctx->comm_stream));
    m->comm_pending = true;
  }
  return HL_OK;
}

// The launches of `queue` as a graph on the device, or false with nothing queued and no error left behind (a device without memory
// for it, say).
template <typename F>
bool capture_pass(hl_decoder* m, F queue, cudaGraphExec_t* exec) {
  hl_ctx* ctx = m->ctx;
  cudaGraph_t graph = nullptr;
  bool ok = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
  if (ok) {
    ok = queue() == HL_OK;
    ok = cudaStreamEndCapture(ctx->stream, &graph) == cudaSuccess && ok;
  }
  ok = ok && cudaGraphInstantiate(exec, graph, 0) == cudaSuccess;
  ok = ok && cudaGraphUpload(*exec, ctx->stream) == cudaSuccess;
  if (graph) cudaGraphDestroy(graph);
  if (!ok) {
    if (*exec) cudaGraphExecDestroy(*exec);
    *exec = nullptr;
    m->forked = false;  // what was forked ended with the capture
    cudaGetLastError();
  }
  return ok;
}

// Queues the launches of `queue` on the compute stream, from the second time on as a graph.
template <typename F>
int run_graphed(hl_decoder* m, int kind, F queue) {
  hl_ctx* ctx = m->ctx;
  auto setting = [](const char* name) { const char* e = getenv(name); return e ? e[0] : '\0'; };
  const char dynamic = setting("HEIRLOOM_GEMM_DYNAMIC");
  // Collectives and per-kernel timing are host work of the step; the test hook changes a launch's arguments; and a launch that
  // draws its tiles from the counter carries the counter's value, which no two launches share.
  if (nccl_active(ctx) || ctx->profiler || ctx->gemm_skip_kblock >= 0 || m->comm_pending || dynamic == '1') return queue();
  // A caller that captures the context's stream gets the launches themselves.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  HL_CUDA(cudaStreamIsCapturing(ctx->stream, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return queue();
  const GraphKey key{kind, m->cfg.batch, m->cfg.context, ctx->workspace, ctx->workspace_bytes, ctx->wait_limit_ns, ctx->faults,
                     setting("HEIRLOOM_GEMM_PAIRS"), dynamic};
  std::vector<GraphEntry>& entries = m->graphs.entries;
  GraphEntry* entry = nullptr;
  for (GraphEntry& e : entries)
    if (e.key == key) entry = &e;
  if (!entry) {
    if (entries.size() < kMaxGraphs) entries.emplace_back();
    entry = &*std::min_element(entries.begin(), entries.end(), [](const GraphEntry& a, const GraphEntry& b) { return a.used < b.used; });
    if (entry->exec) {
      HL_CUDA(cudaStreamSynchronize(ctx->stream));
      cudaGraphExecDestroy(entry->exec);
    }
    *entry = GraphEntry{};
    entry->key = key;
    entry->used = ++m->graphs.clock;
    HL_TRY(queue());
    // the plain run may have grown the scratch arena
    entry->key.workspace = ctx->workspace;
    entry->key.workspace_bytes = ctx->workspace_bytes;
    return HL_OK;
  }
  entry->used = ++m->graphs.clock;
  if (entry->plain) return queue();
  if (!entry->exec) {
    const Counters before = ctx->counters;
    if (!capture_pass(m, queue, &entry->exec)) {  // what cannot be captured runs as it did the first time, now and from now on
      entry->plain = true;
      ctx->counters = before;
      return queue();
    }
    Counters& c = entry->counts;
    c.launches = ctx->counters.launches - before.launches;
    c.gemm_tcgen05_launches = ctx->counters.gemm_tcgen05_launches - before.gemm_tcgen05_launches;
    c.gemm_pair_launches = ctx->counters.gemm_pair_launches - before.gemm_pair_launches;
    c.attention_launches = ctx->counters.attention_launches - before.attention_launches;
  } else {
    ctx->counters.launches += entry->counts.launches;
    ctx->counters.gemm_tcgen05_launches += entry->counts.gemm_tcgen05_launches;
    ctx->counters.gemm_pair_launches += entry->counts.gemm_pair_launches;
    ctx->counters.attention_launches += entry->counts.attention_launches;
  }
  HL_CUDA(cudaGraphLaunch(entry->exec, ctx->stream));
  return HL_OK;
}

// ---- one-token steps of generation -----------------------------------------------------------------
// The row of m->decode_state through the model: its q/k/v go to the cache (row `position` of the activations that a
// full-window forward left), every other value of the row to row 0 of its buffer, the logits to row 0 of m->logits.  Row by
// row this is what forward() and forward_f32() compute (N is 1 meanwhile).
int decode_step(hl_decoder* m) {
  hl_ctx* ctx = m->ctx;
  const hl_decoder_config& c = m->cfg;
  const int d = c.d_model;
  const bool amp = c.precision == HL_PRECISION_AMP_BF16;
  const int dt = amp ? HL_BF16 : HL_F32;
  const float* P = m->params;
  auto gemv = [&](const void* x, size_t w, size_t b, void* out, int n, int k, int epilogue = GV_STORE, const void* residual = nullptr,
                  size_t ln_g = 0, size_t ln_b = 0) { return row_gemv(m, x, w, b, out, n, k, epilogue, residual, ln_g, ln_b); };
  const bool fused = row_block_fused(m);
  DecodeRow row{};  // fused: the row so far
  row.table = P + m->off_tok; row.positions = P + m->off_pos; row.state = m->decode_state;
  if (!fused) HL_TRY(decode_embed(ctx, P + m->off_tok, P + m->off_pos, m->decode_state, amp ? (void*)m->x[0] : (void*)m->xf[0], dt, d));
  for (int l = 0; l < c.n_layers; ++l) {
    const LayerOffsets& o = m->lo[l];
    void *x, *next, *qkv, *r;
    if (amp) { x = m->x[l]; next = m->x[l + 1]; qkv = m->la[l].qkv; r = m->la[l].r; }
    else { x = m->xf[l]; next = m->xf[l + 1]; qkv = m->lf[l].qkv; r = m->lf[l].r; }
    if (fused) {
      HL_TRY(row_block_fused(m, l, row, false, &row));
      if (o.is_memory) HL_TRY(decode_row(ctx, row, dt, d));
    } else {
      // the attention output, r and g rows may lie over cached positions' rows: only the q/k/v rows are kept
      DecodeGemv q = gemv(x, o.wqkv, o.bqkv, qkv, 3 * d, d, GV_STORE, nullptr, o.ln1g, o.ln1b);
      q.out_row = m->decode_state;
      q.ld_out = 3 * d;
      HL_TRY(decode_gemv(ctx, q));
      HL_TRY(row_block(m, l, x, true));
    }
    if (o.is_memory) {
      MemoryActs& ma = m->ma[l];
      const int kd = m->mem.key_dim, vd = m->mem.value_dim;
      // f32 weights against the normalised row: as accurate as the pieces the full-window route multiplies
      auto project = [&](const void* in, int in_dtype, size_t w, size_t b, void* out, int out_dtype, int n, int k, int epilogue,
                         const void* residual, bool ln) {
        DecodeGemv p = gemv(in, w, b, out, n, k, epilogue, residual, ln ? o.ln2g : 0, ln ? o.ln2b : 0);
        p.x_dtype = in_dtype; p.w = P + w; p.w_dtype = HL_F32; p.out_dtype = out_dtype;
        return decode_gemv(ctx, p);
      };
      HL_TRY(project(r, dt, o.wq_m, o.bq_m, ma.query, HL_F32, kd, d, GV_STORE, nullptr, true));
      HL_TRY(memory_core_forward(m, l, true));
      HL_TRY(project(r, dt, o.wg_m, o.bg_m, ma.gate, HL_F32, vd, d, GV_GELU, nullptr, true));
      HL_TRY(hl_binary_f32(ctx, HL_MUL, ma.weighted, ma.gate, ma.mv, (size_t)vd));
      HL_TRY(project(ma.mv, HL_F32, o.wout_m, o.bout_m, next, dt, d, vd, GV_RESIDUAL, r, false));
      row = DecodeRow{};
      row.base = next;
    }
  }
  if (fused) return row_head(m, row);
  return decode_head(m, amp ? (const void*)m->x[c.n_layers] : (const void*)m->xf[c.n_layers], dt);
}

int ensure_logits_host(hl_decoder* m) {
  if (!m->logits_host) {
    HL_CUDA(cudaMallocHost(reinterpret_cast<void**>(&m->logits_host), sizeof(float) * (size_t)m->cfg.vocab + 64));
    m->decode_state_host = reinterpret_cast<long long*>(m->logits_host + ((m->cfg.vocab + 3) & ~3));
    m->greedy_host = reinterpret_cast<GreedyPart*>(m->decode_state_host + 2);
  }
  return HL_OK;
}

// The compute stream waits for `ev` of the collective stream.  With per-kernel timing on, the wait is bracketed by two
// timing events: the first completes when the compute stream has run dry, the second when the collective has arrived,
// so their distance is the time this wait left the GPU's compute stream idle.
int wait_on_collective(hl_decoder* m, cudaEvent_t ev) {
  cudaStream_t s = m->ctx->stream;
  const bool timed = m->ctx->profiler != nullptr;
  if (timed) {
    if (m->waits_recorded == m->wait_begin.size()) {
      cudaEvent_t a = nullptr, b = nullptr;
      HL_CUDA(cudaEventCreate(&a));
      HL_CUDA(cudaEventCreate(&b));
      m->wait_begin.push_back(a);
      m->wait_end.push_back(b);
    }
    HL_CUDA(cudaEventRecord(m->wait_begin[m->waits_recorded], s));
  }
  HL_CUDA(cudaStreamWaitEvent(s, ev, 0));
  if (timed) {
    HL_CUDA(cudaEventRecord(m->wait_end[m->waits_recorded], s));
    m->waits_recorded += 1;
  }
  return HL_OK;
}

// Make the compute stream wait for every gradient collective of the step.
int wait_for_collectives(hl_decoder* m) {
  if (m->comm_pending) {
    HL_TRY(wait_on_collective(m, m->comm_done));
    m->comm_pending = false;
  }
  m->ctx->reserve_sms = 0;
  return HL_OK;
}

int optimizer_step(hl_decoder* m) {
  HL_REQUIRE(m->has_opt, "hl_decoder: no optimizer configured (call hl_decoder_set_optimizer)");
  hl_ctx* ctx = m->ctx;
  if (m->opt.clip_norm > 0.f) HL_TRY(wait_for_collectives(m));  // the global norm needs every averaged gradient
  const int world = nccl_world(ctx);
  const float inv_world = 1.0f / (float)world;  // sum then scale by 1/world (src/nn.rs:2100-2117)
  // The norm of the averaged gradients: the clipping factor is worked out on the device, so that the update does not wait for the host
  // to have read the norm, which it does like the reference, to refuse a step whose norm is not finite.
  const bool clipped = m->opt.clip_norm > 0.f;
  if (clipped) HL_TRY(sum_squares_impl(ctx, m->grads, m->arena, m->norm_dev, m->norm_host));
  m->step += 1;
  hl_adamw_params hp{};
  hp.lr = m->opt.lr; hp.beta1 = m->opt.beta1; hp.beta2 = m->opt.beta2; hp.eps = m->opt.eps;
  hp.weight_decay = m->opt.weight_decay;
  hp.clip_scale = inv_world;
  hp.bias_correction1 = (float)(1.0 - pow((double)m->opt.beta1, (double)m->step));
  hp.bias_correction2 = (float)(1.0 - pow((double)m->opt.beta2, (double)m->step));
  if (clipped) {  // every collective has been waited for
    HL_TRY(adam_plan_step(ctx, m->plan, &hp, AdamClip{m->norm_dev, (double)inv_world, (double)m->opt.clip_norm}));
    HL_CUDA(cudaStreamSynchronize(ctx->stream));
    const double sum_sq = (double)m->norm_host[0] * (double)inv_world * (double)inv_world;
    if (sum_sq >= 0.0 && sum_sq <= 1e300) return HL_OK;
    m->step -= 1;  // nothing was updated
    return fail("non-finite or negative global gradient sum-of-squares");
  }
  if (!m->comm_pending) return adam_plan_step(ctx, m->plan, &hp);
  // Collectives still in flight: update the arena in groups of buckets, each group as soon as its last
  // all-reduce has finished, so the update of the early buckets overlaps the reduction of the late ones.
  const size_t chunk = (size_t)adam_plan_chunk_elements(m->plan);
  const int chunks_total = adam_plan_chunk_count(m->plan);
  constexpr size_t kGroup = 5;  // buckets per launch
  int first = 0;
  for (size_t b0 = 0; b0 < m->n_buckets; b0 += kGroup) {
    const size_t b1 = std::min(b0 + kGroup, m->n_buckets);
    size_t start, end;
    bucket_range(m->arena, m->bucket_elems, b1 - 1, &start, &end);
    // chunks that lie completely inside the buckets reduced so far (a chunk that straddles the boundary waits
    // for the next group; the last group takes everything that is left)
    const int upto = b1 == m->n_buckets ? chunks_total : (int)(end / chunk);
    // The gradients of the value table and of the token-embedding table are not final when their buckets are: their
    // rows are summed over the ranks by the row exchanges that follow the last bucket on the collective stream.  A
    // group that reaches into such a table waits for the end of that stream's work (which covers every bucket too).
    const size_t range_end = b1 == m->n_buckets ? m->arena : (size_t)upto * chunk;
    const bool reaches_values = (m->has_memory && range_end > m->off_val) || (m->sparse_tok_exchange && range_end > m->off_tok);
    HL_TRY(wait_on_collective(m, reaches_values ? m->comm_done : m->bucket_done[b1 - 1]));
    HL_TRY(adam_plan_step_range(ctx, m->plan, &hp, first, upto - first));
    first = upto;
  }
  m->comm_pending = false;
  ctx->reserve_sms = 0;
  return HL_OK;
}

int refresh_shadow(hl_decoder* m, size_t offset, size_t numel) {
  return hl_cast(m->ctx, m->params + offset, HL_F32, m->shadow + offset, HL_BF16, numel);
}

}  // namespace
}  // namespace hl

extern "C" {

static int decoder_create_impl(hl_ctx* ctx, const hl_decoder_config* cfg, const hl_memory_config* mem, hl_decoder** out);

int hl_decoder_create(hl_ctx* ctx, const hl_decoder_config* cfg, hl_decoder** out) {
  return decoder_create_impl(ctx, cfg, nullptr, out);
}

int hl_memory_decoder_create(hl_ctx* ctx, const hl_decoder_config* cfg, const hl_memory_config* mem, hl_decoder** out) {
  HL_REQUIRE(mem, "hl_memory_decoder_create: null memory configuration");
  return decoder_create_impl(ctx, cfg, mem, out);
}

int hl_decoder_selected_indices(hl_decoder* m, int layer, int64_t* host, long long count) {
  HL_REQUIRE(m && host, "hl_decoder_selected_indices: null argument");
  HL_REQUIRE(m->has_memory && layer >= 0 && layer < m->cfg.n_layers && m->lo[layer].is_memory,
             "hl_decoder_selected_indices: block " + std::to_string(layer) + " has no memory feed-forward");
  HL_REQUIRE(count == (long long)m->N * m->mem.top_k, "hl_decoder_selected_indices: expected tokens * top_k entries");
  return hl_memory_copy_indices(m->ctx, host, m->ma[layer].idx, count);
}

static int decoder_create_impl(hl_ctx* ctx, const hl_decoder_config* cfg, const hl_memory_config* mem, hl_decoder** out) {
  HL_REQUIRE(ctx && cfg && out, "hl_decoder_create: null argument");
  *out = nullptr;
  int side = 0;
  if (mem && mem->n_memory_layers > 0) {
    HL_REQUIRE(mem->n_memory_layers <= 16, "hl_memory_decoder_create: at most 16 memory layers");
    for (int i = 0; i < mem->n_memory_layers; ++i)
      HL_REQUIRE(mem->memory_layers[i] >= 0 && mem->memory_layers[i] < cfg->n_layers,
                 "hl_memory_decoder_create: memory layer index out of range");
    HL_REQUIRE(mem->slots > 0 && mem->key_dim > 0 && mem->value_dim > 0 && mem->top_k > 0,
               "hl_memory_decoder_create: memory sizes must be positive");
    side = (int)sqrt((double)mem->slots);
    HL_REQUIRE((long long)side * side == mem->slots,
               "product-key memory lookup requires square memory_slots, got " + std::to_string(mem->slots));
    HL_REQUIRE(mem->key_dim % 2 == 0, "product-key memory lookup requires even memory_key_dim, got " + std::to_string(mem->key_dim));
    HL_REQUIRE(mem->memory_heads == 1, "memory_heads=" + std::to_string(mem->memory_heads) +
                                           " requested, but the memory feed-forward supports one memory head");
    HL_REQUIRE(mem->value_dim % 8 == 0 && mem->key_dim % 8 == 0, "hl_memory_decoder_create: key_dim and value_dim must be multiples of 8");
    HL_REQUIRE(side <= 2048 && mem->top_k <= 1024, "hl_memory_decoder_create: side <= 2048 and top_k <= 1024");
  }
  HL_REQUIRE(cfg->vocab > 0 && cfg->d_model > 0 && cfg->n_layers > 0 && cfg->n_heads > 0 && cfg->d_ff > 0 &&
                 cfg->context > 0 && cfg->batch > 0,
             "hl_decoder_create: every size must be positive");
  HL_REQUIRE(cfg->d_model % cfg->n_heads == 0, "hl_decoder_create: d_model must be divisible by n_heads");
  HL_REQUIRE(cfg->precision == HL_PRECISION_AMP_BF16 || cfg->precision == HL_PRECISION_F32,
             "hl_decoder_create: precision must be HL_PRECISION_F32 or HL_PRECISION_AMP_BF16");
  const bool amp = cfg->precision == HL_PRECISION_AMP_BF16;
  if (amp) {
    HL_REQUIRE(cfg->d_model % 8 == 0 && cfg->d_ff % 8 == 0 && cfg->vocab % 8 == 0 && cfg->d_model <= 1024,
               "hl_decoder_create: d_model (<= 1024), d_ff and vocab must be multiples of 8");
    if (mem && mem->n_memory_layers > 0)  // the projections' contraction is read piecewise in whole 64-element blocks
      HL_REQUIRE(cfg->d_model % 64 == 0 && mem->value_dim % 32 == 0 && mem->key_dim % 32 == 0 &&
                     (cfg->batch * cfg->context) % 64 == 0,
                 "hl_memory_decoder_create: the bf16 route needs d_model and batch*context to be multiples of 64, "
                 "key_dim and value_dim of 32");
  } else {
    HL_REQUIRE(cfg->d_model % 4 == 0 && cfg->d_model <= 1024,
               "hl_decoder_create: the f32 route needs d_model to be a multiple of 4 and at most 1024");
  }
  hl_decoder* m = new hl_decoder();
  m->ctx = ctx;
  m->cfg = *cfg;
  m->N = cfg->batch * cfg->context;
  m->flash_ok = cfg->d_model / cfg->n_heads == 64 || cfg->d_model / cfg->n_heads == 128;
  if (mem && mem->n_memory_layers > 0) {
    m->has_memory = true;
    m->mem = *mem;
    m->side = side;
  }
  plan_parameters(m);
  auto cleanup = [&](int rc) { hl_decoder_destroy(m); return rc; };
  cudaError_t e;
  const size_t fb = sizeof(float) * m->arena;
#define HL_ALLOC(ptr, bytes)                                              \
  e = cudaMalloc(reinterpret_cast<void**>(&(ptr)), (bytes));               \
  if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaMalloc(" #ptr ")"));
  HL_ALLOC(m->params, fb)
  HL_ALLOC(m->grads, fb)
  HL_ALLOC(m->m, fb)
  HL_ALLOC(m->v, fb)
  HL_ALLOC(m->shadow, sizeof(__nv_bfloat16) * m->arena)
  size_t act = 0;
  auto plan = [&](bool measure_only) { if (amp) plan_activations(m, measure_only, &act); else plan_activations_f32(m, measure_only, &act); };
  // Copies of operands for weight gradients beside or behind the backward pass (up to 256 MB, or a gigabyte) are only made where the
  // device has a gigabyte left behind them and behind the attention's scratch, so that a model fits wherever it did without them;
  // and not beside a communicator, which uses none of them.  Asking for the free memory takes a millisecond, a fifth of a small
  // model's creation: copies below 32 MB, a block of the driver's pool, are made where their allocation succeeds.
  m->lean = true;
  plan(true);
  const size_t without = act;
  m->lean = nccl_active(ctx);
  plan(true);
  if (act > without) {
    bool room = true;
    if (act - without >= (size_t(32) << 20)) {
      const size_t scores = (size_t)cfg->batch * cfg->n_heads * cfg->context * cfg->context * sizeof(float);
      const size_t behind = kGroupBytes + (amp && m->flash_ok ? flash_attention_backward_scratch_bytes(cfg->batch, cfg->context, cfg->n_heads,
                                                                                                      cfg->d_model / cfg->n_heads) : scores);
      size_t free_bytes = 0, total_bytes = 0;
      e = cudaMemGetInfo(&free_bytes, &total_bytes);
      if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaMemGetInfo"));
      room = free_bytes >= act + behind;
    }
    if (!room || cudaMalloc(reinterpret_cast<void**>(&m->act_arena), act) != cudaSuccess) {
      cudaGetLastError();
      m->act_arena = nullptr;
      m->lean = true;
      plan(true);
    }
  }
  m->act_bytes = act;
  if (!m->act_arena) {
    HL_ALLOC(m->act_arena, act)
  }
#undef HL_ALLOC
  plan(false);
  cudaMemsetAsync(m->params, 0, fb, ctx->stream);
  cudaMemsetAsync(m->grads, 0, fb, ctx->stream);
  cudaMemsetAsync(m->m, 0, fb, ctx->stream);
  cudaMemsetAsync(m->v, 0, fb, ctx->stream);
  cudaMemsetAsync(m->shadow, 0, sizeof(__nv_bfloat16) * m->arena, ctx->stream);
  e = cudaMallocHost(reinterpret_cast<void**>(&m->loss_host), 64);
  if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaMallocHost"));
  m->norm_host = m->loss_host + 8;
  m->m_union_count_host = reinterpret_cast<int*>(m->loss_host + 12);
  m->tok_union_count_host = reinterpret_cast<int*>(m->loss_host + 13);
  if (const char* e = getenv("HEIRLOOM_SPARSE_EMBEDDING_EXCHANGE")) m->sparse_tok_exchange = atoi(e) != 0;
  hl_adamw_tensor whole{m->params, m->grads, m->m, m->v, m->shadow, (uint64_t)m->arena};
  int rc = adam_plan_create(ctx, &whole, 1, &m->plan);
  if (rc != HL_OK) return cleanup(rc);
  if (m->has_memory) {
    auto span = [&](size_t begin, size_t end) {
      return hl_adamw_tensor{m->params + begin, m->grads + begin, m->m + begin, m->v + begin, m->shadow + begin,
                             (uint64_t)(end - begin)};
    };
    hl_adamw_tensor tables = span(m->off_kl, m->tables_end);
    rc = adam_plan_create(ctx, &tables, 1, &m->plan_tables);
    if (rc != HL_OK) return cleanup(rc);
    hl_adamw_tensor rest[2] = {span(0, m->off_val), span(m->tables_end, m->arena)};
    rc = adam_plan_create(ctx, rest, 2, &m->plan_no_values);
    if (rc != HL_OK) return cleanup(rc);
  }
  m->n_buckets = (m->arena + m->bucket_elems - 1) / m->bucket_elems;
  m->bucket_ready.resize(m->n_buckets);
  m->bucket_done.resize(m->n_buckets);
  for (auto& ev : m->bucket_done) {
    cudaError_t ee = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (ee != cudaSuccess) { ev = nullptr; return fail_cuda(ee, "cudaEventCreate(bucket_done)"); }
  }
  for (auto& ev : m->bucket_ready) {
    e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaEventCreate"));
  }
  for (cudaEvent_t* ev : {&m->rows_known, &m->tok_count_ready, &m->val_count_ready}) {
    e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    if (e != cudaSuccess) { *ev = nullptr; return fail_cuda(e, "cudaEventCreate(row exchange)"); }
  }
  {
    e = cudaStreamCreateWithFlags(&m->side_stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->fork_event, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->join_event, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->zero_event, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->sort_event, cudaEventDisableTiming);
    if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaStreamCreate(side)"));
  }
  e = cudaEventCreateWithFlags(&m->comm_done, cudaEventDisableTiming);
  if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaEventCreate"));
  e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cleanup(fail_cuda(e, "cudaStreamSynchronize"));
  ctx->counters.allocations += 6;
  ctx->counters.allocated_bytes += 4 * fb + sizeof(__nv_bfloat16) * m->arena + act;
  *out = m;
  return HL_OK;
}

void hl_decoder_destroy(hl_decoder* m) {
  if (!m) return;
  if (m->ctx) {
    cudaStreamSynchronize(m->ctx->stream);
    cudaStreamSynchronize(m->ctx->comm_stream);
  }
  for (auto ev : m->bucket_ready) if (ev) cudaEventDestroy(ev);
  for (auto ev : m->bucket_done) if (ev) cudaEventDestroy(ev);
  if (m->comm_done) cudaEventDestroy(m->comm_done);
  if (m->side_stream) cudaStreamDestroy(m->side_stream);
  if (m->fork_event) cudaEventDestroy(m->fork_event);
  if (m->zero_event) cudaEventDestroy(m->zero_event);
  if (m->sort_event) cudaEventDestroy(m->sort_event);
  if (m->join_event) cudaEventDestroy(m->join_event);
  for (cudaEvent_t ev : {m->rows_known, m->tok_count_ready, m->val_count_ready}) if (ev) cudaEventDestroy(ev);
  for (auto ev : m->wait_begin) cudaEventDestroy(ev);
  for (auto ev : m->wait_end) cudaEventDestroy(ev);
  adam_plan_destroy(m->plan);
  adam_plan_destroy(m->plan_tables);
  adam_plan_destroy(m->plan_no_values);
  if (m->m_packed) cudaFree(m->m_packed);
  if (m->tok_packed) cudaFree(m->tok_packed);
  cudaFree(m->params); cudaFree(m->grads); cudaFree(m->m); cudaFree(m->v); cudaFree(m->shadow); cudaFree(m->act_arena);
  if (m->loss_host) cudaFreeHost(m->loss_host);
  if (m->logits_host) cudaFreeHost(m->logits_host);
  m->graphs.clear();
  delete m;
}

int hl_decoder_param_count(hl_decoder* m) { return m ? (int)m->slots.size() : 0; }

int hl_decoder_param_info(hl_decoder* m, int index, char* name_out, size_t name_cap, long long* numel, int* rank,
                          long long shape_out[2]) {
  HL_REQUIRE(m, "hl_decoder_param_info: null model");
  HL_REQUIRE(index >= 0 && index < (int)m->slots.size(), "hl_decoder_param_info: parameter index out of range");
  const Slot& s = m->slots[index];
  if (name_out && name_cap > 0) {
    strncpy(name_out, s.name.c_str(), name_cap - 1);
    name_out[name_cap - 1] = 0;
  }
  if (numel) *numel = (long long)s.numel;
  if (rank) *rank = s.rank;
  if (shape_out) { shape_out[0] = s.shape[0]; shape_out[1] = s.shape[1]; }
  return HL_OK;
}

static int slot_io(hl_decoder* m, int index, long long numel, const Slot** out, const char* who) {
  HL_REQUIRE(m, std::string(who) + ": null model");
  HL_REQUIRE(index >= 0 && index < (int)m->slots.size(), std::string(who) + ": parameter index out of range");
  const Slot& s = m->slots[index];
  HL_REQUIRE(numel == (long long)s.numel, std::string(who) + ": parameter " + s.name + " has " + std::to_string(s.numel) +
                                              " elements, got " + std::to_string(numel));
  *out = &s;
  return HL_OK;
}

int hl_decoder_set_param(hl_decoder* m, int index, const float* host, long long numel) {
  const Slot* s;
  HL_TRY(slot_io(m, index, numel, &s, "hl_decoder_set_param"));
  HL_TRY(hl_memcpy_h2d(m->ctx, m->params + s->offset, host, sizeof(float) * s->numel));
  m->cached = 0;
  return refresh_shadow(m, s->offset, s->numel);
}

int hl_decoder_get_param(hl_decoder* m, int index, float* host, long long numel) {
  const Slot* s;
  HL_TRY(slot_io(m, index, numel, &s, "hl_decoder_get_param"));
  return hl_memcpy_d2h(m->ctx, host, m->params + s->offset, sizeof(float) * s->numel);
}

int hl_decoder_get_grad(hl_decoder* m, int index, float* host, long long numel) {
  const Slot* s;
  HL_TRY(slot_io(m, index, numel, &s, "hl_decoder_get_grad"));
  HL_TRY(hl::wait_for_collectives(m));
  return hl_memcpy_d2h(m->ctx, host, m->grads + s->offset, sizeof(float) * s->numel);
}

int hl_decoder_get_moments(hl_decoder* m, int index, float* m_host, float* v_host, long long numel) {
  const Slot* s;
  HL_TRY(slot_io(m, index, numel, &s, "hl_decoder_get_moments"));
  HL_TRY(hl_memcpy_d2h(m->ctx, m_host, m->m + s->offset, sizeof(float) * s->numel));
  return hl_memcpy_d2h(m->ctx, v_host, m->v + s->offset, sizeof(float) * s->numel);
}

int hl_decoder_set_optimizer(hl_decoder* m, const hl_adamw_config* opt) {
  HL_REQUIRE(m && opt, "hl_decoder_set_optimizer: null argument");
  HL_REQUIRE(opt->lr >= 0.f && opt->beta1 >= 0.f && opt->beta1 < 1.f && opt->beta2 >= 0.f && opt->beta2 < 1.f &&
                 opt->eps > 0.f && opt->weight_decay >= 0.f,
             "hl_decoder_set_optimizer: invalid AdamW hyper-parameters");
  m->opt = *opt;
  m->has_opt = true;
  m->step = 0;
  HL_CUDA(cudaMemsetAsync(m->m, 0, sizeof(float) * m->arena, m->ctx->stream));
  HL_CUDA(cudaMemsetAsync(m->v, 0, sizeof(float) * m->arena, m->ctx->stream));
  return HL_OK;
}

long long hl_decoder_optimizer_steps(hl_decoder* m) { return m ? m->step : 0; }

int hl_decoder_set_moments(hl_decoder* m, int index, const float* m_host, const float* v_host, long long numel) {
  const Slot* s;
  HL_TRY(slot_io(m, index, numel, &s, "hl_decoder_set_moments"));
  HL_REQUIRE(m_host && v_host, "hl_decoder_set_moments: null argument");
  HL_REQUIRE(m->has_opt, "hl_decoder_set_moments: no optimizer configured (call hl_decoder_set_optimizer)");
  HL_TRY(hl_memcpy_h2d(m->ctx, m->m + s->offset, m_host, sizeof(float) * s->numel));
  return hl_memcpy_h2d(m->ctx, m->v + s->offset, v_host, sizeof(float) * s->numel);
}

int hl_decoder_set_optimizer_steps(hl_decoder* m, long long steps) {
  HL_REQUIRE(m, "hl_decoder_set_optimizer_steps: null model");
  HL_REQUIRE(m->has_opt, "hl_decoder_set_optimizer_steps: no optimizer configured (call hl_decoder_set_optimizer)");
  HL_REQUIRE(steps >= 0, "hl_decoder_set_optimizer_steps: the step counter cannot be negative");
  m->step = steps;
  return HL_OK;
}

int hl_decoder_forward_backward(hl_decoder* m, const int64_t* tokens_dev, const int64_t* targets_dev) {
  HL_REQUIRE(m && tokens_dev && targets_dev, "hl_decoder_forward_backward: null argument");
  const unsigned long long before = m->ctx->counters.launches;
  if (tokens_dev != m->tokens)
    HL_CUDA(cudaMemcpyAsync(m->tokens, tokens_dev, sizeof(int64_t) * m->N, cudaMemcpyDeviceToDevice, m->ctx->stream));
  if (targets_dev != m->targets)
    HL_CUDA(cudaMemcpyAsync(m->targets, targets_dev, sizeof(int64_t) * m->N, cudaMemcpyDeviceToDevice, m->ctx->stream));
  m->cached = 0;  // the pass overwrites the cached rows from its first kernel on, whether or not it gets to its end
  HL_TRY(run_graphed(m, GRAPH_STEP, [m]() -> int {
    struct Sorting {  // a backward pass follows
      hl_decoder* m;
      ~Sorting() { m->sorted = false; }
    } sorting{m};
    m->sorted = beside(m);
    HL_TRY(zero_tables_beside(m));
    HL_TRY(prepare_token_rows(m));  // data parallel: the union of the ranks' token rows forms while forward runs
    if (m->cfg.precision == HL_PRECISION_AMP_BF16) {
      HL_TRY(forward(m));
      HL_TRY(prepare_value_rows(m));
      return backward(m);
    }
    HL_TRY(forward_f32(m));
    HL_TRY(prepare_value_rows(m));
    return backward_f32(m);
  }));
  m->launches_last_step = m->ctx->counters.launches - before;
  return HL_OK;
}

int hl_decoder_optimizer_step(hl_decoder* m) {
  HL_REQUIRE(m, "hl_decoder_optimizer_step: null model");
  const unsigned long long before = m->ctx->counters.launches;
  m->cached = 0;
  HL_TRY(optimizer_step(m));
  m->launches_last_step += m->ctx->counters.launches - before;
  return HL_OK;
}

namespace hl {
namespace {

constexpr int kTableLeft = 1, kTableRight = 2, kTableValue = 4, kTablesAll = 7;

// The rows the sparse policies work on, as one list for all memory blocks (a row chosen by several blocks or tokens
// is updated once; memory_sparse_adamw_updates, src/memory_transformer.rs:1293-1424), split into the half-key rows.
// Under data parallelism the list is the union over the ranks, formed by the exchange at the end of backward:
// every rank updates the rows any rank selected, with the averaged gradient (src/bin/heirloom/runtime.rs:4171-4214).
int gather_selection(hl_decoder* m, size_t* total_out) {
  hl_ctx* ctx = m->ctx;
  const size_t per_layer = (size_t)m->N * m->mem.top_k;
  size_t total = 0;
  if (nccl_active(ctx)) {
    HL_REQUIRE(m->union_n >= 0, "hl_decoder: sparse-row update requested, but no backward pass has run yet");
    HL_TRY(wait_for_collectives(m));
    total = (size_t)m->union_n;
    HL_CUDA(cudaMemcpyAsync(m->m_sel_all, m->m_union_rows, sizeof(int64_t) * total, cudaMemcpyDeviceToDevice, ctx->stream));
  } else {
    for (int l = 0; l < m->cfg.n_layers; ++l) {
      if (!m->lo[l].is_memory) continue;
      HL_CUDA(cudaMemcpyAsync(m->m_sel_all + total, m->ma[l].idx, sizeof(int64_t) * per_layer, cudaMemcpyDeviceToDevice,
                              ctx->stream));
      total += per_layer;
    }
  }
  if (total > 0) HL_TRY(hl_product_key_split_rows(ctx, m->m_sel_all, m->m_sel_left, m->m_sel_right, (long long)total, m->side));
  *total_out = total;
  return HL_OK;
}

struct SparseTable {
  size_t offset;
  const int64_t* rows;
  const unsigned char* mask;
  int n_rows, row_dim;
};

// SMFT: a table row is updated only where its mask allows (memory_sparse_adamw_updates_with_mask,
// src/memory_transformer.rs:1426-1468)
void sparse_tables(hl_decoder* m, int which, SparseTable out[3], int* count) {
  const int half = m->mem.key_dim / 2;
  int n = 0;
  if (which & kTableLeft) out[n++] = {m->off_kl, m->m_sel_left, m->smft_on ? m->smft_left_mask : nullptr, m->side, half};
  if (which & kTableRight) out[n++] = {m->off_kr, m->m_sel_right, m->smft_on ? m->smft_right_mask : nullptr, m->side, half};
  if (which & kTableValue)
    out[n++] = {m->off_val, m->m_sel_all, m->smft_on ? m->smft_value_mask : nullptr, m->mem.slots, m->mem.value_dim};
  *count = n;
}

// adds the sum of squares of the active rows of the chosen tables to *sum_dev (f64, on the device)
int sparse_sum_squares(hl_decoder* m, size_t total, int which, double* sum_dev) {
  SparseTable t[3];
  int n = 0;
  sparse_tables(m, which, t, &n);
  for (int i = 0; i < n; ++i)
    HL_TRY(hl_sparse_rows_sum_squares_f32(m->ctx, m->grads + t[i].offset, t[i].rows, (long long)total, t[i].mask,
                                          m->m_row_flags, t[i].n_rows, t[i].row_dim, sum_dev));
  return HL_OK;
}

int sparse_adamw(hl_decoder* m, size_t total, int which, const hl_adamw_params& hp) {
  SparseTable t[3];
  int n = 0;
  sparse_tables(m, which, t, &n);
  for (int i = 0; i < n; ++i)
    HL_TRY(hl_sparse_adamw_rows_f32(m->ctx, m->params + t[i].offset, m->grads + t[i].offset, m->m + t[i].offset,
                                    m->v + t[i].offset, t[i].rows, (long long)total, t[i].mask, m->m_row_flags, t[i].n_rows,
                                    t[i].row_dim, &hp, 0));
  return HL_OK;
}

hl_adamw_params step_params(hl_decoder* m, double clip) {
  hl_adamw_params hp{};
  hp.lr = m->opt.lr; hp.beta1 = m->opt.beta1; hp.beta2 = m->opt.beta2; hp.eps = m->opt.eps;
  hp.weight_decay = m->opt.weight_decay;
  hp.clip_scale = (float)clip * (1.0f / (float)nccl_world(m->ctx));  // summed gradients are averaged (src/nn.rs:2100-2117)
  hp.bias_correction1 = (float)(1.0 - pow((double)m->opt.beta1, (double)m->step));
  hp.bias_correction2 = (float)(1.0 - pow((double)m->opt.beta2, (double)m->step));
  return hp;
}

// clip factor from a sum of squares of summed (not yet averaged) gradients
int clip_from_sum(hl_decoder* m, double sum_sq, const char* what, double* clip) {
  *clip = 1.0;
  if (!(sum_sq >= 0.0) || sum_sq > 1e300) return fail(std::string("non-finite or negative ") + what + " sum-of-squares");
  const double norm = sqrt(sum_sq) / (double)nccl_world(m->ctx);  // norm of the averaged gradient
  if (norm > (double)m->opt.clip_norm) *clip = (double)m->opt.clip_norm / (norm + 1e-12);
  return HL_OK;
}

int step_sparse_rows(hl_decoder* m) {
  hl_ctx* ctx = m->ctx;
  size_t total = 0;
  HL_TRY(gather_selection(m, &total));
  if (total == 0) { m->step += 1; return HL_OK; }
  m->step += 1;  // every sparse call advances the step counter (src/nn.rs:2262)
  HL_CUDA(cudaMemsetAsync(m->m_row_flags, 0, (size_t)m->mem.slots, ctx->stream));
  double clip = 1.0;
  if (m->opt.clip_norm > 0.f) {
    // norm over the active rows of the three tables only (clip_scale_for_sparse_row_updates, src/nn.rs:2667-2774)
    HL_CUDA(cudaMemsetAsync(m->norm_dev64, 0, sizeof(double), ctx->stream));
    HL_TRY(sparse_sum_squares(m, total, kTablesAll, m->norm_dev64));
    double sum_sq = 0.0;
    HL_TRY(hl_memcpy_d2h(ctx, &sum_sq, m->norm_dev64, sizeof(double)));
    HL_TRY(clip_from_sum(m, sum_sq, "sparse selected gradient", &clip));
  }
  return sparse_adamw(m, total, kTablesAll, step_params(m, clip));
}

// `MemoryOnly` (src/bin/heirloom/runtime.rs:2440-2450; AdamW::step_parameter_indices_mut, src/nn.rs:2222-2254):
// dense AdamW on the memory tables alone, clip norm over those tables.
int step_memory_only(hl_decoder* m) {
  hl_ctx* ctx = m->ctx;
  HL_TRY(wait_for_collectives(m));
  const size_t begin = m->off_kl, n = m->tables_end - m->off_kl;
  double clip = 1.0;
  if (m->opt.clip_norm > 0.f) {
    HL_TRY(hl_sum_squares_f32(ctx, m->grads + begin, n, m->norm_dev));
    float sum = 0.f;
    HL_TRY(hl_memcpy_d2h(ctx, &sum, m->norm_dev, sizeof(float)));
    HL_TRY(clip_from_sum(m, (double)sum, "memory table gradient", &clip));
  }
  m->step += 1;
  const hl_adamw_params hp = step_params(m, clip);
  return adam_plan_step(ctx, m->plan_tables, &hp);
}

// Dense AdamW everywhere except the value table, row-set AdamW on the value rows the step selected: one step count,
// one clip factor from the dense gradients plus the active value rows.  The value table (slots x value_dim) is by
// far the largest parameter and only tokens*top_k of its rows carry a gradient, so this skips both the dense pass
// over it and the decay of rows nobody read.
int step_dense_plus_sparse_values(hl_decoder* m) {
  hl_ctx* ctx = m->ctx;
  size_t total = 0;
  HL_TRY(gather_selection(m, &total));  // waits for the collectives under data parallelism
  HL_CUDA(cudaMemsetAsync(m->m_row_flags, 0, (size_t)m->mem.slots, ctx->stream));
  double clip = 1.0;
  if (m->opt.clip_norm > 0.f) {
    const size_t tail = m->tables_end, tail_n = m->arena - m->tables_end;
    HL_TRY(hl_sum_squares_f32(ctx, m->grads, m->off_val, m->norm_dev));
    HL_TRY(hl_sum_squares_f32(ctx, m->grads + tail, tail_n, m->norm_dev + 1));
    HL_CUDA(cudaMemsetAsync(m->norm_dev64, 0, sizeof(double), ctx->stream));
    if (total > 0) HL_TRY(sparse_sum_squares(m, total, kTableValue, m->norm_dev64));
    float dense[2] = {0.f, 0.f};
    double rows = 0.0;
    HL_TRY(hl_memcpy_d2h(ctx, dense, m->norm_dev, sizeof(dense)));
    HL_TRY(hl_memcpy_d2h(ctx, &rows, m->norm_dev64, sizeof(double)));
    HL_TRY(clip_from_sum(m, (double)dense[0] + (double)dense[1] + rows, "gradient", &clip));
  }
  m->step += 1;
  const hl_adamw_params hp = step_params(m, clip);
  HL_TRY(adam_plan_step(ctx, m->plan_no_values, &hp));
  if (total > 0) HL_TRY(sparse_adamw(m, total, kTableValue, hp));
  return HL_OK;
}

}  // namespace
}  // namespace hl

int hl_decoder_optimizer_step_sparse_rows(hl_decoder* m) {
  return hl_decoder_optimizer_step_policy(m, HL_MEMORY_UPDATE_SPARSE_ROWS);
}

int hl_decoder_optimizer_step_policy(hl_decoder* m, int policy) {
  HL_REQUIRE(m, "hl_decoder_optimizer_step_policy: null model");
  if (policy == HL_MEMORY_UPDATE_FROZEN) return HL_OK;  // no optimizer step at all (runtime.rs:2421-2423)
  HL_REQUIRE(m->has_opt, "hl_decoder: no optimizer configured (call hl_decoder_set_optimizer)");
  if (policy == HL_MEMORY_UPDATE_FULL) return hl_decoder_optimizer_step(m);
  HL_REQUIRE(m->has_memory, "hl_decoder_optimizer_step_policy: the model has no memory layers");
  const unsigned long long before = m->ctx->counters.launches;
  m->cached = 0;
  int rc;
  switch (policy) {
    case HL_MEMORY_UPDATE_MEMORY_ONLY: rc = hl::step_memory_only(m); break;
    case HL_MEMORY_UPDATE_SPARSE_ROWS: rc = hl::step_sparse_rows(m); break;
    case HL_MEMORY_UPDATE_DENSE_PLUS_SPARSE_VALUES: rc = hl::step_dense_plus_sparse_values(m); break;
    default: return hl::fail("hl_decoder_optimizer_step_policy: unknown policy " + std::to_string(policy));
  }
  m->launches_last_step += m->ctx->counters.launches - before;
  return rc;
}

int hl_decoder_memory_access_counts(hl_decoder* m, unsigned long long* counts_dev) {
  HL_REQUIRE(m && counts_dev, "hl_decoder_memory_access_counts: null argument");
  HL_REQUIRE(m->has_memory, "hl_decoder_memory_access_counts: the model has no memory layers");
  const long long per_layer = (long long)m->N * m->mem.top_k;
  for (int l = 0; l < m->cfg.n_layers; ++l)
    if (m->lo[l].is_memory)
      HL_TRY(hl_memory_access_count_rows_i64_u64(m->ctx, m->ma[l].idx, per_layer, m->mem.slots, counts_dev));
  return HL_OK;
}

int hl_decoder_set_smft_masks(hl_decoder* m, const unsigned char* value_mask_host, const unsigned char* left_mask_host,
                              const unsigned char* right_mask_host) {
  HL_REQUIRE(m, "hl_decoder_set_smft_masks: null model");
  HL_REQUIRE(m->has_memory, "hl_decoder_set_smft_masks: the model has no memory layers");
  if (!value_mask_host && !left_mask_host && !right_mask_host) { m->smft_on = false; return HL_OK; }
  HL_REQUIRE(value_mask_host && left_mask_host && right_mask_host, "hl_decoder_set_smft_masks: give all three masks or none");
  hl_ctx* ctx = m->ctx;
  HL_CUDA(cudaMemcpyAsync(m->smft_value_mask, value_mask_host, (size_t)m->mem.slots, cudaMemcpyHostToDevice, ctx->stream));
  HL_CUDA(cudaMemcpyAsync(m->smft_left_mask, left_mask_host, (size_t)m->side, cudaMemcpyHostToDevice, ctx->stream));
  HL_CUDA(cudaMemcpyAsync(m->smft_right_mask, right_mask_host, (size_t)m->side, cudaMemcpyHostToDevice, ctx->stream));
  HL_CUDA(cudaStreamSynchronize(ctx->stream));  // the host buffers may be freed on return
  m->smft_on = true;
  return HL_OK;
}

int hl_decoder_train_step_device(hl_decoder* m, const int64_t* tokens_dev, const int64_t* targets_dev) {
  HL_TRY(hl_decoder_forward_backward(m, tokens_dev, targets_dev));
  return hl_decoder_optimizer_step(m);
}

int hl_decoder_train_step(hl_decoder* m, const int64_t* tokens_host, const int64_t* targets_host, float* loss_host) {
  HL_REQUIRE(m && tokens_host && targets_host, "hl_decoder_train_step: null argument");
  hl_ctx* ctx = m->ctx;
  HL_CUDA(cudaMemcpyAsync(m->tokens, tokens_host, sizeof(int64_t) * m->N, cudaMemcpyHostToDevice, ctx->stream));
  HL_CUDA(cudaMemcpyAsync(m->targets, targets_host, sizeof(int64_t) * m->N, cudaMemcpyHostToDevice, ctx->stream));
  ctx->counters.h2d_bytes += 2 * sizeof(int64_t) * (size_t)m->N;
  HL_TRY(hl_decoder_forward_backward(m, m->tokens, m->targets));
  HL_TRY(hl_decoder_optimizer_step(m));
  ctx->counters.d2h_bytes += sizeof(float);  // the loss kernel wrote it to pinned host memory as well
  HL_TRY(hl_ctx_sync(ctx));
  if (loss_host) *loss_host = m->loss_host[0];
  return HL_OK;
}

namespace {
// Runs the forward pass over `sequences` rows of `time` tokens (both at most what the model was
// created for), restoring the configured sizes afterwards.
struct ScopedShape {
  hl_decoder* m;
  int batch, context, n;
  ScopedShape(hl_decoder* model, int sequences, int time) : m(model), batch(model->cfg.batch), context(model->cfg.context), n(model->N) {
    m->cfg.batch = sequences;
    m->cfg.context = time;
    m->N = sequences * time;
  }
  ~ScopedShape() {
    m->cfg.batch = batch;
    m->cfg.context = context;
    m->N = n;
  }
};
}  // namespace

int hl_decoder_eval_loss(hl_decoder* m, const int64_t* tokens_dev, const int64_t* targets_dev, int sequences,
                         float* loss_host) {
  HL_REQUIRE(m && tokens_dev && targets_dev && loss_host, "hl_decoder_eval_loss: null argument");
  HL_REQUIRE(sequences > 0 && sequences <= m->cfg.batch,
             "hl_decoder_eval_loss: sequences must be between 1 and the batch the model was created for");
  const size_t n = (size_t)sequences * m->cfg.context;
  HL_CUDA(cudaMemcpyAsync(m->tokens, tokens_dev, sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, m->ctx->stream));
  HL_CUDA(cudaMemcpyAsync(m->targets, targets_dev, sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, m->ctx->stream));
  {
    ScopedShape shape(m, sequences, m->cfg.context);
    m->cached = 0;
    HL_TRY(run_graphed(m, GRAPH_LOSS, [m]() -> int {
      if (m->cfg.precision == HL_PRECISION_AMP_BF16) return forward(m, Forward::loss);
      HL_TRY(forward_f32(m));
      return cross_entropy_impl(m->ctx, m->logits, m->cfg.vocab, m->targets, m->N, m->cfg.vocab, 1.0f, m->loss_dev, nullptr,
                                nullptr, HL_BF16, m->cfg.vocab);
    }));
  }
  HL_CUDA(cudaMemcpyAsync(loss_host, m->loss_dev, sizeof(float), cudaMemcpyDeviceToHost, m->ctx->stream));
  m->ctx->counters.d2h_bytes += sizeof(float);
  return hl_ctx_sync(m->ctx);  // an id out of range or an expired wait: no loss
}

// The row of logits that a pass left in m->logits, or with `greedy` only the choice out of it, on its way to the host.
// A short row is written to pinned memory by the product itself, and so is the choice: no copy behind the last kernel.
constexpr int kDirectVocab = 4096;
struct RowTarget {
  hl_decoder* m;
  RowTarget(hl_decoder* model, bool greedy) : m(model) {
    m->row_logits = !greedy && m->cfg.vocab <= kDirectVocab ? m->logits_host : nullptr;
  }
  ~RowTarget() { m->row_logits = nullptr; }
};
static int queue_result(hl_decoder* m, bool greedy) {
  hl_ctx* ctx = m->ctx;
  if (greedy) return decode_greedy(ctx, m->logits, m->cfg.vocab, m->greedy, m->greedy_host);
  if (!m->row_logits)
    HL_CUDA(cudaMemcpyAsync(m->logits_host, m->logits, sizeof(float) * (size_t)m->cfg.vocab, cudaMemcpyDeviceToHost, ctx->stream));
  return HL_OK;
}
// With the status words: a pass that gave up or met an id out of range has no result, and the graphs that hold its launches have to
// be told (their launch numbers repeat, and a number that was not read stays behind).
static int finish_result(hl_decoder* m, bool greedy) {
  HL_TRY(hl_ctx_sync(m->ctx));
  m->ctx->counters.d2h_bytes += greedy ? sizeof(GreedyPart) : sizeof(float) * (size_t)m->cfg.vocab;
  return HL_OK;
}

static int run_window(hl_decoder* m, const int64_t* window, cudaMemcpyKind kind, int window_len, bool greedy) {
  HL_REQUIRE(window_len >= 1, "next_token_logits requires at least one token");
  HL_REQUIRE(window_len <= m->cfg.context, "hl_decoder_next_token_logits: the window is longer than the model's context");
  hl_ctx* ctx = m->ctx;
  HL_TRY(ensure_logits_host(m));
  const RowTarget target(m, greedy);
  HL_CUDA(cudaMemcpyAsync(m->tokens, window, sizeof(int64_t) * window_len, kind, ctx->stream));
  {
    ScopedShape shape(m, 1, window_len);
    m->cached = 0;
    m->decode_state_host[0] = window_len - 1;
    HL_TRY(run_graphed(m, target.m->row_logits ? GRAPH_WINDOW_TO_HOST : GRAPH_WINDOW, [m]() -> int {
      HL_CUDA(cudaMemcpyAsync(m->decode_state, m->decode_state_host, sizeof(long long), cudaMemcpyHostToDevice, m->ctx->stream));
      return m->cfg.precision == HL_PRECISION_AMP_BF16 ? forward(m, Forward::last_position) : forward_f32(m, true);
    }));
  }
  HL_TRY(queue_result(m, greedy));
  return finish_result(m, greedy);
}

static int window_logits(hl_decoder* m, const int64_t* window, cudaMemcpyKind kind, int window_len, float* logits_host) {
  HL_TRY(run_window(m, window, kind, window_len, false));
  memcpy(logits_host, m->logits_host, sizeof(float) * (size_t)m->cfg.vocab);
  return HL_OK;
}

int hl_decoder_next_token_logits(hl_decoder* m, const int64_t* window_dev, int window_len, float* logits_host) {
  HL_REQUIRE(m && window_dev && logits_host, "hl_decoder_next_token_logits: null argument");
  return window_logits(m, window_dev, cudaMemcpyDeviceToDevice, window_len, logits_host);
}

int hl_decoder_prefill(hl_decoder* m, const int64_t* window_host, int window_len, float* logits_host) {
  HL_REQUIRE(m && window_host && logits_host, "hl_decoder_prefill: null argument");
  HL_TRY(window_logits(m, window_host, cudaMemcpyHostToDevice, window_len, logits_host));
  m->cached = decode_applicable(m) ? window_len : 0;
  return HL_OK;
}

int hl_decoder_cached_positions(hl_decoder* m) { return m ? m->cached : 0; }

// One position behind the cached ones.
static int run_next(hl_decoder* m, int64_t token, bool greedy) {
  HL_REQUIRE(m->cached > 0, "hl_decoder_decode_next: no window is cached (call hl_decoder_prefill)");
  HL_REQUIRE(m->cached < m->cfg.context, "hl_decoder_decode_next: the context is full");
  HL_REQUIRE(token >= 0 && token < m->cfg.vocab, "hl_decoder_decode_next: token id out of range");
  hl_ctx* ctx = m->ctx;
  m->decode_state_host[0] = m->cached;
  m->decode_state_host[1] = token;
  const int position = m->cached;
  m->cached = 0;  // until this step has succeeded
  const RowTarget target(m, greedy);
  auto queue = [m, ctx, greedy]() -> int {
    HL_CUDA(cudaMemcpyAsync(m->decode_state, m->decode_state_host, 2 * sizeof(long long), cudaMemcpyHostToDevice, ctx->stream));
    {
      const int n = m->N;
      m->N = 1;
      const int rc = decode_step(m);
      m->N = n;
      HL_TRY(rc);
    }
    return queue_result(m, greedy);
  };
  HL_TRY(run_graphed(m, greedy ? GRAPH_DECODE_GREEDY : GRAPH_DECODE, queue));  // position and token are read from memory: the same sequence every time
  HL_TRY(finish_result(m, greedy));
  ctx->counters.h2d_bytes += 2 * sizeof(long long);
  m->cached = position + 1;
  return HL_OK;
}

int hl_decoder_decode_next(hl_decoder* m, int64_t token, float* logits_host) {
  HL_REQUIRE(m && logits_host, "hl_decoder_decode_next: null argument");
  HL_TRY(run_next(m, token, false));
  memcpy(logits_host, m->logits_host, sizeof(float) * (size_t)m->cfg.vocab);
  return HL_OK;
}

int hl_decoder_generate_token(hl_decoder* m, const int64_t* tokens, long long length, int appended, const hl_sampling_options* o,
                              double draw, int64_t* token, double* probability, double* log_probability) {
  HL_REQUIRE(m && tokens && o && token && probability && log_probability, "hl_decoder_generate_token: null argument");
  HL_REQUIRE(length >= 1, "next_token_logits requires at least one token");
  // without penalties and filters the choice at temperature 0 is the row's last maximum
  const bool greedy = o->temperature == 0.0 && o->top_k <= 0 && !(o->top_p > 0.0 && o->top_p < 1.0) &&
                      !(o->repetition_penalty > 1.0) && o->frequency_penalty == 0.0 && o->presence_penalty == 0.0;
  const int context = m->cfg.context;
  if (appended && length <= context && m->cached == length - 1) {
    HL_TRY(run_next(m, tokens[length - 1], greedy));
  } else {
    const int window = (int)std::min<long long>(length, context);
    HL_TRY(run_window(m, tokens + (length - window), cudaMemcpyHostToDevice, window, greedy));
    m->cached = decode_applicable(m) ? window : 0;
  }
  if (greedy) {
    const GreedyPart& g = *m->greedy_host;
    HL_REQUIRE(g.index >= 0, "non-finite generation logits");
    *token = g.index;
    *probability = 1.0 / g.sum;
    *log_probability = std::log(std::max(*probability, std::numeric_limits<double>::min()));
    return HL_OK;
  }
  HL_REQUIRE(all_finite_f32(m->logits_host, (size_t)m->cfg.vocab), "non-finite generation logits");
  return hl_sample_token(m->logits_host, HL_F32, m->cfg.vocab, tokens, length, o, draw, token, probability, log_probability);
}

int hl_decoder_loss(hl_decoder* m, float* loss_host) {
  HL_REQUIRE(m && loss_host, "hl_decoder_loss: null argument");
  return hl_memcpy_d2h(m->ctx, loss_host, m->loss_dev, sizeof(float));
}

unsigned long long hl_decoder_launches_last_step(hl_decoder* m) { return m ? m->launches_last_step : 0; }

int hl_decoder_comm_exposed_ms(hl_decoder* m, float* total_ms, int* waits) {
  HL_REQUIRE(m && total_ms, "hl_decoder_comm_exposed_ms: null argument");
  HL_CUDA(cudaStreamSynchronize(m->ctx->stream));
  float sum = 0.f;
  for (size_t i = 0; i < m->waits_recorded; ++i) {
    float ms = 0.f;
    HL_CUDA(cudaEventElapsedTime(&ms, m->wait_begin[i], m->wait_end[i]));
    sum += ms;
  }
  *total_ms = sum;
  if (waits) *waits = (int)m->waits_recorded;
  m->waits_recorded = 0;
  return HL_OK;
}

long long hl_ddp_bucket_count(long long arena_elems, long long bucket_elems) {
  if (arena_elems <= 0 || bucket_elems <= 0) return 0;
  return (arena_elems + bucket_elems - 1) / bucket_elems;
}

int hl_ddp_ready_buckets(long long arena_elems, long long bucket_elems, long long next_bucket, long long done_elems,
                         long long* starts, long long* counts, int capacity) {
  if (arena_elems <= 0 || bucket_elems <= 0 || next_bucket < 0 || !starts || !counts || capacity < 0) {
    hl::fail("hl_ddp_ready_buckets: invalid argument");
    return -1;
  }
  const long long total = hl_ddp_bucket_count(arena_elems, bucket_elems);
  int n = 0;
  for (long long b = next_bucket; b < total && n < capacity; ++b) {
    size_t start, end;
    hl::bucket_range((size_t)arena_elems, (size_t)bucket_elems, (size_t)b, &start, &end);
    if ((long long)end > done_elems) break;
    starts[n] = (long long)start;
    counts[n] = (long long)(end - start);
    ++n;
  }
  return n;
}

}  // extern "C"
