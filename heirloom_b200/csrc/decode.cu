// One-token steps, where decode_block.cu has no form for the sizes and in memory blocks: matrix-vector products and attention of
// one query row against the kept keys and values (the q/k/v rows that a full-window forward leaves in its activations).
//
// What bounds them: a step of the GPT-sized model reads 250 MB of bf16 weights (38 us at the copy rate) through some sixty
// dependent kernels, so it is bound by the latency of each: launch, input row, weights, reduction.  Hence a warp per output
// element with its weight loads in flight before the kernel waits for its predecessor (programmatic dependent launch), layer
// norms folded into the product that reads them (every CTA normalises the row again, which is cheaper than a kernel of its
// own), and a step that can be captured and replayed.
#include "decode.cuh"

namespace hl {
namespace {

constexpr int GV_WARPS = 8;
constexpr int GV_THREADS = GV_WARPS * 32;

struct GemvArgs {
  const void* x;        // [k]
  const float *gamma, *beta;  // layer norm of x first (null: none)
  const void* w;        // [n][k]
  const float* bias;    // [n]
  const void* residual; // [n], GV_RESIDUAL
  void* out;            // [n], row *out_row of it when out_row is given
  const long long* out_row;
  long long ld_out;
  int n, k;
  int epilogue;
  int warps_per_row;    // power of two; 1 with a layer norm
  bool vec;             // rows of w, and x, start on 16 bytes
};

// out = epilogue(W · x + bias).  WT/XT/OT: weights, input, output; Acc: float on the bf16 route, double where the f32
// route's sums are f64.  The values are rounded where the full-window kernels round them.  A lane holds the same 32 elements
// of x and of the weight row, so that a row needs no shared memory and a layer norm two warp sums; rows longer than 1024
// are shared by several warps.  Three CTAs an SM (two with f64 sums): with gamma and beta in registers there were two (one),
// and half of the loads that the memory wants in flight (50304 x 768: 30 -> 26 us; a step of the GPT-sized model 3.1 -> 2.8 ms
// for a prefix of 500 and 8 tokens).
template <typename WT, typename XT, typename OT, typename Acc>
__global__ void __launch_bounds__(GV_THREADS, sizeof(WT) == 2 ? 3 : 2)
decode_gemv_kernel(const GemvArgs a) {
  constexpr int PN = Pack<WT>::N, STEP = 32 * PN, U = GV_SPAN / STEP;
  __shared__ Acc parts[GV_WARPS];
  __shared__ __align__(16) float affine[2][GV_SPAN];  // gamma and beta, here before the input row is
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wpr = a.warps_per_row, part = warp % wpr, k = a.k;
  const int row_step = gridDim.x * (GV_WARPS / wpr);
  const int spans = (k + GV_SPAN * wpr - 1) / (GV_SPAN * wpr);  // how often the warps of a row move on
  const XT* x = static_cast<const XT*>(a.x);
  auto column = [&](int span, int u) { return (span * wpr + part) * GV_SPAN + u * STEP + lane * PN; };
  // Weights on their way: the next span of this row or of the warp's next one.
  uint4 raw[U];
  int row = blockIdx.x * (GV_WARPS / wpr) + warp / wpr;
  int fetch_row = row, fetch_span = 0;
  auto fetch = [&]() {
    if (fetch_row < a.n) {
      const WT* w = static_cast<const WT*>(a.w) + (size_t)fetch_row * k;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = column(fetch_span, u);
        raw[u] = c < k ? __ldg(reinterpret_cast<const uint4*>(w + c)) : make_uint4(0, 0, 0, 0);
      }
    }
    if (++fetch_span == spans) { fetch_span = 0; fetch_row += row_step; }
  };
  // weights and bias do not depend on any kernel of the step
  if (a.vec) fetch();
  if (a.gamma)
    for (int c = threadIdx.x * 4; c < k; c += GV_THREADS * 4) {
      cp_async16(&affine[0][c], a.gamma + c);
      cp_async16(&affine[1][c], a.beta + c);
    }
  float bias = a.bias && row < a.n ? __ldg(a.bias + row) : 0.f;
  pdl_trigger();
  pdl_wait();
  const OT* residual = static_cast<const OT*>(a.residual);
  float res = a.epilogue == GV_RESIDUAL && row < a.n ? as_f32(residual[row]) : 0.f;
  const long long out_row = a.out_row ? *a.out_row : 0;
  OT* out = static_cast<OT*>(a.out) + out_row * a.ld_out;
  float xv[U][PN];
  auto load_span = [&](int span) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = column(span, u);
      if (c < k) {
        load_x(x + c, xv[u]);
      } else {
#pragma unroll
        for (int e = 0; e < PN; ++e) xv[u][e] = 0.f;
      }
    }
  };
  if (a.vec) load_span(0);
  if (a.gamma) {  // one span, one warp per row
    cp_async_wait_all();
    __syncthreads();
    Acc sum = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int e = 0; e < PN; ++e) sum += (Acc)xv[u][e];
    }
    const Acc mean = warp_sum(sum) / (Acc)k;
    Acc sq = 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (column(0, u) < k) {
#pragma unroll
        for (int e = 0; e < PN; ++e) { const Acc d = (Acc)xv[u][e] - mean; sq += d * d; }
      }
    const Acc rstd = (Acc)1 / sqrt(warp_sum(sq) / (Acc)k + (Acc)1e-5f);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (const int c = column(0, u); c < k) {
        float g[PN], b[PN];
        load_x(&affine[0][c], g);
        load_x(&affine[1][c], b);
#pragma unroll
        for (int e = 0; e < PN; ++e) {
          const float y = (float)(((Acc)xv[u][e] - mean) * rstd * (Acc)g[e] + (Acc)b[e]);
          xv[u][e] = sizeof(XT) == 2 ? bf16_round(y) : y;
        }
      }
  }
  for (int base = blockIdx.x * (GV_WARPS / wpr); base < a.n; base += row_step, row += row_step) {
    Acc acc = 0;
    if (row >= a.n) {
    } else if (a.vec) {
      for (int span = 0; span < spans; ++span) {
        uint4 now[U];
#pragma unroll
        for (int u = 0; u < U; ++u) now[u] = raw[u];
        fetch();  // travels while these are multiplied
        if (spans > 1) load_span(span);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float v[PN];
          Pack<WT>::unpack(now[u], v);
#pragma unroll
          for (int e = 0; e < PN; ++e) acc += (Acc)v[e] * (Acc)xv[u][e];
        }
      }
    } else {
      const WT* w = static_cast<const WT*>(a.w) + (size_t)row * k;
      for (int c = part * 32 + lane; c < k; c += 32 * wpr) acc += (Acc)as_f32(w[c]) * (Acc)as_f32(x[c]);
    }
    acc = warp_sum(acc);
    if (wpr > 1) {
      if (lane == 0) parts[warp] = acc;
      __syncthreads();
      if (part == 0)
        for (int i = 1; i < wpr; ++i) acc += parts[warp + i];
    }
    if (lane == 0 && part == 0 && row < a.n) {
      // f32 rows round the product before the bias is added, the tensor-core route adds it to the accumulator
      float y = (float)acc;
      if (a.bias) y = y + bias;
      if (a.epilogue == GV_GELU) {
        y = sizeof(OT) == 2 ? gelu_fwd_fast(bf16_round(y)) : (float)gelu_fwd<double>((double)y);
      } else if (a.epilogue == GV_RESIDUAL) {
        y = sizeof(OT) == 2 ? res + bf16_round(y) : res + y;
      }
      if constexpr (sizeof(OT) == 2) out[row] = to_bf16(y); else out[row] = y;
    }
    if (row + row_step < a.n) {
      if (a.bias) bias = __ldg(a.bias + row + row_step);
      if (a.epilogue == GV_RESIDUAL) res = as_f32(residual[row + row_step]);
    }
    if (wpr > 1) __syncthreads();
  }
}

// Row *pos of the q/k/v rows against rows 0 .. *pos: a cluster of eight CTAs per head, each over an eighth of the keys; their
// maxima, sums and weighted values are pushed into CTA 0's shared memory.  Eight lanes take a key, sixteen bytes each.
//
// Bound by latency: a few hundred bytes of keys a thread behind a chain of dependent steps.  Only the newest row comes from the
// kernel before this one, so the older keys and values are on their way into shared memory (`staged`, where they fit) while
// that one still runs, and the chain that is left starts at the query (12 heads of 64 at 500 positions: 9.8 us before).
constexpr int DA_CTAS = 8;
constexpr int DA_THREADS = 128;
constexpr int DA_SLOTS = DA_THREADS / 8;  // keys at a time
template <typename T, typename Acc>
__global__ void __launch_bounds__(DA_THREADS)
decode_attention_kernel(const T* __restrict__ qkv, long long ld, int channels, const long long* __restrict__ pos,
                        T* __restrict__ out, int hd, int chunk_cap, bool staged, bool settled) {
  extern __shared__ double da_smem[];
  T* kept = reinterpret_cast<T*>(da_smem);   // staged: [2][chunk_cap][hd] keys, then values
  Acc* q = reinterpret_cast<Acc*>(kept + (staged ? (size_t)2 * chunk_cap * hd : 0));  // [hd]
  Acc* s = q + hd;                           // [chunk_cap] scores, then weights
  Acc* part = s + chunk_cap;                 // [DA_SLOTS][hd] weighted values per key slot
  Acc* all = part + DA_SLOTS * hd;           // CTA 0: [DA_CTAS][hd + 2] weighted values, maximum, sum of every CTA
  __shared__ Acc red[32], slot_sums[DA_SLOTS];
  cg::cluster_group cluster = cg::this_cluster();
  pdl_trigger();
  const int rank = (int)(blockIdx.x % DA_CTAS), h = (int)(blockIdx.x / DA_CTAS);
  const T* base = qkv + (long long)h * hd;
  const int sub = threadIdx.x & 7, slot = threadIdx.x >> 3;
  constexpr int PN = Pack<T>::N;
  const bool vec = hd % PN == 0 && channels % PN == 0 && ld % PN == 0;
  // The position was copied here before the first kernel of the sequence started.
  const long long t = *pos;
  const int keys = (int)t + 1, chunk = (keys + DA_CTAS - 1) / DA_CTAS;
  const int k0 = min(keys, rank * chunk), k1 = min(keys, k0 + chunk);
  const int units = hd / PN;  // 16-byte pieces of a row
  auto stage = [&](int key, int u) {
#pragma unroll
    for (int kv = 0; kv < 2; ++kv)
      cp_async16(kept + ((size_t)kv * chunk_cap + (key - k0)) * hd + u * PN, base + (1 + kv) * channels + (long long)key * ld + u * PN);
  };
  if (!settled) pdl_wait();  // the rows below the position come from the predecessor as well
  if (staged)
    for (int key = k0 + slot; key < min(k1, (int)t); key += DA_SLOTS)
      for (int u = sub; u < units; u += 8) stage(key, u);
  cluster.sync();  // CTA 0 has started: its shared memory may be written
  pdl_wait();
  if (staged) {
    if (k1 == keys && k1 > k0 && (int)threadIdx.x < units) stage((int)t, threadIdx.x);
  }
  for (int c = threadIdx.x; c < hd; c += DA_THREADS) q[c] = (Acc)as_f32(base[t * ld + c]);
  if (staged) cp_async_wait_all();
  __syncthreads();
  const Acc scale = (Acc)1 / sqrt((Acc)hd);
  Acc mx = -INFINITY;
#pragma unroll 4
  for (int key = k0 + slot; key - slot < k1; key += DA_SLOTS) {
    Acc dot = 0;
    if (key < k1) {
      const T* kr = staged ? kept + (size_t)(key - k0) * hd : base + channels + (long long)key * ld;
      if (vec) {
        for (int c = sub * PN; c < hd; c += 8 * PN) {
          float kv[PN];
          Pack<T>::unpack(*reinterpret_cast<const uint4*>(kr + c), kv);
#pragma unroll
          for (int e = 0; e < PN; ++e) dot += q[c + e] * (Acc)kv[e];
        }
      } else {
        for (int c = sub; c < hd; c += 8) dot += q[c] * (Acc)as_f32(kr[c]);
      }
    }
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    dot += __shfl_xor_sync(0xffffffffu, dot, 4);
    if (key < k1) {
      dot *= scale;
      if (sub == 0) s[key - k0] = dot;
      mx = max(mx, dot);
    }
  }
  mx = block_max(mx, red, (Acc)-INFINITY);
  Acc weights = 0;  // sum over this slot's keys
  // every lane of a key takes the exponential again: cheaper than a pass and a barrier of their own
  if (vec) {
    for (int c = sub * PN; c < hd; c += 8 * PN) {
      Acc acc[PN];
#pragma unroll
      for (int e = 0; e < PN; ++e) acc[e] = 0;
      weights = 0;
#pragma unroll 4
      for (int key = k0 + slot; key < k1; key += DA_SLOTS) {
        float vv[PN];
        const T* vr = staged ? kept + ((size_t)chunk_cap + (key - k0)) * hd : base + 2 * channels + (long long)key * ld;
        Pack<T>::unpack(*reinterpret_cast<const uint4*>(vr + c), vv);
        const Acc w = exp(s[key - k0] - mx);
        weights += w;
#pragma unroll
        for (int e = 0; e < PN; ++e) acc[e] += w * (Acc)vv[e];
      }
#pragma unroll
      for (int e = 0; e < PN; ++e) part[slot * hd + c + e] = acc[e];
    }
  } else {
    for (int c = sub; c < hd; c += 8) {
      Acc acc = 0;
      weights = 0;
      for (int key = k0 + slot; key < k1; key += DA_SLOTS) {
        const Acc w = exp(s[key - k0] - mx);
        weights += w;
        acc += w * (Acc)as_f32(base[2 * channels + (long long)key * ld + c]);
      }
      part[slot * hd + c] = acc;
    }
  }
  if (sub == 0) slot_sums[slot] = weights;
  __syncthreads();
  Acc* mine = cluster.map_shared_rank(all, 0) + rank * (hd + 2);
  for (int c = threadIdx.x; c < hd; c += DA_THREADS) {
    Acc v = 0;
#pragma unroll
    for (int i = 0; i < DA_SLOTS; ++i) v += part[i * hd + c];
    mine[c] = v;
  }
  if (threadIdx.x == 0) {
    Acc sum = 0;
#pragma unroll
    for (int i = 0; i < DA_SLOTS; ++i) sum += slot_sums[i];
    mine[hd] = mx;
    mine[hd + 1] = sum;
  }
  cluster.sync();
  if (rank != 0) return;
  Acc m = -INFINITY, l = 0, f[DA_CTAS];
#pragma unroll
  for (int r = 0; r < DA_CTAS; ++r) m = max(m, all[r * (hd + 2) + hd]);
#pragma unroll
  for (int r = 0; r < DA_CTAS; ++r) {
    const Acc mr = all[r * (hd + 2) + hd];
    f[r] = mr == (Acc)-INFINITY ? (Acc)0 : exp(mr - m);
    l += f[r] * all[r * (hd + 2) + hd + 1];
  }
  for (int c = threadIdx.x; c < hd; c += DA_THREADS) {
    Acc v = 0;
#pragma unroll
    for (int r = 0; r < DA_CTAS; ++r) v += f[r] * all[r * (hd + 2) + c];
    const float y = (float)(v / l);
    if constexpr (sizeof(T) == 2) out[h * hd + c] = to_bf16(y); else out[h * hd + c] = y;
  }
}

// The embedding row of the state's token at the state's position.
template <typename T>
__global__ void decode_embed_kernel(const float* __restrict__ table, const float* __restrict__ positions,
                                    const long long* __restrict__ state /* position, token */, T* __restrict__ out, int dim) {
  pdl_trigger();
  pdl_wait();
  const float* a = table + state[1] * dim;
  const float* b = positions + state[0] * dim;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < dim; c += gridDim.x * blockDim.x) {
    if constexpr (sizeof(T) == 2) out[c] = to_bf16(bf16_round(a[c]) + bf16_round(b[c]));
    else out[c] = a[c] + b[c];
  }
}

// Greedy choice.  A block takes 2048 logits, eight a thread; the block that finishes last adds the blocks' sums in their order.
// Replaces 200 KB to the host and 145 us of sampling there (50304 logits) by 16 bytes and 6 us.
__device__ __forceinline__ void greedy_better(float& m, int& i, float m2, int i2) {
  if (m2 > m || (m2 == m && i2 > i)) { m = m2; i = i2; }
}
__global__ void __launch_bounds__(256)
decode_greedy_kernel(const float* __restrict__ logits, int vocab, GreedyPart* __restrict__ parts, GreedyPart* __restrict__ out,
                     unsigned* __restrict__ ticket) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sm_max[8];
  __shared__ int sm_index[8], sm_bad;
  __shared__ double sm_sum[8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sm_bad = 0;
  __syncthreads();
  float v[8], m = -INFINITY;
  int index = -1;
  bool bad = false;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int i = blockIdx.x * 2048 + u * 256 + threadIdx.x;
    v[u] = i < vocab ? logits[i] : -INFINITY;
    if (i < vocab) {
      bad |= !isfinite(v[u]);
      greedy_better(m, index, v[u], i);
    }
  }
  if (bad) sm_bad = 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) greedy_better(m, index, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, index, o));
  if (lane == 0) { sm_max[warp] = m; sm_index[warp] = index; }
  __syncthreads();
  m = sm_max[0];
  index = sm_index[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) greedy_better(m, index, sm_max[w], sm_index[w]);
  double s = 0.0;
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (v[u] > -INFINITY) s += exp((double)v[u] - (double)m);
  s = warp_sum(s);
  if (lane == 0) sm_sum[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    s = 0.0;
    for (int w = 0; w < 8; ++w) s += sm_sum[w];
    parts[blockIdx.x] = GreedyPart{s, m, sm_bad ? -1 : index};
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || warp != 0) return;
  __threadfence();
  m = -INFINITY;
  index = -1;
  bad = false;
  for (int b = lane; b < (int)gridDim.x; b += 32) {
    const float pm = __ldcg(&parts[b].max);
    const int pi = __ldcg(&parts[b].index);
    bad |= pi < 0;
    greedy_better(m, index, pm, pi);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) greedy_better(m, index, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, index, o));
  bad = __any_sync(0xffffffffu, bad);
  s = 0.0;
  for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(&parts[b].sum) * exp((double)__ldcg(&parts[b].max) - (double)m);
  s = warp_sum(s);
  if (lane == 0) {
    *out = GreedyPart{s, m, bad ? -1 : index};
    *ticket = 0u;
  }
}

template <typename WT, typename XT, typename OT, typename Acc>
int launch_gemv(hl_ctx* ctx, const GemvArgs& a) {
  // every output its own warp (or its share of one) up to eight CTAs per SM; the vocabulary's rows are walked by those
  const int grid = std::min(ceil_div(a.n, GV_WARPS / a.warps_per_row), ctx->sm_count * 8);
  HL_CUDA(launch_pdl(decode_gemv_kernel<WT, XT, OT, Acc>, grid, GV_THREADS, 0, ctx->stream, 1, a));
  count_launch(ctx);
  return HL_OK;
}

}  // namespace

int decode_gemv(hl_ctx* ctx, const DecodeGemv& g) {
  GemvArgs a{g.x, g.gamma, g.beta, g.w, g.bias, g.residual, g.out, g.out_row, g.ld_out, g.n, g.k, g.epilogue, 1, false};
  const int per16 = g.w_dtype == HL_BF16 ? 8 : 4;
  a.vec = g.k % per16 == 0 && ((reinterpret_cast<uintptr_t>(g.w) | reinterpret_cast<uintptr_t>(g.x)) & 15) == 0;
  HL_REQUIRE(!g.gamma || (a.vec && g.k <= GV_SPAN && (reinterpret_cast<uintptr_t>(g.gamma) & 15) == 0 &&
                          (reinterpret_cast<uintptr_t>(g.beta) & 15) == 0),
             "decode_gemv: a layer norm takes rows of up to 1024 elements on 16-byte boundaries");
  while (a.warps_per_row < GV_WARPS && a.warps_per_row * GV_SPAN < g.k) a.warps_per_row *= 2;
  if (g.w_dtype == HL_BF16)
    return g.out_dtype == HL_BF16 ? launch_gemv<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16, float>(ctx, a)
                                  : launch_gemv<__nv_bfloat16, __nv_bfloat16, float, float>(ctx, a);
  if (g.x_dtype == HL_BF16) return launch_gemv<float, __nv_bfloat16, float, double>(ctx, a);
  return g.out_dtype == HL_BF16 ? launch_gemv<float, float, __nv_bfloat16, double>(ctx, a)
                                : launch_gemv<float, float, float, double>(ctx, a);
}

size_t decode_attention_smem(int dtype, int hd, int context) {
  const size_t acc = dtype == HL_BF16 ? 4 : 8;
  return acc * ((size_t)hd + (size_t)ceil_div(context, DA_CTAS) + (size_t)DA_SLOTS * hd + (size_t)DA_CTAS * (hd + 2));
}

template <typename T, typename Acc>
int launch_decode_attention(hl_ctx* ctx, const T* qkv, long long ld, const long long* pos, T* out, int channels, int n_heads, int context,
                            bool settled) {
  const int hd = channels / n_heads, cap = ceil_div(context, DA_CTAS);
  size_t smem = decode_attention_smem(sizeof(T) == 2 ? HL_BF16 : HL_F32, hd, context);
  const size_t rows = sizeof(T) * 2 * (size_t)cap * hd;
  // staged while two CTAs still fit on an SM; longer contexts read keys and values where they lie
  const bool staged = smem + rows <= 110 * 1024 && hd % Pack<T>::N == 0 && channels % Pack<T>::N == 0 && ld % Pack<T>::N == 0 &&
                      (reinterpret_cast<uintptr_t>(qkv) & 15) == 0;
  if (staged) smem += rows;
  auto kern = decode_attention_kernel<T, Acc>;
  HL_ALLOW_SHARED(ctx, 110 * 1024, kern);
  HL_CUDA(launch_pdl(kern, n_heads * DA_CTAS, DA_THREADS, smem, ctx->stream, DA_CTAS, qkv, ld, channels, pos, out, hd, cap, staged,
                     settled));
  count_launch(ctx);
  return HL_OK;
}

int decode_attention(hl_ctx* ctx, const void* qkv, int dtype, long long ld, const long long* pos, void* out, int channels,
                     int n_heads, int context, bool settled) {
  return dtype == HL_BF16 ? launch_decode_attention<__nv_bfloat16, float>(ctx, (const __nv_bfloat16*)qkv, ld, pos, (__nv_bfloat16*)out,
                                                                          channels, n_heads, context, settled)
                          : launch_decode_attention<float, double>(ctx, (const float*)qkv, ld, pos, (float*)out, channels, n_heads, context, settled);
}

int decode_greedy(hl_ctx* ctx, const float* logits, int vocab, GreedyPart* parts, GreedyPart* out) {
  HL_CUDA(launch_pdl(decode_greedy_kernel, greedy_parts(vocab), 256, 0, ctx->stream, 1, logits, vocab, parts, out,
                     ctx->gemm_sched + 9));  // a word of the context's zeroed counters
  count_launch(ctx);
  return HL_OK;
}

int decode_embed(hl_ctx* ctx, const float* table, const float* positions, const long long* state, void* out, int dtype, int dim) {
  const int grid = ceil_div(dim, 256);
  if (dtype == HL_BF16)
    HL_CUDA(launch_pdl(decode_embed_kernel<__nv_bfloat16>, grid, 256, 0, ctx->stream, 1, table, positions, state, (__nv_bfloat16*)out, dim));
  else
    HL_CUDA(launch_pdl(decode_embed_kernel<float>, grid, 256, 0, ctx->stream, 1, table, positions, state, (float*)out, dim));
  count_launch(ctx);
  return HL_OK;
}

}  // namespace hl
