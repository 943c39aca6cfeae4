// One-token steps of a decoder whose window is already in the activation buffers: matrix-vector products and attention of
// one query row against the kept keys and values (the q/k/v rows that a full-window forward leaves in its activations).
//
// What bounds them: a step of the GPT-sized model reads 250 MB of bf16 weights (38 us at the copy rate) through some sixty
// dependent kernels, so it is bound by the latency of each: launch, input row, weights, reduction.  Hence a warp per output
// element with all of its weight loads in flight at once, layer norms folded into the product that reads them (every CTA
// normalises the row again, which is cheaper than a kernel of its own), and a step that can be captured and replayed.
#include <cooperative_groups.h>

#include "kernels.h"

namespace hl {
namespace {

namespace cg = cooperative_groups;

constexpr int GV_WARPS = 8;
constexpr int GV_THREADS = GV_WARPS * 32;

template <typename T> __device__ __forceinline__ float as_f32(T x);
template <> __device__ __forceinline__ float as_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float as_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> struct Pack;  // sixteen bytes of weights
template <> struct Pack<float> {
  static constexpr int N = 4;
  __device__ static void unpack(const uint4& u, float (&v)[4]) {
    v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
  }
};
template <> struct Pack<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void unpack(const uint4& u, float (&v)[8]) {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
};

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
  bool vec;             // rows of w start on 16 bytes
};

// out = epilogue(W · x + bias).  WT/XT/OT: weights, input, output; Acc: float on the bf16 route, double where the f32
// route's sums are f64.  The values are rounded where the full-window kernels round them.
template <typename WT, typename XT, typename OT, typename Acc>
__global__ void __launch_bounds__(GV_THREADS)
decode_gemv_kernel(const GemvArgs a) {
  extern __shared__ float gv_x[];  // the input row, normalised and rounded to the type it is stored in
  __shared__ Acc red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const XT* x = static_cast<const XT*>(a.x);
  const int k = a.k;
  if (a.gamma) {
    Acc sum = 0;
    for (int c = threadIdx.x; c < k; c += GV_THREADS) {
      const float v = as_f32(x[c]);
      gv_x[c] = v;
      sum += (Acc)v;
    }
    const Acc mean = block_sum(sum, red) / (Acc)k;
    Acc sq = 0;
    for (int c = threadIdx.x; c < k; c += GV_THREADS) { const Acc d = (Acc)gv_x[c] - mean; sq += d * d; }
    const Acc rstd = (Acc)1 / sqrt(block_sum(sq, red) / (Acc)k + (Acc)1e-5f);
    for (int c = threadIdx.x; c < k; c += GV_THREADS) {
      const float y = (float)(((Acc)gv_x[c] - mean) * rstd * (Acc)a.gamma[c] + (Acc)a.beta[c]);
      gv_x[c] = sizeof(XT) == 2 ? bf16_round(y) : y;
    }
  } else {
    for (int c = threadIdx.x; c < k; c += GV_THREADS) gv_x[c] = as_f32(x[c]);
  }
  __syncthreads();
  constexpr int PN = Pack<WT>::N, STEP = 32 * PN, U = 4;
  OT* out = static_cast<OT*>(a.out) + (a.out_row ? *a.out_row * a.ld_out : 0);
  for (int row = blockIdx.x * GV_WARPS + warp; row < a.n; row += gridDim.x * GV_WARPS) {
    const WT* w = static_cast<const WT*>(a.w) + (size_t)row * k;
    Acc acc = 0;
    if (a.vec) {
      for (int c0 = lane * PN; c0 < k; c0 += U * STEP) {
        uint4 raw[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          raw[u] = c0 + u * STEP < k ? __ldg(reinterpret_cast<const uint4*>(w + c0 + u * STEP)) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + u * STEP;
          if (c < k) {
            float v[PN];
            Pack<WT>::unpack(raw[u], v);
#pragma unroll
            for (int e = 0; e < PN; ++e) acc += (Acc)v[e] * (Acc)gv_x[c + e];
          }
        }
      }
    } else {
      for (int c = lane; c < k; c += 32) acc += (Acc)as_f32(w[c]) * (Acc)gv_x[c];
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      // f32 rows round the product before the bias is added, the tensor-core route adds it to the accumulator
      float y = (float)acc;
      if (a.bias) y = y + a.bias[row];
      if (a.epilogue == GV_GELU) {
        y = sizeof(OT) == 2 ? gelu_fwd_fast(bf16_round(y)) : (float)gelu_fwd<double>((double)y);
      } else if (a.epilogue == GV_RESIDUAL) {
        const float r = as_f32(static_cast<const OT*>(a.residual)[row]);
        y = sizeof(OT) == 2 ? r + bf16_round(y) : r + y;
      }
      if constexpr (sizeof(OT) == 2) out[row] = to_bf16(y); else out[row] = y;
    }
  }
}

// Row *pos of the q/k/v rows against rows 0 .. *pos: a cluster of eight CTAs per head, each over an eighth of the keys; the
// partial maxima, sums and weighted values meet in CTA 0 through distributed shared memory.
constexpr int DA_CTAS = 8;
constexpr int DA_THREADS = 128;
template <typename T, typename Acc>
__global__ void __launch_bounds__(DA_THREADS)
decode_attention_kernel(const T* __restrict__ qkv, long long ld, int channels, const long long* __restrict__ pos,
                        T* __restrict__ out, int hd, int chunk_cap) {
  extern __shared__ double da_smem[];
  Acc* q = reinterpret_cast<Acc*>(da_smem);  // [hd]
  Acc* s = q + hd;                           // [chunk_cap] scores, then weights
  Acc* o = s + chunk_cap;                    // [hd] weighted values of this CTA
  Acc* part = o + hd;                        // [DA_THREADS] sums of the thread groups over their keys
  __shared__ Acc stat[2];                    // maximum, sum
  __shared__ Acc red[32];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)(blockIdx.x % DA_CTAS), h = (int)(blockIdx.x / DA_CTAS);
  const long long t = *pos;
  const int keys = (int)t + 1, chunk = (keys + DA_CTAS - 1) / DA_CTAS;
  const int k0 = min(keys, rank * chunk), k1 = min(keys, k0 + chunk);
  const T* base = qkv + (long long)h * hd;
  const Acc scale = (Acc)1 / sqrt((Acc)hd);
  for (int c = threadIdx.x; c < hd; c += DA_THREADS) { q[c] = (Acc)as_f32(base[t * ld + c]); o[c] = 0; }
  __syncthreads();
  // eight lanes per key
  const int sub = threadIdx.x & 7, who = threadIdx.x >> 3;
  Acc mx = -INFINITY;
  for (int key = k0 + who; key - who < k1; key += DA_THREADS / 8) {
    Acc dot = 0;
    if (key < k1) {
      const T* kr = base + channels + (long long)key * ld;
      for (int c = sub; c < hd; c += 8) dot += q[c] * (Acc)as_f32(kr[c]);
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
  Acc sum = 0;
  for (int i = threadIdx.x; i < k1 - k0; i += DA_THREADS) {
    const Acc e = exp(s[i] - mx);
    s[i] = e;
    sum += e;
  }
  sum = block_sum(sum, red);
  __syncthreads();
  // channels across the threads; heads narrower than the block split the keys over groups of threads
  const int groups = max(1, DA_THREADS / hd);
  for (int c0 = 0; c0 < hd; c0 += DA_THREADS) {
    const int c = c0 + (groups > 1 ? (int)threadIdx.x % hd : (int)threadIdx.x), g = groups > 1 ? (int)threadIdx.x / hd : 0;
    Acc acc = 0;
    if (c < hd && g < groups) {
      const T* vr = base + 2 * channels + c;
#pragma unroll 4
      for (int key = k0 + g; key < k1; key += groups) acc += s[key - k0] * (Acc)as_f32(vr[(long long)key * ld]);
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    if (c < hd && g == 0) {
      for (int i = 1; i < groups; ++i) acc += part[threadIdx.x + i * hd];
      o[c] = acc;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { stat[0] = mx; stat[1] = sum; }
  cluster.sync();
  if (rank == 0) {
    Acc m = -INFINITY, l = 0;
    for (int r = 0; r < DA_CTAS; ++r) m = max(m, *cluster.map_shared_rank(&stat[0], r));
    Acc f[DA_CTAS];
    for (int r = 0; r < DA_CTAS; ++r) {
      const Acc mr = *cluster.map_shared_rank(&stat[0], r);
      f[r] = mr == (Acc)-INFINITY ? (Acc)0 : exp(mr - m);
      l += f[r] * *cluster.map_shared_rank(&stat[1], r);
    }
    for (int c = threadIdx.x; c < hd; c += DA_THREADS) {
      Acc v = 0;
      for (int r = 0; r < DA_CTAS; ++r) v += f[r] * *cluster.map_shared_rank(o + c, r);
      const float y = (float)(v / l);
      if constexpr (sizeof(T) == 2) out[h * hd + c] = to_bf16(y); else out[h * hd + c] = y;
    }
  }
  cluster.sync();  // no CTA leaves while CTA 0 reads its shared memory
}

// The embedding row of the state's token at the state's position.
template <typename T>
__global__ void decode_embed_kernel(const float* __restrict__ table, const float* __restrict__ positions,
                                    const long long* __restrict__ state /* position, token */, T* __restrict__ out, int dim) {
  const float* a = table + state[1] * dim;
  const float* b = positions + state[0] * dim;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < dim; c += gridDim.x * blockDim.x) {
    if constexpr (sizeof(T) == 2) out[c] = to_bf16(bf16_round(a[c]) + bf16_round(b[c]));
    else out[c] = a[c] + b[c];
  }
}

template <typename WT, typename XT, typename OT, typename Acc>
int launch_gemv(hl_ctx* ctx, const GemvArgs& a) {
  const size_t smem = sizeof(float) * (size_t)a.k;
  auto kern = decode_gemv_kernel<WT, XT, OT, Acc>;
  static bool configured = false;
  if (!configured) {
    HL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDecodeMaxRow * (int)sizeof(float)));
    configured = true;
  }
  // every output its own warp up to eight CTAs per SM; the vocabulary's rows are walked by those
  const int grid = std::min(ceil_div(a.n, GV_WARPS), ctx->sm_count * 8);
  kern<<<grid, GV_THREADS, smem, ctx->stream>>>(a);
  HL_LAUNCH_CHECK("decode_gemv_kernel");
  count_launch(ctx);
  return HL_OK;
}

}  // namespace

int decode_gemv(hl_ctx* ctx, const DecodeGemv& g) {
  HL_REQUIRE(g.k <= kDecodeMaxRow, "decode_gemv: input row too long");
  GemvArgs a{g.x, g.gamma, g.beta, g.w, g.bias, g.residual, g.out, g.out_row, g.ld_out, g.n, g.k, g.epilogue, false};
  const int per16 = g.w_dtype == HL_BF16 ? 8 : 4;
  a.vec = g.k % per16 == 0 && (reinterpret_cast<uintptr_t>(g.w) & 15) == 0;
  if (g.w_dtype == HL_BF16)
    return g.out_dtype == HL_BF16 ? launch_gemv<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16, float>(ctx, a)
                                  : launch_gemv<__nv_bfloat16, __nv_bfloat16, float, float>(ctx, a);
  if (g.x_dtype == HL_BF16) return launch_gemv<float, __nv_bfloat16, float, double>(ctx, a);
  return g.out_dtype == HL_BF16 ? launch_gemv<float, float, __nv_bfloat16, double>(ctx, a)
                                : launch_gemv<float, float, float, double>(ctx, a);
}

size_t decode_attention_smem(int dtype, int hd, int context) {
  const size_t acc = dtype == HL_BF16 ? 4 : 8;
  return acc * (2 * (size_t)hd + (size_t)ceil_div(context, DA_CTAS) + DA_THREADS);
}

int decode_attention(hl_ctx* ctx, const void* qkv, int dtype, long long ld, const long long* pos, void* out, int channels,
                     int n_heads, int context) {
  const int hd = channels / n_heads, cap = ceil_div(context, DA_CTAS);
  const size_t smem = decode_attention_smem(dtype, hd, context);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n_heads * DA_CTAS));
  cfg.blockDim = dim3(DA_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = DA_CTAS; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (dtype == HL_BF16)
    HL_CUDA(cudaLaunchKernelEx(&cfg, decode_attention_kernel<__nv_bfloat16, float>, (const __nv_bfloat16*)qkv, ld, channels, pos,
                               (__nv_bfloat16*)out, hd, cap));
  else
    HL_CUDA(cudaLaunchKernelEx(&cfg, decode_attention_kernel<float, double>, (const float*)qkv, ld, channels, pos, (float*)out, hd,
                               cap));
  HL_LAUNCH_CHECK("decode_attention_kernel");
  count_launch(ctx);
  return HL_OK;
}

int decode_embed(hl_ctx* ctx, const float* table, const float* positions, const long long* state, void* out, int dtype, int dim) {
  const int grid = ceil_div(dim, 256);
  if (dtype == HL_BF16) decode_embed_kernel<<<grid, 256, 0, ctx->stream>>>(table, positions, state, (__nv_bfloat16*)out, dim);
  else decode_embed_kernel<<<grid, 256, 0, ctx->stream>>>(table, positions, state, (float*)out, dim);
  HL_LAUNCH_CHECK("decode_embed_kernel");
  count_launch(ctx);
  return HL_OK;
}

}  // namespace hl
