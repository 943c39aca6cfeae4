// 128-bit vectorised elementwise kernels, casts, bias add / bias gradient and grid reductions.
// Reference counterparts are one-thread-per-element scalar PTX entries
// (heirloom-kernels/src/ptx/kernels.ptx:6-312, :4610-4907).
#include "kernels.h"

namespace hl {
namespace {

constexpr int EW_THREADS = 256;

inline int ew_grid(hl_ctx* ctx, size_t vec_items) {
  size_t blocks = (vec_items + EW_THREADS - 1) / EW_THREADS;
  size_t cap = (size_t)ctx->sm_count * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct OpAdd { __device__ float operator()(float a, float b) const { return a + b; } };
struct OpSub { __device__ float operator()(float a, float b) const { return a - b; } };
struct OpMul { __device__ float operator()(float a, float b) const { return a * b; } };
struct OpDiv { __device__ float operator()(float a, float b) const { return a / b; } };

template <typename Op>
__global__ void binary_f32_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out,
                                  size_t n, bool vec) {
  pdl_begin();
  Op op;
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (vec) {
    const size_t n4 = n / 4;
    for (size_t i = tid; i < n4; i += stride) {
      const float4 x = reinterpret_cast<const float4*>(a)[i], y = reinterpret_cast<const float4*>(b)[i];
      reinterpret_cast<float4*>(out)[i] = make_float4(op(x.x, y.x), op(x.y, y.y), op(x.z, y.z), op(x.w, y.w));
    }
    for (size_t i = n4 * 4 + tid; i < n; i += stride) out[i] = op(a[i], b[i]);
  } else {
    for (size_t i = tid; i < n; i += stride) out[i] = op(a[i], b[i]);
  }
}

// Unary f32 map with an optional second input; F(x, y).
template <typename F>
__global__ void map_f32_kernel(const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ out,
                               size_t n, bool vec, F f) {
  pdl_begin();
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (vec) {
    const size_t n4 = n / 4;
    for (size_t i = tid; i < n4; i += stride) {
      const float4 a = x ? reinterpret_cast<const float4*>(x)[i] : make_float4(0, 0, 0, 0);
      const float4 b = y ? reinterpret_cast<const float4*>(y)[i] : make_float4(0, 0, 0, 0);
      reinterpret_cast<float4*>(out)[i] = make_float4(f(a.x, b.x), f(a.y, b.y), f(a.z, b.z), f(a.w, b.w));
    }
    for (size_t i = n4 * 4 + tid; i < n; i += stride) out[i] = f(x ? x[i] : 0.f, y ? y[i] : 0.f);
  } else {
    for (size_t i = tid; i < n; i += stride) out[i] = f(x ? x[i] : 0.f, y ? y[i] : 0.f);
  }
}

// bf16 map over 8-element vectors; F(x, y) in f32, result rounded to bf16.
template <typename F>
__global__ void map_bf16_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ y,
                                __nv_bfloat16* __restrict__ out, size_t n, bool vec, F f) {
  pdl_begin();
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (vec) {
    const size_t n8 = n / 8;
    for (size_t i = tid; i < n8; i += stride) {
      const uint4 a = reinterpret_cast<const uint4*>(x)[i];
      const uint4 b = y ? reinterpret_cast<const uint4*>(y)[i] : make_uint4(0, 0, 0, 0);
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
      uint32_t ow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 af = unpack_bf16x2(aw[j]), bf = unpack_bf16x2(bw[j]);
        ow[j] = pack_bf16x2(f(af.x, bf.x), f(af.y, bf.y));
      }
      reinterpret_cast<uint4*>(out)[i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
    for (size_t i = n8 * 8 + tid; i < n; i += stride)
      out[i] = to_bf16(f(from_bf16(x[i]), y ? from_bf16(y[i]) : 0.f));
  } else {
    for (size_t i = tid; i < n; i += stride) out[i] = to_bf16(f(from_bf16(x[i]), y ? from_bf16(y[i]) : 0.f));
  }
}

__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, size_t n,
                                        bool vec) {
  pdl_begin();
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (vec) {
    const size_t n8 = n / 8;
    for (size_t i = tid; i < n8; i += stride) {
      const float4 a = reinterpret_cast<const float4*>(src)[2 * i], b = reinterpret_cast<const float4*>(src)[2 * i + 1];
      reinterpret_cast<uint4*>(dst)[i] =
          make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    }
    for (size_t i = n8 * 8 + tid; i < n; i += stride) dst[i] = to_bf16(src[i]);
  } else {
    for (size_t i = tid; i < n; i += stride) dst[i] = to_bf16(src[i]);
  }
}

__global__ void cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, size_t n,
                                        bool vec) {
  pdl_begin();
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (vec) {
    const size_t n8 = n / 8;
    for (size_t i = tid; i < n8; i += stride) {
      const uint4 a = reinterpret_cast<const uint4*>(src)[i];
      const float2 f0 = unpack_bf16x2(a.x), f1 = unpack_bf16x2(a.y), f2 = unpack_bf16x2(a.z), f3 = unpack_bf16x2(a.w);
      reinterpret_cast<float4*>(dst)[2 * i] = make_float4(f0.x, f0.y, f1.x, f1.y);
      reinterpret_cast<float4*>(dst)[2 * i + 1] = make_float4(f2.x, f2.y, f3.x, f3.y);
    }
    for (size_t i = n8 * 8 + tid; i < n; i += stride) dst[i] = from_bf16(src[i]);
  } else {
    for (size_t i = tid; i < n; i += stride) dst[i] = from_bf16(src[i]);
  }
}

__global__ void bias_add_f32_kernel(const float* __restrict__ x, const float* __restrict__ bias, float* __restrict__ out,
                                    size_t total, int cols) {
  pdl_begin();
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = tid; i < total; i += stride) out[i] = x[i] + bias[i % cols];
}

// Column sums, stage 1: each block owns a slab of rows and 32 columns; threads (32 x 8) walk
// rows with coalesced 32-wide reads, partial sums in double, then a shared-memory reduce.
template <typename T>
__global__ void colsum_partial_kernel(const T* __restrict__ g, double* __restrict__ partial, int rows, int cols,
                                      int rows_per_block) {
  pdl_begin();
  __shared__ double tile[8][33];
  const int col = blockIdx.x * 32 + threadIdx.x;
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(rows, r0 + rows_per_block);
  double acc = 0.0;
  if (col < cols) {
    for (int r = r0 + threadIdx.y; r < r1; r += 8) {
      float v;
      if constexpr (sizeof(T) == 2) v = from_bf16(g[(size_t)r * cols + col]);
      else v = g[(size_t)r * cols + col];
      acc += (double)v;
    }
  }
  tile[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && col < cols) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += tile[j][threadIdx.x];
    partial[(size_t)blockIdx.y * cols + col] = s;
  }
}

__global__ void colsum_final_kernel(const double* __restrict__ partial, float* __restrict__ out, int cols, int slabs) {
  pdl_begin();
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= cols) return;
  double s = 0.0;
  for (int j = 0; j < slabs; ++j) s += partial[(size_t)j * cols + col];
  out[col] = (float)s;
}

// f32 -> f64 with integer instructions (rebias the exponent, shift; zero keeps its bits, subnormals, infinities and NaNs go
// through the instruction): the conversion instruction takes a warp about 14 cycles of its SM, which would bound a
// reduction of f32 values at half the memory rate.
__device__ __forceinline__ double widen_f32(float x) {
  const uint32_t u = __float_as_uint(x), t = u << 1;
  if (t - 0x01000000u >= 0xfe000000u && t != 0u) return (double)x;
  const uint32_t hi = t == 0u ? u : ((u & 0x7fffffffu) >> 3) + 0x38000000u + (u & 0x80000000u);
  return __hiloint2double((int)hi, (int)(u << 29));
}

// Grid reduction: per-block double partial sums, folded in a fixed order by a second kernel.  Four 16-byte loads a thread in
// flight and a partial sum each: one scalar load at a time reached 1.1 TB/s on a 54 M-element gradient (187 us), this is
// bound by the loads (see the block count in reduce_impl).
template <int MODE>  // 0 sum, 1 sum of squares
__global__ void __launch_bounds__(256)
reduce_partial_kernel(const float* __restrict__ x, size_t n, bool vec, double* __restrict__ partial) {
  pdl_begin();
  __shared__ double sm[32];
  double acc = 0.0;
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  auto term = [](float f) { const double v = widen_f32(f); return MODE == 1 ? v * v : v; };
  size_t done = 0;
  if (vec) {
    const size_t n4 = n / 4;
    for (size_t i = tid; i < n4; i += 4 * stride) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[u] = i + u * stride < n4 ? __ldg(reinterpret_cast<const float4*>(x) + i + u * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 4; ++u) acc += (term(v[u].x) + term(v[u].y)) + (term(v[u].z) + term(v[u].w));
    }
    done = n4 * 4;
  }
  for (size_t i = done + tid; i < n; i += stride) acc += term(x[i]);
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

__global__ void reduce_final_kernel(const double* __restrict__ partial, int count, double scale, float* __restrict__ out,
                                    float* __restrict__ out_host) {
  pdl_begin();
  __shared__ double sm[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) acc += partial[i];
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) {
    out[0] = (float)(acc * scale);
    if (out_host) out_host[0] = (float)(acc * scale);
  }
}

// `out_host`: pinned memory that gets the result as well, or null.
int reduce_impl(hl_ctx* ctx, const float* x, size_t n, float* out_dev, int mode, double scale, float* out_host = nullptr) {
  HL_REQUIRE(ctx && out_dev && (x || n == 0), "reduction: null argument");
  const int blocks = (int)std::min<size_t>(std::max<size_t>((n + 4095) / 4096, 1), (size_t)ctx->sm_count * 8);
  const bool vec = aligned16(x);
  int rc = ensure_workspace(ctx, sizeof(double) * blocks);
  if (rc != HL_OK) return rc;
  double* partial = reinterpret_cast<double*>(ctx->workspace);
  if (mode == 1) pdl(reduce_partial_kernel<1>, blocks, 256, 0, ctx->stream).streaming(4.0 * n)(x, n, vec, partial);
  else pdl(reduce_partial_kernel<0>, blocks, 256, 0, ctx->stream).streaming(4.0 * n)(x, n, vec, partial);
  HL_LAUNCH_CHECK("reduce_partial_kernel");
  pdl(reduce_final_kernel, 1, 256, 0, ctx->stream)(partial, blocks, scale, out_dev, out_host);
  HL_LAUNCH_CHECK("reduce_final_kernel");
  count_launch(ctx, 2);
  return HL_OK;
}

}  // namespace

int sum_squares_impl(hl_ctx* ctx, const float* x, size_t n, float* out_dev, float* out_host) {
  return reduce_impl(ctx, x, n, out_dev, 1, 1.0, out_host);
}

int bias_grad_impl(hl_ctx* ctx, const void* grad_out, int dtype, float* grad_bias, int rows, int cols, FoldBatch* defer) {
  HL_REQUIRE(ctx && grad_out && grad_bias, "hl_bias_grad: null argument");
  HL_REQUIRE(rows > 0 && cols > 0, "hl_bias_grad: rows and cols must be positive");
  HL_REQUIRE(dtype == HL_F32 || dtype == HL_BF16, "hl_bias_grad: dtype must be f32 or bf16");
  ProfileScope prof(ctx, HL_PROF_BIAS_GRAD, (double)rows * cols * (double)dtype_size(dtype));
  if (colsum_fast_applicable(dtype, cols, grad_out)) return colsum_fast(ctx, grad_out, dtype, grad_bias, rows, cols, defer);
  int slabs = std::min(std::max(rows / 256, 1), 64);
  const int rows_per_block = ceil_div(rows, slabs);
  slabs = ceil_div(rows, rows_per_block);
  int rc = ensure_workspace(ctx, sizeof(double) * (size_t)slabs * cols);
  if (rc != HL_OK) return rc;
  double* partial = reinterpret_cast<double*>(ctx->workspace);
  dim3 grid(ceil_div(cols, 32), slabs), block(32, 8);
  if (dtype == HL_BF16)
    pdl(colsum_partial_kernel<__nv_bfloat16>, grid, block, 0, ctx->stream)(
        reinterpret_cast<const __nv_bfloat16*>(grad_out), partial, rows, cols, rows_per_block);
  else
    pdl(colsum_partial_kernel<float>, grid, block, 0, ctx->stream)(reinterpret_cast<const float*>(grad_out), partial,
                                                                    rows, cols, rows_per_block);
  HL_LAUNCH_CHECK("colsum_partial_kernel");
  pdl(colsum_final_kernel, ceil_div(cols, 256), 256, 0, ctx->stream)(partial, grad_bias, cols, slabs);
  HL_LAUNCH_CHECK("colsum_final_kernel");
  count_launch(ctx, 2);
  return HL_OK;
}

}  // namespace hl

using namespace hl;

namespace hl {
namespace {

__device__ __forceinline__ void load8(const float* p, float (&x)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&x)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(x[4], x[5], x[6], x[7]);
}
__device__ __forceinline__ void put_pieces(const PieceDest& d, unsigned row, unsigned col, const uint4 (&piece)[3]) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (j < d.n) {
      const uint4 v = d.id[j] == 0 ? piece[0] : d.id[j] == 1 ? piece[1] : piece[2];
      *reinterpret_cast<uint4*>(d.out + row * d.ld + j * d.piece + col) = v;
    }
}

// Bound by memory: eight values a thread, sixteen bytes a store, an operand that is wanted both stacked and side by side read
// once.  An element a thread with two-byte stores took 20.9 us for three pieces of 16384 x 512 and 17.0 for two, one layout each.
__global__ void split_pieces_kernel(const float* __restrict__ src, unsigned groups, unsigned per_row, const PieceDest a, const PieceDest b) {
  pdl_begin();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += gridDim.x * blockDim.x) {
    const unsigned row = i / per_row, col = (i - row * per_row) * 8;
    float x[8];
    load8(src + (size_t)i * 8, x);
    uint4 piece[3];
    split8_bf16(x, piece);
    put_pieces(a, row, col, piece);
    put_pieces(b, row, col, piece);
  }
}

// The gate of a memory block and what the next product reads of it in one pass over memory: 166 MB for 16384 x 512 where a kernel
// for each op moved 231 MB forward, and 281 MB instead of 451 MB backward.
__global__ void memory_gate_fwd_kernel(const float* __restrict__ gpre, const float* __restrict__ weighted, float* __restrict__ gate,
                                       float* __restrict__ mv, unsigned groups, unsigned per_row, const PieceDest a) {
  pdl_begin();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += gridDim.x * blockDim.x) {
    const unsigned row = i / per_row, col = (i - row * per_row) * 8;
    const size_t at = (size_t)i * 8;
    float g[8], w[8];
    load8(gpre + at, g);
    load8(weighted + at, w);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      g[e] = (float)gelu_fwd<double>((double)g[e]);
      w[e] *= g[e];
    }
    store8(gate + at, g);
    store8(mv + at, w);
    uint4 piece[3];
    split8_bf16(w, piece);
    put_pieces(a, row, col, piece);
  }
}
__global__ void memory_gate_bwd_kernel(const float* __restrict__ dmv, const float* __restrict__ gate, const float* __restrict__ weighted,
                                       const float* __restrict__ gpre, float* __restrict__ dweighted, float* __restrict__ dgpre,
                                       unsigned groups, unsigned per_row, const PieceDest a, const PieceDest b) {
  pdl_begin();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += gridDim.x * blockDim.x) {
    const unsigned row = i / per_row, col = (i - row * per_row) * 8;
    const size_t at = (size_t)i * 8;
    float d[8], t[8], x[8];
    load8(dmv + at, d);
    load8(gate + at, t);
    load8(gpre + at, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) t[e] *= d[e];
    store8(dweighted + at, t);
    load8(weighted + at, t);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = (float)((double)(d[e] * t[e]) * gelu_grad<double>((double)x[e]));
    store8(dgpre + at, x);
    uint4 piece[3];
    split8_bf16(x, piece);
    put_pieces(a, row, col, piece);
    put_pieces(b, row, col, piece);
  }
}

bool dest_fits(const PieceDest& d) { return d.n == 0 || (d.ld % 8 == 0 && d.piece % 8 == 0 && aligned16(d.out)); }
bool pieces_fit(long long rows, int cols, const PieceDest& a, const PieceDest& b) {
  return cols % 8 == 0 && rows * (cols / 8) < (1ll << 31) && dest_fits(a) && dest_fits(b);
}

}  // namespace

int split_pieces(hl_ctx* ctx, const float* src, long long rows, int cols, const PieceDest& a, const PieceDest& b) {
  HL_REQUIRE(aligned16(src) && pieces_fit(rows, cols, a, b), "split_pieces: rows of eight values on 16 bytes");
  const unsigned groups = (unsigned)(rows * (cols / 8));
  pdl(split_pieces_kernel, ew_grid(ctx, groups), EW_THREADS, 0, ctx->stream).streaming(16.0 * groups * (2 + a.n + b.n))(src, groups, (unsigned)(cols / 8), a, b);
  HL_LAUNCH_CHECK("split_pieces_kernel");
  count_launch(ctx);
  return HL_OK;
}

int memory_gate_forward(hl_ctx* ctx, const float* gpre, const float* weighted, float* gate, float* mv, long long rows, int cols, const PieceDest& a) {
  HL_REQUIRE(pieces_fit(rows, cols, a, PieceDest{}), "memory_gate_forward: rows of eight values on 16 bytes");
  const unsigned groups = (unsigned)(rows * (cols / 8));
  pdl(memory_gate_fwd_kernel, ew_grid(ctx, groups), EW_THREADS, 0, ctx->stream).streaming(16.0 * groups * (8 + a.n))(gpre, weighted, gate, mv, groups,
                                                                                                                     (unsigned)(cols / 8), a);
  HL_LAUNCH_CHECK("memory_gate_fwd_kernel");
  count_launch(ctx);
  return HL_OK;
}

int memory_gate_backward(hl_ctx* ctx, const float* dmv, const float* gate, const float* weighted, const float* gpre, float* dweighted, float* dgpre,
                         long long rows, int cols, const PieceDest& a, const PieceDest& b) {
  HL_REQUIRE(pieces_fit(rows, cols, a, b), "memory_gate_backward: rows of eight values on 16 bytes");
  const unsigned groups = (unsigned)(rows * (cols / 8));
  pdl(memory_gate_bwd_kernel, ew_grid(ctx, groups), EW_THREADS, 0, ctx->stream).streaming(16.0 * groups * (12 + a.n + b.n))(
      dmv, gate, weighted, gpre, dweighted, dgpre, groups, (unsigned)(cols / 8), a, b);
  HL_LAUNCH_CHECK("memory_gate_bwd_kernel");
  count_launch(ctx);
  return HL_OK;
}

}  // namespace hl

extern "C" {

int hl_binary_f32(hl_ctx* ctx, int op, const float* a, const float* b, float* out, size_t n) {
  HL_REQUIRE(ctx && ((a && b && out) || n == 0), "hl_binary_f32: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(a) && aligned16(b) && aligned16(out);
  const int grid = ew_grid(ctx, vec ? n / 4 + 1 : n);
  switch (op) {
    case HL_ADD: pdl(binary_f32_kernel<OpAdd>, grid, EW_THREADS, 0, ctx->stream)(a, b, out, n, vec); break;
    case HL_SUB: pdl(binary_f32_kernel<OpSub>, grid, EW_THREADS, 0, ctx->stream)(a, b, out, n, vec); break;
    case HL_MUL: pdl(binary_f32_kernel<OpMul>, grid, EW_THREADS, 0, ctx->stream)(a, b, out, n, vec); break;
    case HL_DIV: pdl(binary_f32_kernel<OpDiv>, grid, EW_THREADS, 0, ctx->stream)(a, b, out, n, vec); break;
    default: return fail("hl_binary_f32: unknown op");
  }
  HL_LAUNCH_CHECK("binary_f32_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_scale_f32(hl_ctx* ctx, const float* a, float s, float* out, size_t n) {
  HL_REQUIRE(ctx && ((a && out) || n == 0), "hl_scale_f32: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(a) && aligned16(out);
  map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
      a, (const float*)nullptr, out, n, vec, [s] __device__(float x, float) { return x * s; });
  HL_LAUNCH_CHECK("scale_f32");
  count_launch(ctx);
  return HL_OK;
}

int hl_fill_f32(hl_ctx* ctx, float* out, float value, size_t n) {
  HL_REQUIRE(ctx && (out || n == 0), "hl_fill_f32: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(out);
  map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
      (const float*)nullptr, (const float*)nullptr, out, n, vec, [value] __device__(float, float) { return value; });
  HL_LAUNCH_CHECK("fill_f32");
  count_launch(ctx);
  return HL_OK;
}

// ---- plain SGD, index ranges and index concatenation ---------------------------------------------------------
static __global__ void sgd_update_kernel(float* __restrict__ param, const float* __restrict__ grad, float lr, size_t n) {
  pdl_begin();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    param[i] = __fsub_rn(param[i], __fmul_rn(lr, grad[i]));  // two roundings, as the reference's mul then sub
}
static __global__ void arange_i64_kernel(int64_t* __restrict__ out, size_t n) {
  pdl_begin();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = (int64_t)i;
}
static __global__ void copy_i64_kernel(const int64_t* __restrict__ src, int64_t* __restrict__ dst, size_t n) {
  pdl_begin();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

int hl_sgd_update_f32(hl_ctx* ctx, float* param, const float* grad, float lr, size_t n) {
  HL_REQUIRE(ctx && ((param && grad) || n == 0), "hl_sgd_update_f32: null argument");
  HL_REQUIRE(lr > 0.f, "sgd_update_f32_buffer learning rate must be positive, got " + std::to_string(lr));
  if (n == 0) return HL_OK;
  pdl(sgd_update_kernel, ew_grid(ctx, n), EW_THREADS, 0, ctx->stream)(param, grad, lr, n);
  HL_LAUNCH_CHECK("sgd_update_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_arange_i64(hl_ctx* ctx, int64_t* out, size_t n) {
  HL_REQUIRE(ctx && (out || n == 0), "hl_arange_i64: null argument");
  HL_REQUIRE(n <= 0xffffffffull, "i64_arange len exceeds the u32 launch limit");
  if (n == 0) return HL_OK;
  pdl(arange_i64_kernel, ew_grid(ctx, n), EW_THREADS, 0, ctx->stream)(out, n);
  HL_LAUNCH_CHECK("arange_i64_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_concat_i64(hl_ctx* ctx, const int64_t* const* inputs, const size_t* lengths, int count, int64_t* out, size_t out_capacity) {
  HL_REQUIRE(ctx && inputs && lengths, "hl_concat_i64: null argument");
  HL_REQUIRE(count >= 1, "concat_i64_buffers requires at least one input buffer");
  size_t total = 0;
  for (int i = 0; i < count; ++i) {
    HL_REQUIRE(lengths[i] == 0 || inputs[i], "hl_concat_i64: null input buffer");
    HL_REQUIRE(total + lengths[i] >= total, "concat_i64_buffers total length overflow");
    total += lengths[i];
  }
  HL_REQUIRE(total <= out_capacity, "hl_concat_i64: the output holds " + std::to_string(out_capacity) + " elements, the inputs " +
                                        std::to_string(total));
  HL_REQUIRE(out || total == 0, "hl_concat_i64: null output");
  size_t offset = 0;
  for (int i = 0; i < count; ++i) {
    if (lengths[i] == 0) continue;
    pdl(copy_i64_kernel, ew_grid(ctx, lengths[i]), EW_THREADS, 0, ctx->stream)(inputs[i], out + offset, lengths[i]);
    HL_LAUNCH_CHECK("copy_i64_kernel");
    count_launch(ctx);
    offset += lengths[i];
  }
  return HL_OK;
}

int hl_relu_f32(hl_ctx* ctx, const float* x, float* out, size_t n) {
  HL_REQUIRE(ctx && ((x && out) || n == 0), "hl_relu_f32: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(x) && aligned16(out);
  map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
      x, (const float*)nullptr, out, n, vec, [] __device__(float v, float) { return v > 0.f ? v : 0.f; });
  HL_LAUNCH_CHECK("relu_f32");
  count_launch(ctx);
  return HL_OK;
}

int hl_relu_backward_f32(hl_ctx* ctx, const float* x, const float* grad_out, float* grad_in, size_t n) {
  HL_REQUIRE(ctx && ((x && grad_out && grad_in) || n == 0), "hl_relu_backward_f32: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(x) && aligned16(grad_out) && aligned16(grad_in);
  map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
      x, grad_out, grad_in, n, vec, [] __device__(float v, float g) { return v > 0.f ? g : 0.f; });
  HL_LAUNCH_CHECK("relu_backward_f32");
  count_launch(ctx);
  return HL_OK;
}

int hl_cast(hl_ctx* ctx, const void* src, int src_dtype, void* dst, int dst_dtype, size_t n) {
  HL_REQUIRE(ctx && ((src && dst) || n == 0), "hl_cast: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(src) && aligned16(dst);
  const int grid = ew_grid(ctx, vec ? n / 8 + 1 : n);
  if (src_dtype == HL_F32 && dst_dtype == HL_BF16) {
    pdl(cast_f32_to_bf16_kernel, grid, EW_THREADS, 0, ctx->stream)((const float*)src, (__nv_bfloat16*)dst, n, vec);
  } else if (src_dtype == HL_BF16 && dst_dtype == HL_F32) {
    pdl(cast_bf16_to_f32_kernel, grid, EW_THREADS, 0, ctx->stream)((const __nv_bfloat16*)src, (float*)dst, n, vec);
  } else if (src_dtype == HL_F32 && dst_dtype == HL_F32) {
    map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
        (const float*)src, (const float*)nullptr, (float*)dst, n, vec,
        [] __device__(float v, float) { return bf16_round(v); });
  } else {
    return fail("hl_cast: supported pairs are f32->bf16, bf16->f32 and the f32 bf16-round-trip");
  }
  HL_LAUNCH_CHECK("cast kernel");
  count_launch(ctx);
  return HL_OK;
}

// The same for rows that are no multiple of eight values, or not on 16 bytes: an element a thread.
static __global__ void split_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long rows, int cols,
                                  int mode_bits) {
  pdl_begin();
  const int mode = mode_bits & 3;
  const bool stacked = (mode_bits & HL_SPLIT_STACK_ROWS) != 0;
  const int pieces = mode == HL_SPLIT_HI_LO ? 2 : 3;
  const long long n = rows * cols;
  const long long piece_stride = stacked ? n : cols;            // distance between the pieces of one element
  const long long ld = stacked ? cols : (long long)pieces * cols;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / cols;
    const int c = (int)(i - r * cols);
    const float x = src[i];
    const __nv_bfloat16 hi = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(hi);
    const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
    const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
    __nv_bfloat16* out = dst + r * ld + c;
    out[0] = hi;
    if (mode == HL_SPLIT_HI_MID_LO) { out[piece_stride] = mid; out[2 * piece_stride] = lo; }
    else if (mode == HL_SPLIT_HI_HI_LO) { out[piece_stride] = hi; out[2 * piece_stride] = mid; }
    else out[piece_stride] = mid;
  }
}

int hl_split_bf16_f32(hl_ctx* ctx, const float* src, void* dst, long long rows, int cols, int mode) {
  HL_REQUIRE(ctx && src && dst, "hl_split_bf16_f32: null argument");
  HL_REQUIRE(rows > 0 && cols > 0, "hl_split_bf16_f32: requires non-zero rows/cols");
  HL_REQUIRE((mode & ~(3 | HL_SPLIT_STACK_ROWS)) == 0 && (mode & 3) != 3, "hl_split_bf16_f32: unknown mode");
  const int n = (mode & 3) == HL_SPLIT_HI_LO ? 2 : 3, second = (mode & 3) == HL_SPLIT_HI_HI_LO ? 0 : 1, third = (mode & 3) == HL_SPLIT_HI_HI_LO ? 1 : 2;
  __nv_bfloat16* out = (__nv_bfloat16*)dst;
  const PieceDest dest = mode & HL_SPLIT_STACK_ROWS ? pieces_stacked(out, rows, cols, n, 0, second, third)
                                                    : pieces_beside(out, (long long)n * cols, cols, n, 0, second, third);
  if (aligned16(src) && pieces_fit(rows, cols, dest, PieceDest{})) return split_pieces(ctx, src, rows, cols, dest);
  pdl(split_bf16_kernel, ew_grid(ctx, (size_t)rows * cols), EW_THREADS, 0, ctx->stream)(src, (__nv_bfloat16*)dst, rows, cols, mode);
  HL_LAUNCH_CHECK("split_bf16_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_gelu(hl_ctx* ctx, const void* x, void* out, int dtype, size_t n) {
  HL_REQUIRE(ctx && ((x && out) || n == 0), "hl_gelu: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(x) && aligned16(out);
  if (dtype == HL_F32) {
    // f32 tensors are evaluated in double so the f32 result is correctly rounded from the
    // same f64 expression the reference evaluates.
    map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
        (const float*)x, (const float*)nullptr, (float*)out, n, vec,
        [] __device__(float v, float) { return (float)gelu_fwd<double>((double)v); });
  } else if (dtype == HL_BF16) {
    map_bf16_kernel<<<ew_grid(ctx, vec ? n / 8 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)nullptr, (__nv_bfloat16*)out, n, vec,
        [] __device__(float v, float) { return gelu_fwd_f(v); });
  } else {
    return fail("hl_gelu: dtype must be f32 or bf16");
  }
  HL_LAUNCH_CHECK("gelu kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_gelu_backward(hl_ctx* ctx, const void* x, const void* grad_out, void* grad_in, int dtype, size_t n) {
  HL_REQUIRE(ctx && ((x && grad_out && grad_in) || n == 0), "hl_gelu_backward: null argument");
  if (n == 0) return HL_OK;
  const bool vec = aligned16(x) && aligned16(grad_out) && aligned16(grad_in);
  if (dtype == HL_F32) {
    map_f32_kernel<<<ew_grid(ctx, vec ? n / 4 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
        (const float*)x, (const float*)grad_out, (float*)grad_in, n, vec,
        [] __device__(float v, float g) { return (float)((double)g * gelu_grad<double>((double)v)); });
  } else if (dtype == HL_BF16) {
    map_bf16_kernel<<<ew_grid(ctx, vec ? n / 8 + 1 : n), EW_THREADS, 0, ctx->stream>>>(
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)grad_out, (__nv_bfloat16*)grad_in, n, vec,
        [] __device__(float v, float g) { return g * gelu_grad_f(v); });
  } else {
    return fail("hl_gelu_backward: dtype must be f32 or bf16");
  }
  HL_LAUNCH_CHECK("gelu backward kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_bias_add_f32(hl_ctx* ctx, const float* x, const float* bias, float* out, int rows, int cols) {
  HL_REQUIRE(ctx && x && bias && out, "hl_bias_add_f32: null argument");
  HL_REQUIRE(rows > 0 && cols > 0, "hl_bias_add_f32: rows and cols must be positive");
  const size_t total = (size_t)rows * cols;
  pdl(bias_add_f32_kernel, ew_grid(ctx, total), EW_THREADS, 0, ctx->stream)(x, bias, out, total, cols);
  HL_LAUNCH_CHECK("bias_add_f32_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_bias_grad(hl_ctx* ctx, const void* grad_out, int dtype, float* grad_bias, int rows, int cols) {
  return bias_grad_impl(ctx, grad_out, dtype, grad_bias, rows, cols);
}

int hl_sum_f32(hl_ctx* ctx, const float* x, size_t n, float* out_dev) { return reduce_impl(ctx, x, n, out_dev, 0, 1.0); }
int hl_mean_f32(hl_ctx* ctx, const float* x, size_t n, float* out_dev) {
  HL_REQUIRE(n > 0, "hl_mean_f32: empty input");
  return reduce_impl(ctx, x, n, out_dev, 0, 1.0 / (double)n);
}
int hl_sum_squares_f32(hl_ctx* ctx, const float* x, size_t n, float* out_dev) {
  return reduce_impl(ctx, x, n, out_dev, 1, 1.0);
}

}  // extern "C"
