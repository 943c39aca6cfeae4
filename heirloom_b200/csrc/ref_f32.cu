// f32 kernels with f64 accumulation for the f32 parity route: strided matmul and causal
// attention with materialised probabilities.  These follow the reference's f32 CUDA entries
// (heirloom-kernels/src/ptx/kernels.ptx:1290-1659 matmul, :3760-4609 attention) in what they
// compute, but accumulate in double so that their f32 results round from the same f64 values
// the reference's CPU path produces (src/tensor.rs:577-590).
//
// Every product runs on the f64 tensor instruction (mma.m8n8k4): operands are widened once, on their way into shared
// memory, and a warp then reads one f64 per lane and operand fragment for 256 multiply-adds, where plain f64 FMAs read
// two operands per multiply-add out of a 16 x 16 tile.
#include <cooperative_groups.h>

#include "kernels.h"
#include "tc05.cuh"

namespace hl {
namespace {

namespace cg = cooperative_groups;

// D (8x8) += A (8x4, row lane/4, k lane%4) * B (4x8, k lane%4, column lane/4); D: row lane/4, columns 2*(lane%4) + {0,1}
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ double widen(float x) { return (double)x; }
__device__ __forceinline__ double widen(__nv_bfloat16 x) { return (double)__bfloat162float(x); }
__device__ __forceinline__ void narrow(float* p, double v) { *p = (float)v; }
__device__ __forceinline__ void narrow(__nv_bfloat16* p, double v) { *p = __float2bfloat16_rn((float)v); }  // through f32

// ---- strided matmul --------------------------------------------------------------------------------
// One CTA of eight warps per TM x TN output tile: 64 x 64 when those fill the chip, else 32 x 32.
//
// The large tile goes through k in steps of 32, copied ahead as f32 by cp.async (four bytes a copy: any stride, zero fill at the
// edges); each thread widens the elements it copied itself into one of two f64 buffers, and one barrier a step separates
// widening from multiplying.  Shared rows are padded so that a half warp's fragment (4 rows x 4 k) falls into 16 different
// 8-byte banks whichever index is contiguous, and the four combinations of contiguous indices are compiled apart.
//
// The small tile is for products that take microseconds, where steps, barriers and instructions counted for more than the
// multiply-adds (1024 x 512 x 128: 3.7 us of those, 14.6 us in steps as above).  Four groups of two warps take 32 of every 128 k
// each, a warp 32 rows by 16 columns of all of the tile, so that its fragments come straight from memory, sixteen bytes a load
// and all of them in flight, are widened in registers and meet the other groups' sums once, at the end.  Which k, row or column
// stands in which place of a fragment is free as long as both operands, or the result, agree; it is chosen so that what a
// lane needs is contiguous.
//
// Small outputs with a long contraction (weight gradients) are shared by the CTAs of a cluster: each takes a part of k,
// and the parts are added in rank order through distributed shared memory, so the result does not depend on timing.
// Two independent products may share a launch (an input gradient beside its weight gradient).
constexpr int F64_THREADS = 256;
constexpr int F64_BK = 32;
constexpr int F64_JOBS = 2;

struct F64Job {
  F64Gemm g;
  int cta0;              // first CTA of this product
  int tiles, tiles_n;    // output tiles, tile columns
  int split;             // CTAs per tile: 1 or the cluster size
  int k_tiles_per_rank;
};
struct F64Jobs {
  F64Job job[F64_JOBS];
  int count;
  int cluster;
};

__device__ __forceinline__ void copy_async4(float* dst_shared, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_shared)), "l"(src),
               "r"(in ? 4 : 0)
               : "memory");
}

// One operand of a tile, ROWS x 32 a step.  KM: the contraction index is contiguous in memory.
template <int ROWS, bool KM>
struct F64Operand {
  static constexpr int PER_THREAD = ROWS * F64_BK / F64_THREADS;
  static constexpr int LD = KM ? F64_BK + 4 : ROWS + 4;     // [row][k] or [k][row]
  static constexpr int ROW = KM ? LD : 1, K = KM ? 1 : LD;  // element strides in the f64 buffer
  static constexpr int I_ROWS = KM ? F64_THREADS / F64_BK : 0, I_K = KM ? 0 : F64_THREADS / ROWS;  // from one copy to the next
  const float* p;      // this thread's first element of the next step
  long long i_step, k_step;
  unsigned rows_in;    // per copy: its row exists
  int k_left;          // contraction elements from this thread's first one to the end
  int slot;            // its place in the f64 buffer
  __device__ __forceinline__ void init(const float* base, long long row_stride, long long k_stride, int row0, int rows, int k0, int k) {
    const int tid = threadIdx.x;
    const int r = KM ? tid / F64_BK : tid % ROWS, kk = KM ? tid % F64_BK : tid / ROWS;
    p = base + (row0 + r) * row_stride + (k0 + kk) * k_stride;
    i_step = I_ROWS * row_stride + I_K * k_stride;
    k_step = F64_BK * k_stride;
    rows_in = 0;
#pragma unroll
    for (int i = 0; i < PER_THREAD; ++i) rows_in |= (row0 + r + i * I_ROWS < rows ? 1u : 0u) << i;
    k_left = k - (k0 + kk);
    slot = r * ROW + kk * K;
  }
  __device__ __forceinline__ void request(float* dst, const float* safe) {
    const float* q = p;
#pragma unroll
    for (int i = 0; i < PER_THREAD; ++i) {
      const bool in = ((rows_in >> i) & 1u) && i * I_K < k_left;
      copy_async4(dst + i * F64_THREADS, in ? q : safe, in);
      q += i_step;
    }
    p += k_step;
    k_left -= F64_BK;
  }
  __device__ __forceinline__ void widen_into(double* dst, const float* src) const {
#pragma unroll
    for (int i = 0; i < PER_THREAD; ++i) dst[slot + i * (I_ROWS * ROW + I_K * K)] = (double)src[i * F64_THREADS];
  }
};

template <int TM, int TN>
struct F64Tile {
  static constexpr int WK = 1;                             // groups of warps along k
  static constexpr int WM = 4, WN = 2;                     // warps along the tile
  static_assert(WM * WN * 32 == F64_THREADS, "eight warps");
  static constexpr int FM = TM / (8 * WM), FN = TN / (8 * WN);  // 8 x 8 fragments per warp
  static constexpr int A_ELEMS = TM * (F64_BK + 4), B_ELEMS = TN * (F64_BK + 4);  // either layout fits
  static_assert(F64_BK * (TM + 4) <= A_ELEMS && F64_BK * (TN + 4) <= B_ELEMS, "both layouts share the buffers");
  static constexpr int LDC = TN + 2;
  static constexpr int PART = TM * LDC + TM;               // the tile's sums and the row sums
  static_assert(PART <= 2 * (A_ELEMS + B_ELEMS), "the output tile reuses the operand buffers");
  static constexpr int RAW = (TM + TN) * F64_BK;           // one copied step, in the order the threads copied it
  static constexpr int DEPTH = 2;
  static constexpr size_t SMEM = sizeof(double) * 2 * (A_ELEMS + B_ELEMS) + sizeof(float) * DEPTH * RAW;
};

template <int TM, int TN, bool A_KM, bool B_KM>
__device__ __forceinline__ void f64_tile_sums(const F64Gemm& g, double* smem, int row0, int col0, int kt0, int kt1, bool sums) {
  using Z = F64Tile<TM, TN>;
  using OA = F64Operand<TM, A_KM>;
  using OB = F64Operand<TN, B_KM>;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* raw = reinterpret_cast<float*>(smem + 2 * (Z::A_ELEMS + Z::B_ELEMS)) + tid;
  OA oa;
  OB ob;
  oa.init(g.a, g.a_row, g.a_col, row0, g.m, kt0 * F64_BK, g.k);
  ob.init(g.b, g.b_col, g.b_row, col0, g.n, kt0 * F64_BK, g.k);
  const int steps = kt1 - kt0;
  auto request = [&](int step) {
    if (step < steps) {
      float* dst = raw + step % Z::DEPTH * Z::RAW;
      oa.request(dst, g.a);
      ob.request(dst + OA::PER_THREAD * F64_THREADS, g.b);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int wm = warp / Z::WN * (Z::FM * 8), wn = warp % Z::WN * (Z::FN * 8);
  const int fr = lane >> 2, fk = lane & 3;
  double acc[Z::FM][Z::FN][2], rs[Z::FM][2];
#pragma unroll
  for (int i = 0; i < Z::FM; ++i) {
    rs[i][0] = rs[i][1] = 0.0;
#pragma unroll
    for (int j = 0; j < Z::FN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  }
  const bool my_sums = sums && wn == 0;
#pragma unroll
  for (int s = 0; s < Z::DEPTH; ++s) request(s);
  for (int step = 0; step < steps; ++step) {
    double* buf = smem + (step & 1) * (Z::A_ELEMS + Z::B_ELEMS);
    asm volatile("cp.async.wait_group %0;" ::"n"(Z::DEPTH - 1) : "memory");  // this thread's copies of the step have landed
    const float* src = raw + step % Z::DEPTH * Z::RAW;
    oa.widen_into(buf, src);
    ob.widen_into(buf + Z::A_ELEMS, src + OA::PER_THREAD * F64_THREADS);
    request(step + Z::DEPTH);
    __syncthreads();
    const double* sa = buf + (wm + fr) * OA::ROW + fk * OA::K;
    const double* sb = buf + Z::A_ELEMS + (wn + fr) * OB::ROW + fk * OB::K;
#pragma unroll
    for (int kk = 0; kk < F64_BK; kk += 4) {
      double fa[Z::FM], fb[Z::FN];
#pragma unroll
      for (int i = 0; i < Z::FM; ++i) fa[i] = sa[i * 8 * OA::ROW + kk * OA::K];
#pragma unroll
      for (int j = 0; j < Z::FN; ++j) fb[j] = sb[j * 8 * OB::ROW + kk * OB::K];
#pragma unroll
      for (int i = 0; i < Z::FM; ++i)
#pragma unroll
        for (int j = 0; j < Z::FN; ++j) dmma(acc[i][j], fa[i], fb[j]);
      if (my_sums) {  // row sums of A: a bias gradient rides on its weight gradient
#pragma unroll
        for (int i = 0; i < Z::FM; ++i) dmma(rs[i], fa[i], 1.0);
      }
    }
  }
  __syncthreads();
  double* sc = smem;
#pragma unroll
  for (int i = 0; i < Z::FM; ++i) {
#pragma unroll
    for (int j = 0; j < Z::FN; ++j) {
      double* d = sc + (wm + i * 8 + fr) * Z::LDC + wn + j * 8 + 2 * fk;
      d[0] = acc[i][j][0];
      d[1] = acc[i][j][1];
    }
    if (my_sums && fk == 0) sc[TM * Z::LDC + wm + i * 8 + fr] = rs[i][0];
  }
}

template <>
struct F64Tile<32, 32> {
  static constexpr int WK = 4, LDC = 34, PART = 32 * LDC + 32;
  static constexpr size_t SMEM = sizeof(double) * WK * PART;
};

// Up to four values, zero past `left`; `vec`: they are contiguous and start on their size.
__device__ __forceinline__ float4 load_upto4(const float* p, long long stride, int left, bool vec) {
  if (left >= 4 && vec) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(left > 0 ? __ldg(p) : 0.f, left > 1 ? __ldg(p + stride) : 0.f, left > 2 ? __ldg(p + 2 * stride) : 0.f,
                     left > 3 ? __ldg(p + 3 * stride) : 0.f);
}
// Fragments of 8 * F rows (of A; columns of B) and sixteen k: v[i][s] is this lane's element of fragment i in step s.  Lane (fr,
// fk) stands for k = k0 + 4 fk + s and, with the contraction contiguous (KM), for row i * 8 + fr, else for row fr * F + i.
template <int F, bool KM>
__device__ __forceinline__ void load_fragments(float (&v)[F][4], const float* base, long long row_stride, long long k_stride, int row0,
                                               int rows, int k0, int k_end, bool vec) {
  const int lane = threadIdx.x & 31, fr = lane >> 2, k = k0 + 4 * (lane & 3);
  if constexpr (KM) {
#pragma unroll
    for (int i = 0; i < F; ++i) {
      const int row = row0 + i * 8 + fr;
      const float4 t = load_upto4(base + row * row_stride + k, 1, row < rows ? k_end - k : 0, vec);
      v[i][0] = t.x; v[i][1] = t.y; v[i][2] = t.z; v[i][3] = t.w;
    }
  } else {
    const int row = row0 + fr * F;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int left = k + s < k_end ? rows - row : 0;
      const float* p = base + row * row_stride + (k + s) * k_stride;
      if constexpr (F == 4) {
        const float4 t = load_upto4(p, row_stride, left, vec);
        v[0][s] = t.x; v[1][s] = t.y; v[2][s] = t.z; v[3][s] = t.w;
      } else {
        static_assert(F == 2, "two or four fragments");
        float2 t;
        if (left >= 2 && vec) t = __ldg(reinterpret_cast<const float2*>(p));
        else t = make_float2(left > 0 ? __ldg(p) : 0.f, left > 1 ? __ldg(p + row_stride) : 0.f);
        v[0][s] = t.x; v[1][s] = t.y;
      }
    }
  }
}

// The 32 x 32 tile: this warp's sums over its group's k, to the group's place in shared memory.
template <bool A_KM, bool B_KM>
__device__ __forceinline__ void f64_small_sums(const F64Gemm& g, double* smem, int row0, int col0, int kt0, int kt1, bool sums) {
  using Z = F64Tile<32, 32>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int group = warp >> 1, wn = (warp & 1) * 16;
  // one index contiguous, strides along the other that keep sixteen bytes
  const bool vec_a = (A_KM || g.a_row == 1) && ((A_KM ? g.a_row : g.a_col) & 3) == 0 && (reinterpret_cast<uintptr_t>(g.a) & 15) == 0;
  const bool vec_b = (B_KM || g.b_col == 1) && ((B_KM ? g.b_col : g.b_row) & 3) == 0 && (reinterpret_cast<uintptr_t>(g.b) & 15) == 0;
  double acc[4][2][2], rs[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    rs[i] = 0.0;
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  }
  const int k_end = min(g.k, kt1 * F64_BK);
  for (int kt = kt0 + group; kt < kt1; kt += Z::WK) {
    float a[2][4][4], b[2][2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      load_fragments<4, A_KM>(a[h], g.a, g.a_row, g.a_col, row0, g.m, kt * F64_BK + h * 16, k_end, vec_a);
      load_fragments<2, B_KM>(b[h], g.b, g.b_col, g.b_row, col0 + wn, g.n, kt * F64_BK + h * 16, k_end, vec_b);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const double b0 = (double)b[h][0][s], b1 = (double)b[h][1][s];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double av = (double)a[h][i][s];
          dmma(acc[i][0], av, b0);
          dmma(acc[i][1], av, b1);
          if (sums) rs[i] += av;  // row sums of A: a bias gradient rides on its weight gradient
        }
      }
  }
  double* sc = smem + group * Z::PART;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = A_KM ? i * 8 + fr : fr * 4 + i;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) sc[row * Z::LDC + wn + (B_KM ? j * 8 + 2 * fk + e : (2 * fk + e) * 2 + j)] = acc[i][j][e];
    if (sums && wn == 0) {
      double t = rs[i];
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      if (fk == 0) sc[32 * Z::LDC + row] = t;
    }
  }
}

template <int TM, int TN>
__global__ void __launch_bounds__(F64_THREADS, 2)
f64_gemm_kernel(const F64Jobs jobs) {
  pdl_begin();
  using Z = F64Tile<TM, TN>;
  extern __shared__ double f64_smem[];
  const int which = (jobs.count > 1 && (int)blockIdx.x >= jobs.job[1].cta0) ? 1 : 0;
  const F64Job& jb = jobs.job[which];
  const F64Gemm& g = jb.g;
  const int local = (int)blockIdx.x - jb.cta0;
  const int tile = jb.split > 1 ? local / jb.split : local;
  const int rank = jb.split > 1 ? local % jb.split : 0;
  if (tile >= jb.tiles) return;
  const int tid = threadIdx.x;
  const int row0 = (tile / jb.tiles_n) * TM, col0 = (tile % jb.tiles_n) * TN;
  const int kt0 = rank * jb.k_tiles_per_rank, kt1 = max(kt0, min((g.k + F64_BK - 1) / F64_BK, kt0 + jb.k_tiles_per_rank));
  const bool sums = g.row_sum != nullptr && col0 == 0;
  if constexpr (TM == 32) {
    if (g.a_col == 1) {
      if (g.b_row == 1) f64_small_sums<true, true>(g, f64_smem, row0, col0, kt0, kt1, sums);
      else f64_small_sums<true, false>(g, f64_smem, row0, col0, kt0, kt1, sums);
    } else {
      if (g.b_row == 1) f64_small_sums<false, true>(g, f64_smem, row0, col0, kt0, kt1, sums);
      else f64_small_sums<false, false>(g, f64_smem, row0, col0, kt0, kt1, sums);
    }
  } else if (g.a_col == 1) {
    if (g.b_row == 1) f64_tile_sums<TM, TN, true, true>(g, f64_smem, row0, col0, kt0, kt1, sums);
    else f64_tile_sums<TM, TN, true, false>(g, f64_smem, row0, col0, kt0, kt1, sums);
  } else {
    if (g.b_row == 1) f64_tile_sums<TM, TN, false, true>(g, f64_smem, row0, col0, kt0, kt1, sums);
    else f64_tile_sums<TM, TN, false, false>(g, f64_smem, row0, col0, kt0, kt1, sums);
  }
  const int parts = jb.split;
  cg::cluster_group cluster = cg::this_cluster();
  __syncthreads();
  auto groups = [&](int at) {  // the sums of this CTA's groups of warps, in order
    double v = f64_smem[at];
#pragma unroll
    for (int w = 1; w < Z::WK; ++w) v += f64_smem[w * Z::PART + at];
    return v;
  };
  if (parts > 1) {
    if (Z::WK > 1)  // added up before the other CTAs of the cluster read them
      for (int at = tid; at < Z::PART; at += F64_THREADS) f64_smem[at] = groups(at);
    cluster.sync();
  }
  auto total = [&](int at) {  // over the CTAs of the cluster, in order
    if (parts == 1) return groups(at);
    double v = 0.0;
    for (int p = 0; p < parts; ++p) v += *cluster.map_shared_rank(f64_smem + at, p);
    return v;
  };
  for (int e = rank * F64_THREADS + tid; e < TM * TN; e += parts * F64_THREADS) {
    const int r = e / TN, c = e % TN;
    const int row = row0 + r, col = col0 + c;
    if (row >= g.m || col >= g.n) continue;
    const double v = total(r * Z::LDC + c);
    const long long at = row * g.o_row + col * g.o_col;
    float y = g.epilogue == F64_ACCUMULATE ? (float)((double)g.out[at] + v) : (float)v;
    if (g.bias) y = y + __ldg(g.bias + col);
    if (g.epilogue == F64_GELU) g.aux_out[at] = (float)gelu_fwd<double>((double)y);
    else if (g.epilogue == F64_RESIDUAL) y = g.aux_in[at] + y;
    else if (g.epilogue == F64_DGELU) y = (float)((double)y * gelu_grad<double>((double)g.aux_in[at]));
    g.out[at] = y;
  }
  if (sums && rank == 0 && tid < TM && row0 + tid < g.m) g.row_sum[row0 + tid] = (float)total(TM * Z::LDC + tid);
  if (parts > 1) tc05::cluster_meet();  // no CTA leaves while another still reads its part
}

template <int TM, int TN>
int launch_f64_gemm(hl_ctx* ctx, const F64Gemm* problems, int count) {
  constexpr size_t smem = F64Tile<TM, TN>::SMEM;
  auto kern = f64_gemm_kernel<TM, TN>;
  HL_ALLOW_SHARED(ctx, smem, kern);
  F64Jobs jobs{};
  jobs.count = count;
  // A contraction longer than 256 is shared as long as its tiles leave SMs idle; eight CTAs is the largest portable cluster.
  int want[F64_JOBS];
  jobs.cluster = 1;
  for (int i = 0; i < count; ++i) {
    F64Job& j = jobs.job[i];
    j.g = problems[i];
    j.tiles_n = ceil_div(j.g.n, TN);
    j.tiles = ceil_div(j.g.m, TM) * j.tiles_n;
    want[i] = 1;
    while (want[i] < 8 && ceil_div(j.g.k, F64_BK) > 8 * want[i] && (long long)j.tiles * want[i] < 2 * ctx->sm_count) want[i] *= 2;
    jobs.cluster = std::max(jobs.cluster, want[i]);
  }
  long long ctas = 0;
  for (int i = 0; i < count; ++i) {
    F64Job& j = jobs.job[i];
    j.cta0 = (int)ctas;
    j.split = want[i] > 1 ? jobs.cluster : 1;
    j.k_tiles_per_rank = ceil_div(ceil_div(j.g.k, F64_BK), j.split);
    ctas += j.split > 1 ? (long long)j.tiles * j.split : ceil_div_ll(j.tiles, jobs.cluster) * jobs.cluster;
  }
  HL_REQUIRE(ctas <= 0x7fffffffLL, "hl_matmul_f32_strided: too many tiles for one launch");
  HL_CUDA(launch_pdl(kern, (unsigned)ctas, F64_THREADS, smem, ctx->stream, jobs.cluster, jobs));
  count_launch(ctx);
  return HL_OK;
}

// ---- causal attention ------------------------------------------------------------------------------
// q, k, v, out: rows of [B*T, *] with heads interleaved along the channels (column h*hd + j, as
// src/tensor.rs:5156-5177) and a row stride each, f32 or bf16 (widened exactly).  probs: [B,H,T,T].
//
// One CTA of eight warps per 16 query rows of one (batch, head); the rows' scores against every visible key stay in shared
// memory as f64, so each score is formed once (a lane per key walking the channels formed it three times, from
// uncoalesced rows).  Bound by latency: a few thousand multiply-adds a CTA behind global loads, reductions and f64 exponentials.
// So everything a CTA reads is requested at once and stays (`resident`, wherever keys and values fit: T 128 up to 80
// channels), the rows of a warp go through the softmax side by side, and every warp has several chains of products.
// B16 H4 T64 hd32, one after the other as a user calls them: forward 76 us at first, then 9 with the keys in tiles of 32 behind
// two barriers each.
constexpr int AT_WARPS = 8;
constexpr int AT_THREADS = AT_WARPS * 32;
constexpr int AT_Q = 16;   // query rows (or key rows) per CTA
constexpr int AT_K = 32;   // keys (or queries) per tile where they do not all fit
constexpr int AT_UNITS = 4;   // (8 channels, 8 rows) units per warp and pass: 128 channels at a time
constexpr int AT_ROWS = AT_Q / AT_WARPS;  // rows of a warp in the softmax

__host__ __device__ inline int at_ld(int n) { return (n + 15) / 16 * 16 + 4; }  // 4 mod 16 doubles: conflict-free fragments

__device__ __forceinline__ void at_widen4(const float* p, double (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void at_widen4(const __nv_bfloat16* p, double (&v)[4]) {
  const uint2 t = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16x2(t.x), b = unpack_bf16x2(t.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// rows [r0, r0 + rows) of a head's [T, hd] slice, widened, zero past T.  Columns past hd are left alone: they only reach results
// that are not stored.  Four elements a load where rows allow it, several loads in flight.
template <typename T>
__device__ __forceinline__ void at_load(double* dst, int ld, const T* src, long long ld_src, int r0, int rows, int T_, int hd) {
  if (hd % 4 == 0 && ld_src % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & (4 * sizeof(T) - 1)) == 0) {
    const int pieces = hd / 4, dr = AT_THREADS / pieces, dc = AT_THREADS % pieces;
    int r = (int)threadIdx.x / pieces, c = (int)threadIdx.x % pieces;
    while (r < rows) {
      double v[4][4];
      int at[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        at[u] = r < rows ? r * ld + c * 4 : -1;
        if (r < rows && r0 + r < T_) {
          at_widen4(src + (long long)(r0 + r) * ld_src + c * 4, v[u]);
        } else {
          v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.0;
        }
        r += dr;
        c += dc;
        if (c >= pieces) { c -= pieces; ++r; }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (at[u] >= 0) {
          *reinterpret_cast<double2*>(dst + at[u]) = make_double2(v[u][0], v[u][1]);
          *reinterpret_cast<double2*>(dst + at[u] + 2) = make_double2(v[u][2], v[u][3]);
        }
    }
    return;
  }
  const int width = (hd + 3) / 4 * 4;  // the contraction goes in steps of four channels
  for (int e = threadIdx.x; e < rows * width; e += AT_THREADS) {
    const int r = e / width, c = e % width;
    dst[r * ld + c] = (r0 + r < T_ && c < hd) ? widen(src[(long long)(r0 + r) * ld_src + c]) : 0.0;
  }
}

// S[16][keys] = scale * X · Yᵀ over the keys [0, n_keys): X in sx, Y in sy, all of it or (not resident) through it in tiles
template <typename T>
__device__ __forceinline__ void at_scores(double* ss, int ld_s, const double* sx, double* sy, int ld, const T* y,
                                          long long ld_y, int n_keys, int T_, int hd, double scale, bool resident) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int tile = resident ? n_keys : AT_K;
  for (int key0 = 0; key0 < n_keys; key0 += tile) {
    if (!resident) {
      __syncthreads();
      at_load(sy, ld, y, ld_y, key0, AT_K, T_, hd);
      __syncthreads();
    }
    for (int k8 = warp * 8; k8 < tile; k8 += AT_WARPS * 8) {
      double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      const double* pa = sx + fr * ld + fk;
      const double* pb = sy + (k8 + fr) * ld + fk;
#pragma unroll 4
      for (int c = 0; c < hd; c += 4) {
        const double b = pb[c];
        dmma(acc[0], pa[c], b);
        dmma(acc[1], pa[8 * ld + c], b);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        double* d = ss + (i * 8 + fr) * ld_s + key0 + k8 + 2 * fk;
        d[0] = acc[i][0] * scale;
        d[1] = acc[i][1] * scale;
      }
    }
  }
  __syncthreads();
}

// out rows = W[16][n_keys] · Y: W in sw (f64), Y in sy as above
template <typename T, typename OT>
__device__ __forceinline__ void at_weighted(const double* sw, int ld_s, double* sy, int ld, const T* y, long long ld_y,
                                            OT* out, long long ld_out, int t0, int n_keys, int T_, int hd, bool resident) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int units = (hd + 7) / 8 * 2;  // unit: 8 channels (u / 2) of 8 rows (u % 2)
  const int tile = resident ? n_keys : AT_K;
  for (int u0 = 0; u0 < units; u0 += AT_WARPS * AT_UNITS) {
    double acc[AT_UNITS][2][2];  // even and odd steps apart
#pragma unroll
    for (int i = 0; i < AT_UNITS; ++i) acc[i][0][0] = acc[i][0][1] = acc[i][1][0] = acc[i][1][1] = 0.0;
    for (int key0 = 0; key0 < n_keys; key0 += tile) {
      __syncthreads();  // W is complete, and nothing reads the last tile any more
      if (!resident) {
        at_load(sy, ld, y, ld_y, key0, AT_K, T_, hd);
        __syncthreads();
      }
      for (int kk = 0; kk < tile; kk += 8) {
#pragma unroll
        for (int i = 0; i < AT_UNITS; ++i) {
          const int u = u0 + i * AT_WARPS + warp;
          if (u < units) {
            const double* pa = sw + ((u & 1) * 8 + fr) * ld_s + key0 + kk + fk;
            const double* pb = sy + (kk + fk) * ld + (u >> 1) * 8 + fr;
            dmma(acc[i][0], pa[0], pb[0]);
            dmma(acc[i][1], pa[4], pb[4 * ld]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < AT_UNITS; ++i) {
      const int u = u0 + i * AT_WARPS + warp, t = t0 + (u & 1) * 8 + fr, c = (u >> 1) * 8 + 2 * fk;
      if (u < units && t < T_) {
        if (c < hd) narrow(out + (long long)t * ld_out + c, acc[i][0][0] + acc[i][1][0]);
        if (c + 1 < hd) narrow(out + (long long)t * ld_out + c + 1, acc[i][0][1] + acc[i][1][1]);
      }
    }
  }
}

// softmax of the visible part of each row, rounded to f32: into probs (zero past the diagonal), into ss and, when given, into
// sp[16][n_keys].  A warp's rows side by side.
__device__ __forceinline__ void at_softmax(double* ss, int ld_s, float* sp, float* probs, int t0, int n_keys, int T_) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int last = min(t0 + AT_Q, T_);
  double mx[AT_ROWS], sum[AT_ROWS];
#pragma unroll
  for (int i = 0; i < AT_ROWS; ++i) mx[i] = -INFINITY;
  for (int s = lane; s < last; s += 32)
#pragma unroll
    for (int i = 0; i < AT_ROWS; ++i) {
      const int r = i * AT_WARPS + warp;
      if (s <= t0 + r) mx[i] = max(mx[i], ss[r * ld_s + s]);
    }
#pragma unroll
  for (int i = 0; i < AT_ROWS; ++i) mx[i] = warp_max(mx[i]);
#pragma unroll
  for (int i = 0; i < AT_ROWS; ++i) sum[i] = 0.0;
  for (int s = lane; s < last; s += 32)
#pragma unroll
    for (int i = 0; i < AT_ROWS; ++i) {
      const int r = i * AT_WARPS + warp;
      if (s <= t0 + r) {
        const double e = exp(ss[r * ld_s + s] - mx[i]);
        ss[r * ld_s + s] = e;
        sum[i] += e;
      }
    }
#pragma unroll
  for (int i = 0; i < AT_ROWS; ++i) sum[i] = warp_sum(sum[i]);
  for (int s = lane; s < max(n_keys, T_); s += 32)
#pragma unroll
    for (int i = 0; i < AT_ROWS; ++i) {
      const int r = i * AT_WARPS + warp, t = t0 + r;  // rows past T: multiplied as zeros, never stored
      const float p = s <= t && t < T_ ? (float)(ss[r * ld_s + s] / sum[i]) : 0.f;
      if (s < n_keys) {
        ss[r * ld_s + s] = (double)p;
        if (sp) sp[r * n_keys + s] = p;
      }
      if (s < T_ && t < T_) probs[(size_t)t * T_ + s] = p;
    }
}

template <typename T>
__global__ void __launch_bounds__(AT_THREADS)
attention_f64_fwd_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long ld_qkv,
                         T* __restrict__ out, long long ld_out, float* __restrict__ probs, int T_, int H, int hd, unsigned heads,
                         bool resident) {
  pdl_begin();
  extern __shared__ double at_smem[];
  const int step = resident ? 8 : AT_K, padded = (T_ + step - 1) / step * step;
  const int ld = at_ld(hd), ld_s = at_ld(padded);
  double *sx = at_smem, *ss = sx + AT_Q * ld, *sk = ss + AT_Q * ld_s, *sv = resident ? sk + (size_t)padded * ld : sk;
  const int bh = (int)(blockIdx.x % heads), h = bh % H, b = bh / H;
  const int t0 = ((T_ - 1) / AT_Q - (int)(blockIdx.x / heads)) * AT_Q;  // the longest rows first
  const int n_keys = (min(T_, t0 + AT_Q) + step - 1) / step * step;
  const long long head = (long long)b * T_ * ld_qkv + (long long)h * hd;
  at_load(sx, ld, q + head, ld_qkv, t0, AT_Q, T_, hd);
  if (resident) {
    at_load(sk, ld, k + head, ld_qkv, 0, n_keys, T_, hd);
    at_load(sv, ld, v + head, ld_qkv, 0, n_keys, T_, hd);
    __syncthreads();
  }
  at_scores(ss, ld_s, sx, sk, ld, k + head, ld_qkv, n_keys, T_, hd, 1.0 / sqrt((double)hd), resident);
  at_softmax(ss, ld_s, nullptr, probs + (size_t)bh * T_ * T_, t0, n_keys, T_);
  at_weighted(ss, ld_s, sv, ld, v + head, ld_qkv, out + (long long)b * T_ * ld_out + (long long)h * hd, ld_out, t0, n_keys, T_, hd,
              resident);
}

// Per 16 query rows: (the probabilities again, when they were not kept,) dP, dS (to the f32 scratch) and dQ.
template <typename T, bool RECOMPUTE>
__global__ void __launch_bounds__(AT_THREADS)
attention_f64_bwd_rows_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long ld_qkv,
                              float* __restrict__ probs, const T* __restrict__ dout, long long ld_dout,
                              float* __restrict__ ds, T* __restrict__ dq, long long ld_dqkv, int T_, int H, int hd, unsigned heads,
                              bool resident) {
  pdl_begin();
  extern __shared__ double at_smem[];
  const int step = resident ? 8 : AT_K, padded = (T_ + step - 1) / step * step;
  const int ld = at_ld(hd), ld_s = at_ld(padded);
  double *sx = at_smem, *sg = sx + AT_Q * ld, *ss = sg + AT_Q * ld, *sk = ss + AT_Q * ld_s;
  double* sv = resident ? sk + (size_t)padded * ld : sk;
  // [16][n_keys] probabilities; where shared memory is short they are read from (or back from) memory, by the lanes that wrote them
  float* sp = resident ? reinterpret_cast<float*>(sv + (size_t)padded * ld) : nullptr;
  const int bh = (int)(blockIdx.x % heads), h = bh % H, b = bh / H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = ((T_ - 1) / AT_Q - (int)(blockIdx.x / heads)) * AT_Q;
  const int n_keys = (min(T_, t0 + AT_Q) + step - 1) / step * step;
  const long long head = (long long)b * T_ * ld_qkv + (long long)h * hd;
  const double scale = 1.0 / sqrt((double)hd);
  float* pb = probs + (size_t)bh * T_ * T_;
  float* db = ds + (size_t)bh * T_ * T_;
  if constexpr (RECOMPUTE) {
    at_load(sx, ld, q + head, ld_qkv, t0, AT_Q, T_, hd);
  } else if (resident) {
    for (int e = threadIdx.x; e < AT_Q * n_keys; e += AT_THREADS) {
      const int r = e / n_keys, s = e % n_keys;
      sp[e] = t0 + r < T_ && s <= t0 + r ? pb[(size_t)(t0 + r) * T_ + s] : 0.f;
    }
  }
  at_load(sg, ld, dout + (long long)b * T_ * ld_dout + (long long)h * hd, ld_dout, t0, AT_Q, T_, hd);
  if (resident) {
    at_load(sk, ld, k + head, ld_qkv, 0, n_keys, T_, hd);
    at_load(sv, ld, v + head, ld_qkv, 0, n_keys, T_, hd);
    __syncthreads();
  }
  if constexpr (RECOMPUTE) {
    at_scores(ss, ld_s, sx, sk, ld, k + head, ld_qkv, n_keys, T_, hd, scale, resident);
    at_softmax(ss, ld_s, sp, pb, t0, n_keys, T_);
    __syncthreads();  // ss is written again
  }
  at_scores(ss, ld_s, sg, sv, ld, v + head, ld_qkv, n_keys, T_, hd, 1.0, resident);  // dP
  auto prob = [&](int r, int s) {  // s <= t0 + r
    return resident ? sp[r * n_keys + s] : t0 + r < T_ ? pb[(size_t)(t0 + r) * T_ + s] : 0.f;
  };
  double dot[AT_ROWS];
#pragma unroll
  for (int i = 0; i < AT_ROWS; ++i) dot[i] = 0.0;
  for (int s = lane; s < n_keys; s += 32)
#pragma unroll
    for (int i = 0; i < AT_ROWS; ++i) {
      const int r = i * AT_WARPS + warp;
      if (s <= t0 + r) dot[i] += ss[r * ld_s + s] * (double)prob(r, s);
    }
#pragma unroll
  for (int i = 0; i < AT_ROWS; ++i) dot[i] = warp_sum(dot[i]);
  for (int s = lane; s < n_keys; s += 32)  // the column pass reads no further than this row's last tile
#pragma unroll
    for (int i = 0; i < AT_ROWS; ++i) {
      const int r = i * AT_WARPS + warp, t = t0 + r;
      const float d = s <= t && t < T_ ? (float)((double)prob(r, s) * (ss[r * ld_s + s] - dot[i]) * scale) : 0.f;
      ss[r * ld_s + s] = (double)d;
      if (s < T_ && t < T_) db[(size_t)t * T_ + s] = d;
    }
  at_weighted(ss, ld_s, sk, ld, k + head, ld_qkv, dq + (long long)b * T_ * ld_dqkv + (long long)h * hd, ld_dqkv, t0, n_keys, T_, hd,
              resident);
}

// Per 16 key rows: dK[s] = sum_{t>=s} dS[t,s] Q[t], dV[s] = sum_{t>=s} P[t,s] dO[t]; fixed order.  The queries go through shared
// memory `tile` at a time, all of them at once where they fit.
template <typename T>
__global__ void __launch_bounds__(AT_THREADS)
attention_f64_bwd_cols_kernel(const T* __restrict__ q, long long ld_qkv, const float* __restrict__ probs,
                              const float* __restrict__ ds, const T* __restrict__ dout, long long ld_dout,
                              T* __restrict__ dk, T* __restrict__ dv, long long ld_dqkv, int T_, int H, int hd, unsigned heads,
                              int tile) {
  pdl_begin();
  extern __shared__ double at_smem[];
  constexpr int CH = AT_WARPS * AT_UNITS / 2 * 8;  // channels of one pass
  const int ld = at_ld(min(hd, CH));
  constexpr int LDW = AT_Q + 4;
  double *sq = at_smem, *sdo = sq + (size_t)tile * ld, *swd = sdo + (size_t)tile * ld, *swp = swd + tile * LDW;
  const int bh = (int)(blockIdx.x % heads), h = bh % H, b = bh / H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fk = lane & 3;
  const int s0 = (int)(blockIdx.x / heads) * AT_Q;
  const float* pb = probs + (size_t)bh * T_ * T_;
  const float* db = ds + (size_t)bh * T_ * T_;
  const T* qh = q + (long long)b * T_ * ld_qkv + (long long)h * hd;
  const T* gh = dout + (long long)b * T_ * ld_dout + (long long)h * hd;
  for (int c0 = 0; c0 < hd; c0 += CH) {
    const int width = min(hd - c0, CH), units = (width + 7) / 8 * 2;  // unit: 8 channels (u / 2) of 8 key rows (u % 2)
    double ak[AT_UNITS][2][2], av[AT_UNITS][2][2];  // even and odd steps apart
#pragma unroll
    for (int i = 0; i < AT_UNITS; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) ak[i][j][0] = ak[i][j][1] = av[i][j][0] = av[i][j][1] = 0.0;
    for (int t0 = s0 / AT_K * AT_K; t0 < T_; t0 += tile) {
      const int rows = min(tile, (T_ - t0 + 7) / 8 * 8);
      __syncthreads();
      for (int e = threadIdx.x; e < rows * AT_Q; e += AT_THREADS) {
        const int r = e / AT_Q, c = e % AT_Q;
        const bool in = t0 + r < T_ && s0 + c <= t0 + r;
        const size_t at = (size_t)(t0 + r) * T_ + s0 + c;
        swd[r * LDW + c] = in ? (double)db[at] : 0.0;
        swp[r * LDW + c] = in ? (double)pb[at] : 0.0;
      }
      at_load(sq, ld, qh + c0, ld_qkv, t0, rows, T_, width);
      at_load(sdo, ld, gh + c0, ld_dout, t0, rows, T_, width);
      __syncthreads();
      for (int kk = 0; kk < rows; kk += 8) {
#pragma unroll
        for (int i = 0; i < AT_UNITS; ++i) {
          const int u = i * AT_WARPS + warp;
          if (u < units) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int r = kk + j * 4 + fk, w = r * LDW + (u & 1) * 8 + fr, x = r * ld + (u >> 1) * 8 + fr;
              dmma(ak[i][j], swd[w], sq[x]);
              dmma(av[i][j], swp[w], sdo[x]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < AT_UNITS; ++i) {
      const int u = i * AT_WARPS + warp, s = s0 + (u & 1) * 8 + fr, c = (u >> 1) * 8 + 2 * fk;
      if (u < units && s < T_) {
        const long long at = ((long long)b * T_ + s) * ld_dqkv + (long long)h * hd + c0 + c;
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (c + e < width) {
            narrow(dk + at + e, ak[i][0][e] + ak[i][1][e]);
            narrow(dv + at + e, av[i][0][e] + av[i][1][e]);
          }
      }
    }
  }
}

// ---- the same for rows or heads whose scores do not fit in shared memory (T above about 1500): a warp per row ----------
template <typename T>
__global__ void attention_f64_fwd_rows_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                                              long long ld_qkv, T* __restrict__ out, long long ld_out,
                                              float* __restrict__ probs, int B, int T_, int H, int hd) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const long long w = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= (long long)B * H * T_) return;
  const int t = (int)(w % T_), h = (int)((w / T_) % H), b = (int)(w / ((long long)T_ * H));
  const double scale = 1.0 / sqrt((double)hd);
  const long long head = (long long)b * T_ * ld_qkv + (long long)h * hd;
  const T* qr = q + head + (long long)t * ld_qkv;
  float* pr = probs + (((size_t)b * H + h) * T_ + t) * (size_t)T_;
  auto score = [&](int s) {
    const T* kr = k + head + (long long)s * ld_qkv;
    double dot = 0.0;
    for (int j = 0; j < hd; ++j) dot += widen(qr[j]) * widen(kr[j]);
    return dot * scale;
  };
  double mx = -INFINITY;
  for (int s = lane; s <= t; s += 32) mx = max(mx, score(s));
  mx = warp_max(mx);
  double denom = 0.0;
  for (int s = lane; s <= t; s += 32) denom += exp(score(s) - mx);
  denom = warp_sum(denom);
  for (int s = lane; s < T_; s += 32) pr[s] = s <= t ? (float)(exp(score(s) - mx) / denom) : 0.f;
  __syncwarp();
  T* orow = out + ((long long)b * T_ + t) * ld_out + (long long)h * hd;
  for (int j = lane; j < hd; j += 32) {
    double acc = 0.0;
    for (int s = 0; s <= t; ++s) acc += (double)pr[s] * widen(v[head + (long long)s * ld_qkv + j]);
    narrow(orow + j, acc);
  }
}

template <typename T>
__global__ void attention_f64_bwd_long_rows_kernel(const T* __restrict__ k, const T* __restrict__ v, long long ld_qkv,
                                                   const float* __restrict__ probs, const T* __restrict__ dout,
                                                   long long ld_dout, float* __restrict__ ds, T* __restrict__ dq,
                                                   long long ld_dqkv, int B, int T_, int H, int hd) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const long long w = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= (long long)B * H * T_) return;
  const int t = (int)(w % T_), h = (int)((w / T_) % H), b = (int)(w / ((long long)T_ * H));
  const double scale = 1.0 / sqrt((double)hd);
  const long long head = (long long)b * T_ * ld_qkv + (long long)h * hd;
  const float* pr = probs + (((size_t)b * H + h) * T_ + t) * (size_t)T_;
  float* dsr = ds + (((size_t)b * H + h) * T_ + t) * (size_t)T_;
  const T* gor = dout + ((long long)b * T_ + t) * ld_dout + (long long)h * hd;
  auto dp_of = [&](int s) {
    const T* vr = v + head + (long long)s * ld_qkv;
    double dp = 0.0;
    for (int j = 0; j < hd; ++j) dp += widen(gor[j]) * widen(vr[j]);
    return dp;
  };
  double dot_sum = 0.0;
  for (int s = lane; s <= t; s += 32) dot_sum += dp_of(s) * (double)pr[s];
  dot_sum = warp_sum(dot_sum);
  for (int s = lane; s < T_; s += 32) dsr[s] = s <= t ? (float)((double)pr[s] * (dp_of(s) - dot_sum) * scale) : 0.f;
  __syncwarp();
  T* dqr = dq + ((long long)b * T_ + t) * ld_dqkv + (long long)h * hd;
  for (int j = lane; j < hd; j += 32) {
    double acc = 0.0;
    for (int s = 0; s <= t; ++s) acc += (double)dsr[s] * widen(k[head + (long long)s * ld_qkv + j]);
    narrow(dqr + j, acc);
  }
}

constexpr size_t kAttentionSmem = 227 * 1024;
// A row kernel's shared memory; `resident`: keys and values of the whole head in it.
size_t at_rows_smem(int T, int hd, bool backward, bool resident) {
  const int step = resident ? 8 : AT_K, padded = ceil_div(T, step) * step;
  return sizeof(double) * ((size_t)((backward ? 2 : 1) * AT_Q + (resident ? 2 * padded : AT_K)) * at_ld(hd) + (size_t)AT_Q * at_ld(padded)) +
         (backward && resident ? sizeof(float) * AT_Q * (size_t)padded : 0);
}
// Queries that the column kernel holds at a time, a multiple of eight: all of them, or what leaves room for two CTAs an SM.
int at_cols_tile(int T, int hd, size_t* smem) {
  const size_t row = sizeof(double) * (2 * (size_t)at_ld(std::min(hd, AT_WARPS * AT_UNITS / 2 * 8)) + 2 * (AT_Q + 4));
  const int most = std::max(AT_K, (int)(112 * 1024 / row) / 8 * 8);
  const int tile = std::min(ceil_div(T, 8) * 8, most);
  *smem = row * tile;
  return tile;
}

template <typename T>
int attention_forward_t(hl_ctx* ctx, const T* q, const T* k, const T* v, long long ld_qkv, T* out, long long ld_out,
                        float* probs, int B, int Tn, int C, int H) {
  const int hd = C / H;
  const bool resident = at_rows_smem(Tn, hd, false, true) <= kAttentionSmem;
  const size_t smem = at_rows_smem(Tn, hd, false, resident);
  const long long heads = (long long)B * H;
  if (smem <= kAttentionSmem) {
    HL_ALLOW_SHARED(ctx, kAttentionSmem, attention_f64_fwd_kernel<T>);
    pdl(attention_f64_fwd_kernel<T>, (unsigned)(ceil_div(Tn, AT_Q) * heads), AT_THREADS, smem, ctx->stream)(
        q, k, v, ld_qkv, out, ld_out, probs, Tn, H, hd, (unsigned)heads, resident);
    HL_LAUNCH_CHECK("attention_f64_fwd_kernel");
  } else {
    pdl(attention_f64_fwd_rows_kernel<T>, (unsigned)ceil_div_ll(heads * Tn, 4), 128, 0, ctx->stream)(q, k, v, ld_qkv, out, ld_out,
                                                                                                    probs, B, Tn, H, hd);
    HL_LAUNCH_CHECK("attention_f64_fwd_rows_kernel");
  }
  count_launch(ctx);
  return HL_OK;
}

template <typename T, bool RECOMPUTE>
int attention_backward_t(hl_ctx* ctx, const T* q, const T* k, const T* v, long long ld_qkv, float* probs, const T* dout,
                         long long ld_dout, T* dq, T* dk, T* dv, long long ld_dqkv, int B, int Tn, int C, int H) {
  const int hd = C / H;
  const long long heads = (long long)B * H;
  int rc = ensure_workspace(ctx, sizeof(float) * (size_t)heads * Tn * Tn);
  if (rc != HL_OK) return rc;
  float* ds = reinterpret_cast<float*>(ctx->workspace);
  const bool resident = at_rows_smem(Tn, hd, true, true) <= kAttentionSmem;
  const size_t rows = at_rows_smem(Tn, hd, true, resident);
  size_t cols = 0;
  const int tile = at_cols_tile(Tn, hd, &cols);
  HL_ALLOW_SHARED(ctx, kAttentionSmem, attention_f64_bwd_rows_kernel<T, RECOMPUTE>);
  HL_ALLOW_SHARED(ctx, kAttentionSmem, attention_f64_bwd_cols_kernel<T>);
  if (rows <= kAttentionSmem) {
    pdl(attention_f64_bwd_rows_kernel<T, RECOMPUTE>, (unsigned)(ceil_div(Tn, AT_Q) * heads), AT_THREADS, rows, ctx->stream)(
        q, k, v, ld_qkv, probs, dout, ld_dout, ds, dq, ld_dqkv, Tn, H, hd, (unsigned)heads, resident);
    HL_LAUNCH_CHECK("attention_f64_bwd_rows_kernel");
  } else {
    if (RECOMPUTE) {  // the output goes where dQ will be written
      if ((rc = attention_forward_t<T>(ctx, q, k, v, ld_qkv, dq, ld_dqkv, probs, B, Tn, C, H)) != HL_OK) return rc;
    }
    pdl(attention_f64_bwd_long_rows_kernel<T>, (unsigned)ceil_div_ll(heads * Tn, 4), 128, 0, ctx->stream)(
        k, v, ld_qkv, probs, dout, ld_dout, ds, dq, ld_dqkv, B, Tn, H, hd);
    HL_LAUNCH_CHECK("attention_f64_bwd_long_rows_kernel");
  }
  pdl(attention_f64_bwd_cols_kernel<T>, (unsigned)(ceil_div(Tn, AT_Q) * heads), AT_THREADS, cols, ctx->stream)(
      q, ld_qkv, probs, ds, dout, ld_dout, dk, dv, ld_dqkv, Tn, H, hd, (unsigned)heads, tile);
  HL_LAUNCH_CHECK("attention_f64_bwd_cols_kernel");
  count_launch(ctx, 2);
  return HL_OK;
}

int check_attention_dims(int B, int T, int C, int H, const char* who) {
  HL_REQUIRE(H > 0, std::string(who) + ": causal_self_attention requires n_heads > 0");
  HL_REQUIRE(B > 0 && T > 0 && C > 0, std::string(who) + ": batch, time and channels must be positive");
  HL_REQUIRE(C % H == 0, std::string(who) + ": channels " + std::to_string(C) + " must be divisible by n_heads " +
                             std::to_string(H));
  return HL_OK;
}

}  // namespace

int f64_gemm_run(hl_ctx* ctx, const F64Gemm* problems, int count) {
  HL_REQUIRE(count >= 1 && count <= F64_JOBS, "f64_gemm_run: one or two products");
  long long tiles = 0;
  for (int i = 0; i < count; ++i) tiles += (long long)ceil_div(problems[i].m, 64) * ceil_div(problems[i].n, 64);
  // 64 x 64 tiles read half as much per multiply-add; below two per SM the smaller tile's parallelism is worth more
  return tiles >= 2LL * ctx->sm_count ? launch_f64_gemm<64, 64>(ctx, problems, count) : launch_f64_gemm<32, 32>(ctx, problems, count);
}

int attention_f64_forward(hl_ctx* ctx, const void* q, const void* k, const void* v, int dtype, long long ld_qkv, void* out,
                          long long ld_out, float* probs, int batch, int time, int channels, int n_heads) {
  if (dtype == HL_BF16)
    return attention_forward_t<__nv_bfloat16>(ctx, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v,
                                              ld_qkv, (__nv_bfloat16*)out, ld_out, probs, batch, time, channels, n_heads);
  return attention_forward_t<float>(ctx, (const float*)q, (const float*)k, (const float*)v, ld_qkv, (float*)out, ld_out, probs,
                                    batch, time, channels, n_heads);
}

int attention_f64_backward(hl_ctx* ctx, const void* q, const void* k, const void* v, int dtype, long long ld_qkv, float* probs,
                           const void* dout, long long ld_dout, void* dq, void* dk, void* dv, long long ld_dqkv, int batch,
                           int time, int channels, int n_heads) {
  if (dtype == HL_BF16)
    return attention_backward_t<__nv_bfloat16, true>(
        ctx, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, ld_qkv, probs, (const __nv_bfloat16*)dout,
        ld_dout, (__nv_bfloat16*)dq, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, ld_dqkv, batch, time, channels, n_heads);
  return attention_backward_t<float, false>(ctx, (const float*)q, (const float*)k, (const float*)v, ld_qkv, probs,
                                            (const float*)dout, ld_dout, (float*)dq, (float*)dk, (float*)dv, ld_dqkv, batch,
                                            time, channels, n_heads);
}

}  // namespace hl

using namespace hl;

extern "C" {

int hl_matmul_f32_strided(hl_ctx* ctx, const float* a, const hl_matrix_layout* la, const float* b,
                          const hl_matrix_layout* lb, float* out, const hl_matrix_layout* lo, int accumulate) {
  HL_REQUIRE(ctx && a && la && b && lb && out && lo, "hl_matmul_f32_strided: null argument");
  HL_REQUIRE(la->rows > 0 && la->cols > 0 && lb->cols > 0, "hl_matmul_f32_strided: empty operand");
  HL_REQUIRE(la->cols == lb->rows, "hl_matmul_f32_strided: inner dimensions differ (" + std::to_string(la->cols) +
                                       " vs " + std::to_string(lb->rows) + ")");
  HL_REQUIRE(lo->rows == la->rows && lo->cols == lb->cols, "hl_matmul_f32_strided: output shape mismatch");
  HL_REQUIRE(la->rows <= 0x7fffffc0LL && la->cols <= 0x7fffffc0LL && lb->cols <= 0x7fffffc0LL,
             "hl_matmul_f32_strided: too many rows for one launch");
  F64Gemm g{};
  g.a = a + la->offset; g.a_row = la->row_stride; g.a_col = la->col_stride;
  g.b = b + lb->offset; g.b_row = lb->row_stride; g.b_col = lb->col_stride;
  g.out = out + lo->offset; g.o_row = lo->row_stride; g.o_col = lo->col_stride;
  g.m = (int)la->rows; g.n = (int)lb->cols; g.k = (int)la->cols;
  g.epilogue = accumulate ? F64_ACCUMULATE : F64_STORE;
  return f64_gemm_run(ctx, &g, 1);
}

int hl_causal_attention_f32_forward(hl_ctx* ctx, const float* q, const float* k, const float* v, float* out,
                                    float* probs, int batch, int time, int channels, int n_heads) {
  HL_REQUIRE(ctx && q && k && v && out && probs, "hl_causal_attention_f32_forward: null argument");
  int rc = check_attention_dims(batch, time, channels, n_heads, "hl_causal_attention_f32_forward");
  if (rc != HL_OK) return rc;
  return attention_f64_forward(ctx, q, k, v, HL_F32, channels, out, channels, probs, batch, time, channels, n_heads);
}

int hl_causal_attention_f32_backward(hl_ctx* ctx, const float* q, const float* k, const float* v, const float* probs,
                                     const float* grad_out, float* dq, float* dk, float* dv, int batch, int time,
                                     int channels, int n_heads) {
  HL_REQUIRE(ctx && q && k && v && probs && grad_out && dq && dk && dv, "hl_causal_attention_f32_backward: null argument");
  int rc = check_attention_dims(batch, time, channels, n_heads, "hl_causal_attention_f32_backward");
  if (rc != HL_OK) return rc;
  return attention_f64_backward(ctx, q, k, v, HL_F32, channels, const_cast<float*>(probs), grad_out, channels, dq, dk, dv,
                                channels, batch, time, channels, n_heads);
}

}  // extern "C"
