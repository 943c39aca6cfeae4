// Product-key memory layer: side scores with the reference's exact f32 dot order, per-token
// top-k selection (ties to the lower index), differentiable re-scoring of the chosen slots,
// weighted value gather and its gradients, row-set AdamW.  One warp per token replaces the
// reference's one-thread-per-token serial selection (heirloom-kernels/src/ptx/kernels.ptx:1780-2262)
// and its one-thread-per-element gathers (:2317-3259); the O(selected^2) duplicate scan of the
// sparse AdamW kernels (:537-811) becomes a row flag pass.

#include "kernels.h"

namespace hl {
namespace {

constexpr float kNegInf = -INFINITY;

// ---- generic per-row top-k (src/tensor.rs:641-702): descending score, ties to the lower index ----
// One warp per row; k rounds of warp arg-max over the lane's strided elements, chosen entries are
// remembered in a per-lane bit set (cols <= 32*64).
__global__ void topk_rows_kernel(const float* __restrict__ scores, int64_t* __restrict__ out, int rows, int cols, int k) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const float* s = scores + (size_t)row * cols;
  unsigned long long taken = 0ull;  // bit i: element lane + 32*i already chosen
  for (int r = 0; r < k; ++r) {
    float best = kNegInf;
    int best_idx = 0x7fffffff;
    for (int i = 0, c = lane; c < cols; ++i, c += 32) {
      if ((taken >> i) & 1ull) continue;
      const float v = s[c];
      if (best_idx == 0x7fffffff || v > best) { best = v; best_idx = c; }  // strictly greater keeps the lower index
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_idx, o);
      if (oi != 0x7fffffff && (best_idx == 0x7fffffff || ov > best || (ov == best && oi < best_idx))) { best = ov; best_idx = oi; }
    }
    if (best_idx != 0x7fffffff && (best_idx & 31) == lane) taken |= 1ull << (best_idx >> 5);
    if (lane == 0) out[(size_t)row * k + r] = best_idx;
  }
}

// ---- side scores: out[t, s] = sum_j q[t, q_off + j] * keys[s, j], acc = acc + (q*k) in f32 with separately
// rounded multiply and add, j ascending (src/memory_transformer.rs:2029-2034) -------------------------
// Block tile 64 tokens x 128 keys, thread tile 8 tokens x 4 keys; the contraction walks in slices of 64 that are
// staged in shared memory (queries as [j][token], keys as [j][key]), so a step of the inner loop is three 16-byte
// shared-memory loads for 32 multiplies and 32 adds, two an instruction.  Every accumulator still sees j = 0, 1, 2, ... in
// order.  Bound by the multiplies and adds, which may not be fused: 118 us for 16384 x 512 x 256.
constexpr int SS_T = 64;   // tokens per block
constexpr int SS_K = 128;  // keys per block
constexpr int SS_J = 64;   // contraction slice
__global__ void __launch_bounds__(256)
side_scores_kernel(const float* __restrict__ query, long long ld_q, const float* __restrict__ left_keys,
                   const float* __restrict__ right_keys, float* __restrict__ left_out, float* __restrict__ right_out, int tokens,
                   int side, int half_dim, float minus_zero) {
  pdl_begin();
  const bool right = blockIdx.z == 1;
  const float* keys = right ? right_keys : left_keys;
  float* out = right ? right_out : left_out;
  const int q_off = right ? half_dim : 0;
  // A product is formed as q*k + (-0), which rounds like q*k alone.  The compiler fuses a packed multiply and add; it cannot
  // know this addend.
  const float2 zero = both(minus_zero);
  __shared__ __align__(16) float sq[SS_J][SS_T];
  __shared__ __align__(16) float sk[SS_J][SS_K];
  const int t0 = blockIdx.y * SS_T, k0 = blockIdx.x * SS_K;
  const int ty = threadIdx.x >> 5;  // 8 token groups of 8 tokens
  const int tx = threadIdx.x & 31;  // 32 key groups of 4 keys
  float2 acc[8][2];
#pragma unroll
  for (int a = 0; a < 8; ++a) acc[a][0] = acc[a][1] = both(0.f);
  // 16-byte loads need four-element granularity everywhere an address is formed
  const bool vec = (half_dim % 4) == 0 && (ld_q % 4) == 0 && (q_off % 4) == 0 &&
                   ((reinterpret_cast<uintptr_t>(query) | reinterpret_cast<uintptr_t>(keys)) & 15) == 0;
  for (int j0 = 0; j0 < half_dim; j0 += SS_J) {
    // stage the slice transposed.  Consecutive threads take consecutive rows, so the shared-memory stores of a warp
    // fall into 32 different banks; each thread brings four consecutive j of its row with one 16-byte load.
    if (vec) {
      for (int i = threadIdx.x; i < SS_T * (SS_J / 4); i += 256) {
        const int t = i % SS_T, j = (i / SS_T) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + t < tokens && j0 + j < half_dim)
          x = *reinterpret_cast<const float4*>(query + (size_t)(t0 + t) * ld_q + q_off + j0 + j);
        sq[j][t] = x.x; sq[j + 1][t] = x.y; sq[j + 2][t] = x.z; sq[j + 3][t] = x.w;
      }
      for (int i = threadIdx.x; i < SS_K * (SS_J / 4); i += 256) {
        const int kk = i % SS_K, j = (i / SS_K) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k0 + kk < side && j0 + j < half_dim)
          x = __ldg(reinterpret_cast<const float4*>(keys + (size_t)(k0 + kk) * half_dim + j0 + j));
        sk[j][kk] = x.x; sk[j + 1][kk] = x.y; sk[j + 2][kk] = x.z; sk[j + 3][kk] = x.w;
      }
    } else {
      for (int i = threadIdx.x; i < SS_T * SS_J; i += 256) {
        const int t = i % SS_T, j = i / SS_T;
        sq[j][t] = (t0 + t < tokens && j0 + j < half_dim) ? query[(size_t)(t0 + t) * ld_q + q_off + j0 + j] : 0.f;
      }
      for (int i = threadIdx.x; i < SS_K * SS_J; i += 256) {
        const int kk = i % SS_K, j = i / SS_K;
        sk[j][kk] = (k0 + kk < side && j0 + j < half_dim) ? keys[(size_t)(k0 + kk) * half_dim + j0 + j] : 0.f;
      }
    }
    __syncthreads();
    const int jn = min(SS_J, half_dim - j0);
    auto step = [&](int j) {
      const float4 qa = *reinterpret_cast<const float4*>(&sq[j][ty * 8]);
      const float4 qb = *reinterpret_cast<const float4*>(&sq[j][ty * 8 + 4]);
      const float4 kv = *reinterpret_cast<const float4*>(&sk[j][tx * 4]);
      const float qv[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        acc[a][0] = add2(acc[a][0], fma2(both(qv[a]), make_float2(kv.x, kv.y), zero));
        acc[a][1] = add2(acc[a][1], fma2(both(qv[a]), make_float2(kv.z, kv.w), zero));
      }
    };
    if (jn == SS_J) {
#pragma unroll 8
      for (int j = 0; j < SS_J; ++j) step(j);
    } else {
      for (int j = 0; j < jn; ++j) step(j);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int t = t0 + ty * 8 + a;
    if (t >= tokens) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int kk = k0 + tx * 4 + b;
      if (kk < side) out[(size_t)t * side + kk] = (b & 1) ? acc[a][b >> 1].y : acc[a][b >> 1].x;
    }
  }
}

// ---- product-key candidates from side scores (src/memory_transformer.rs:847-924; CUDA twin
// kernels.ptx:2121-2262): top-`beam` per side (desc score, asc index), beam^2 f32 sums, top-k by
// (desc sum, asc slot).  One warp per token; side <= 2048, beam <= 32, top_k <= beam*beam.
//
// A warp a token, and everything it does is a chain of dependent steps, so what counts is their number (2048 tokens: 50 -> 22 us, 16384
// tokens 141 -> 81).  Scores become order-preserving 32-bit keys held in registers, all loaded at once.  The 32nd largest of the lanes'
// two largest keys is a bound that the beam's keys reach and few others (36 of 512 random ones); those are sorted with their
// indices.  Of the sums of two sorted beams only those of ranks i and j with (i + 1)(j + 1) <= top_k can be among the top_k, 119 for
// 32, since as many pairs of lower ranks are no smaller; they are sorted with their slots.  Whatever that does not settle (more than 64
// keys that reach the bound, top_k above 32, infinities and NaNs in a beam, a pair left out that equals the last one taken) goes the
// general way: a four-pass radix select over a per-warp histogram, and a merge of the 32 sorted rows `left[i] + right[.]` with
// one pointer per lane, where a round is two warp reductions and only the winning lane advances. ---------------------------------
constexpr int PK_MAX_PER_LANE = 64;

// a > b as floats  <=>  okey(a) > okey(b); both zeros share a key, a NaN gets the lowest key 1, 0 means "no entry"
__device__ __forceinline__ unsigned okey(float f) {
  if (f != f) return 1u;
  const unsigned u = __float_as_uint(f == 0.f ? 0.f : f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_value(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// A step of a bitonic sort across the lanes, of N values a lane side by side.
template <int N, typename V>
__device__ __forceinline__ void exchange(V (&v)[N], int stride, bool keep_max) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const V other = __shfl_xor_sync(0xffffffffu, v[i], stride);
    v[i] = keep_max ? (v[i] > other ? v[i] : other) : (v[i] < other ? v[i] : other);
  }
}
// Each v[i] in descending order over the lanes.
template <int N, typename V>
__device__ __forceinline__ void sort_lanes(V (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) exchange(v, stride, ((lane & stride) == 0) == ((lane & size) == 0));
}
// The 32 largest of two descending vectors, in no order but one that merge_lanes takes.
template <typename V> __device__ __forceinline__ V upper_half(V a, V b) {
  const V other = __shfl_sync(0xffffffffu, b, 31 - (threadIdx.x & 31));
  return a > other ? a : other;
}
template <int N, typename V>
__device__ __forceinline__ void merge_lanes(V (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) exchange(v, stride, (lane & stride) == 0);
}

struct TopkScratch {  // of a warp
  unsigned hist[256], key[64];
  int index[64];
  float rscore[32];
};

// The beam's keys and indices of one side, sorted across the lanes: key descending, index ascending; zero past the beam.
template <int PER_LANE>
__device__ __forceinline__ unsigned long long radix_beam(const unsigned (&key)[PER_LANE], int beam, TopkScratch& sc) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  // radix select, 8 bits a pass from the top: afterwards `kstar` is the beam-th largest key and `need` says how
  // many entries equal to it belong to the beam
  unsigned kstar = 0u, decided = 0u;
  int need = beam;
#pragma unroll 1
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int b = lane; b < 256; b += 32) sc.hist[b] = 0u;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (key[i] != 0u && (key[i] & decided) == kstar) atomicAdd(&sc.hist[(key[i] >> shift) & 255u], 1u);
    __syncwarp();
    unsigned c[8], mine = 0u;  // the lane owns digits 8*lane .. 8*lane+7
#pragma unroll
    for (int b = 0; b < 8; ++b) { c[b] = sc.hist[lane * 8 + b]; mine += c[b]; }
    unsigned from_here = mine;  // entries whose digit is in this lane's range or above
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_down_sync(full, from_here, o);
      if (lane + o < 32) from_here += y;
    }
    const unsigned above = from_here - mine;
    const bool here = above < (unsigned)need && from_here >= (unsigned)need;
    int digit = 0;
    unsigned over = 0u;
    if (here) {
      unsigned run = above;
      bool found = false;
#pragma unroll
      for (int b = 7; b >= 0; --b) {
        if (!found) {
          if (run + c[b] >= (unsigned)need) { digit = lane * 8 + b; over = run; found = true; }
          else run += c[b];
        }
      }
    }
    const unsigned who = __ballot_sync(full, here);
    const int src = who ? __ffs(who) - 1 : 0;  // who == 0 only with fewer than `beam` entries, which the host rejects
    digit = __shfl_sync(full, digit, src);
    over = __shfl_sync(full, over, src);
    kstar |= (unsigned)digit << shift;
    decided |= 255u << shift;
    need -= (int)over;
    __syncwarp();
  }
  // compaction in index order: everything above the threshold, and the first `need` entries equal to it
  int base = 0, eq_seen = 0;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const bool eq = key[i] == kstar && kstar != 0u;
    const unsigned b_eq = __ballot_sync(full, eq);
    const bool take = (key[i] > kstar && kstar != 0u) || (eq && eq_seen + __popc(b_eq & below) < need);
    eq_seen += __popc(b_eq);
    const unsigned b_take = __ballot_sync(full, take);
    if (take) {
      const int pos = base + __popc(b_take & below);
      if (pos < 32) { sc.key[pos] = key[i]; sc.index[pos] = i * 32 + lane; }
    }
    base += __popc(b_take);
  }
  __syncwarp();
  const bool valid = lane < base && lane < 32;
  unsigned long long v[1] = {valid ? ((unsigned long long)sc.key[lane] << 32) | (0xffffffffu - (unsigned)sc.index[lane]) : 0ull};
  __syncwarp();
  sort_lanes(v);
  return v[0];
}
// The 32nd largest of the lanes' two largest keys, which at least 32 keys reach where there are as many.
template <int PER_LANE>
__device__ __forceinline__ unsigned key_bound(const unsigned (&key)[PER_LANE]) {
  unsigned top[2] = {0u, 0u};
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    top[1] = max(top[1], min(top[0], key[i]));
    top[0] = max(top[0], key[i]);
  }
  sort_lanes(top);
  return max(1u, __reduce_min_sync(0xffffffffu, upper_half(top[0], top[1])));
}
template <int PER_LANE>
__device__ __forceinline__ void load_scores(const float* s, int side, float (&score)[PER_LANE]) {
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) score[i] = s[min(i * 32 + (int)(threadIdx.x & 31), side - 1)];
}
template <int PER_LANE>
__device__ __forceinline__ unsigned long long beam_of_scores(const float (&score)[PER_LANE], int side, int beam, TopkScratch& sc) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  unsigned key[PER_LANE];
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    key[i] = i * 32 + lane < side ? okey(score[i]) : 0u;
  }
  const unsigned bound = key_bound(key);
  int count = 0;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const unsigned who = __ballot_sync(full, key[i] >= bound);
    const int at = count + __popc(who & below);
    if (key[i] >= bound && at < 64) {
      sc.key[at] = key[i];
      sc.index[at] = i * 32 + lane;
    }
    count += __popc(who);
  }
  __syncwarp();
  if (count > 64) return radix_beam(key, beam, sc);
  unsigned long long v[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int at = h * 32 + lane;
    v[h] = at < count ? ((unsigned long long)sc.key[at] << 32) | (0xffffffffu - (unsigned)sc.index[at]) : 0ull;
  }
  __syncwarp();
  sort_lanes(v);
  unsigned long long best[1] = {upper_half(v[0], v[1])};
  merge_lanes(best);
  return lane < beam ? best[0] : 0ull;
}

// The top_k of all sums of the two beams, the general way.
__device__ __noinline__ void merge_beams(unsigned l_key, int l_idx, unsigned r_key, int r_idx, int64_t* out, int64_t* kept, int side, int top_k,
                                         int beam, TopkScratch& sc, int* status) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  sc.key[lane] = r_key;
  sc.index[lane] = r_idx;
  sc.rscore[lane] = okey_value(r_key);
  __syncwarp();
  // row `lane` of the candidate matrix: left[lane] + right[j], non-increasing in j because the right beam is sorted
  // and f32 addition is monotone.  Equal sums sit next to each other; among them the lowest slot goes first.
  const bool has = lane < beam && l_key != 0u;
  const float ls = okey_value(l_key);
  const unsigned beam_mask = beam >= 32 ? 0xffffffffu : ((1u << beam) - 1u);
  unsigned used = 0u;
  unsigned head_key = 0u, head_slot = 0xffffffffu;
  int head_j = 0;
  auto advance = [&]() {
    head_key = 0u;
    head_slot = 0xffffffffu;
    const unsigned avail = ~used & beam_mask;
    if (!has || avail == 0u) return;
    const int j = __ffs(avail) - 1;
    if (sc.key[j] == 0u) return;
    const float sum = __fadd_rn(ls, sc.rscore[j]);
    int best_ri = sc.index[j], best_j = j;
    for (int jj = j + 1; jj < beam; ++jj) {
      if (sc.key[jj] == 0u || !(__fadd_rn(ls, sc.rscore[jj]) == sum)) break;
      if (!((used >> jj) & 1u) && sc.index[jj] < best_ri) { best_ri = sc.index[jj]; best_j = jj; }
    }
    head_key = okey(sum);
    head_slot = (unsigned)(l_idx * side + best_ri);
    head_j = best_j;
  };
  advance();
  for (int r = 0; r < top_k; ++r) {
    const unsigned m = __reduce_max_sync(full, head_key);
    if (m == 0u) {
      if (lane == 0) {
        atomicExch(status + ST_BAD_ARGUMENT, 1);
        out[r] = 0;
        if (kept) kept[r] = 0;
      }
      continue;
    }
    const unsigned bs = __reduce_min_sync(full, head_key == m ? head_slot : 0xffffffffu);
    if (head_key == m && head_slot == bs) {  // slots differ between lanes: exactly one winner
      used |= 1u << head_j;
      advance();
    }
    if (lane == 0) {
      out[r] = (long long)bs;
      if (kept) kept[r] = (long long)bs;
    }
  }
}

// The top_k of all sums of two sorted beams (okey << 32 | ~index, zero past the beam) into `out`, and `kept` where given.
__device__ __forceinline__ void pick_pairs(unsigned long long l, unsigned long long r, int64_t* out, int64_t* kept, int side, int top_k, int beam,
                                           TopkScratch& sc, int* status) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  const unsigned l_key = (unsigned)(l >> 32), r_key = (unsigned)(r >> 32);
  const int l_idx = (int)(0xffffffffu - (unsigned)l), r_idx = (int)(0xffffffffu - (unsigned)r);
  const float ls = okey_value(l_key), rs = okey_value(r_key);
  bool general = top_k > 32 || __any_sync(full, lane < beam && !(isfinite(ls) && isfinite(rs)));
  if (!general) {
    const int mine = lane < beam ? min(beam, top_k / (lane + 1)) : 0;  // pairs of left rank `lane`
    int upto = mine;                                                    // pairs up to and with it
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(full, upto, o);
      if (lane >= o) upto += y;
    }
    const int pairs = __shfl_sync(full, upto, 31);  // at most 119
    auto pair_of = [&](int m) {  // number m * 32 + lane, zero past the last
      const int c = m * 32 + lane;
      int i = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (c >= __shfl_sync(full, upto, i + step - 1)) i += step;
      const int j = (c - __shfl_sync(full, upto - mine, i)) & 31;
      const float sum = __fadd_rn(__shfl_sync(full, ls, i), __shfl_sync(full, rs, j));
      const unsigned slot = (unsigned)(__shfl_sync(full, l_idx, i) * side + __shfl_sync(full, r_idx, j));
      return c < pairs ? ((unsigned long long)okey(sum) << 32) | (0xffffffffu - slot) : 0ull;
    };
    unsigned long long best[1];
    if (pairs <= 32) {  // top_k up to 11 (16384 tokens, sides of 48, top_k 4 72.7 us with all four rows of pairs, 53.5 without)
      best[0] = pair_of(0);
      sort_lanes(best);
    } else {
      unsigned long long v[4] = {pair_of(0), pair_of(1), pair_of(2), pair_of(3)};
      sort_lanes(v);
      unsigned long long two[2] = {upper_half(v[0], v[1]), upper_half(v[2], v[3])};
      merge_lanes(two);
      best[0] = upper_half(two[0], two[1]);
      merge_lanes(best);
    }
    const unsigned last = (unsigned)(__shfl_sync(full, best[0], top_k - 1) >> 32);
    const float next = __fadd_rn(ls, __shfl_sync(full, rs, mine & 31));  // the largest of this rank's pairs that were left out
    general = __any_sync(full, lane < beam && mine < beam && okey(next) == last);
    if (!general && lane < top_k) {
      const long long slot = (long long)(0xffffffffu - (unsigned)best[0]);
      out[lane] = slot;
      if (kept) kept[lane] = slot;
    }
  }
  if (general) merge_beams(l_key, l_idx, r_key, r_idx, out, kept, side, top_k, beam, sc, status);
}

template <int PER_LANE>
__global__ void __launch_bounds__(128)
product_key_topk_kernel(const float* __restrict__ left, const float* __restrict__ right, int64_t* __restrict__ out,
                        int tokens, int side, int top_k, int beam, int* __restrict__ status, int64_t* __restrict__ kept,
                        const long long* __restrict__ kept_row) {
  pdl_begin();
  __shared__ TopkScratch scratch[4];
  const int w = threadIdx.x >> 5;
  const int token = blockIdx.x * 4 + w;
  if (token >= tokens) return;
  TopkScratch& sc = scratch[w];
  float score[PER_LANE];
  load_scores(left + (size_t)token * side, side, score);
  const unsigned long long l = beam_of_scores(score, side, beam, sc);
  load_scores(right + (size_t)token * side, side, score);
  const unsigned long long r = beam_of_scores(score, side, beam, sc);
  pick_pairs(l, r, out + (size_t)token * top_k, kept ? kept + (*kept_row + token) * top_k : nullptr, side, top_k, beam, sc, status);
}

// ---- the same from queries: side scores that decide nothing are not formed exactly ----------------------------------------
// Every score is an f32 sum in a fixed order with separately rounded products (side_scores_kernel), 340 us for 16384 tokens and two
// tables of 512 x 256, of which the selection wants 32 in 512.  So the tensor core forms all of them first out of bf16 pieces, hi * hi +
// lo * hi + hi * lo, and only what can be among the beam's is formed again as it has to be: with |approximate - exact| <= E, every
// key of the beam has an approximate score of at least the beam-th largest minus 2 E.  In terms of S, the norm of the token's half
// query times the largest norm of a half key (sum |q k| <= S): rounding to bf16 leaves up to 2^-8 of a value, and rounding that again up to
// 2^-17 of the value, so that lo * lo is up to 2^-16 S and the two remainders up to 2^-17 S each, 2^-15 S in all; the f32 sum is off by at
// most 2 half * 2^-24 S, and each of the 3 half / 16 tensor-core steps by 17 terms cut off at 2^-23: together less than (5.0e-7 half + 3.06e-5) S.
// The band is taken with 5.4e-7 and 3.2e-5, for what the norms' own sums round.
// Where S is not within 1e-30 and 1e37 (or a norm below 1e-18: its squares and the pieces of such values lose bits), or more than 64 keys come into
// question, all scores of that token and side are formed exactly.  The selections are the same bit by bit.  The kernel takes 226 us of the 276,
// two thirds of the shared memory's rate: rows are staged there for the lanes that walk them; 5 or 6 blocks an SM: 230 and 234.
constexpr int LK_PER_LANE = 16;          // sides of up to 512
constexpr int LK_J = 32, LK_LD = LK_J + 4;  // columns of 32 rows in shared memory at a time, and their pitch
__device__ __forceinline__ const float* shuffle_pointer(const float* p, int lane) {
  return reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), lane));
}
// The exact score of the lane's half query (in shared memory) and half key: rows come in whole segments, a lane walks its own (null: none).
__device__ __forceinline__ float exact_score(const float* key_row, const float* q, int half, float* buf) {
  const int lane = threadIdx.x & 31;
  const float* src[8];
  float4 r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    src[i] = shuffle_pointer(key_row, i * 4 + (lane >> 3));
    if (src[i]) r[i] = __ldg(reinterpret_cast<const float4*>(src[i] += (lane & 7) * 4));
  }
  float acc = 0.f;
#pragma unroll 1
  for (int j0 = 0; j0 < half; j0 += LK_J) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (src[i]) *reinterpret_cast<float4*>(buf + (i * 4 + (lane >> 3)) * LK_LD + (lane & 7) * 4) = r[i];
    __syncwarp();
    if (j0 + LK_J < half) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (src[i]) r[i] = __ldg(reinterpret_cast<const float4*>(src[i] + j0 + LK_J));
    }
    if (!key_row) continue;
#pragma unroll
    for (int j = 0; j < LK_J; j += 4) {
      const float4 k = *reinterpret_cast<const float4*>(buf + lane * LK_LD + j), x = *reinterpret_cast<const float4*>(q + j0 + j);
      acc = __fadd_rn(acc, __fmul_rn(x.x, k.x));
      acc = __fadd_rn(acc, __fmul_rn(x.y, k.y));
      acc = __fadd_rn(acc, __fmul_rn(x.z, k.z));
      acc = __fadd_rn(acc, __fmul_rn(x.w, k.w));
    }
  }
  __syncwarp();
  return acc;
}
// Indices of the keys whose approximate score is no further than `band` below the beam-th largest; their number, -1 when it is above 64.
__device__ __forceinline__ int find_candidates(const float* approximate, int side, int beam, float band, int* cand, TopkScratch& sc) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  float score[LK_PER_LANE];
  unsigned key[LK_PER_LANE];
  load_scores(approximate, side, score);
#pragma unroll
  for (int i = 0; i < LK_PER_LANE; ++i) key[i] = i * 32 + lane < side ? okey(score[i]) : 0u;
  const unsigned bound = key_bound(key);
  const float least = bound > 1u ? okey_value(bound) - band : -INFINITY;
  int count = 0;
#pragma unroll
  for (int i = 0; i < LK_PER_LANE; ++i) {
    const bool take = key[i] != 0u && score[i] >= least;
    const unsigned who = __ballot_sync(full, take);
    const int at = count + __popc(who & below);
    if (take && at < 64) {
      sc.key[at] = key[i];
      sc.index[at] = i * 32 + lane;
    }
    count += __popc(who);
  }
  __syncwarp();
  if (count > 64 || count < beam) return -1;
  unsigned v[2] = {lane < count ? sc.key[lane] : 0u, 32 + lane < count ? sc.key[32 + lane] : 0u};
  unsigned sorted[2] = {v[0], v[1]};
  sort_lanes(sorted);
  unsigned best[1] = {upper_half(sorted[0], sorted[1])};
  merge_lanes(best);
  const float last = okey_value(__shfl_sync(full, best[0], beam - 1)) - band;
  int n = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool take = v[h] != 0u && okey_value(v[h]) >= last;
    const unsigned who = __ballot_sync(full, take);
    if (take) cand[n + __popc(who & below)] = sc.index[h * 32 + lane];
    n += __popc(who);
  }
  __syncwarp();
  return n;
}
// A side's beam out of exact scores of all of its keys.
__device__ __noinline__ unsigned long long exact_beam(const float* keys, const float* q, int side, int half, int beam, float* buf, TopkScratch& sc) {
  float score[LK_PER_LANE];
#pragma unroll
  for (int i = 0; i < LK_PER_LANE; ++i) score[i] = 0.f;
#pragma unroll 1
  for (int i = 0; i < LK_PER_LANE; ++i) {
    if (i * 32 >= side) break;
    const float x = exact_score(keys + (size_t)min(i * 32 + (int)(threadIdx.x & 31), side - 1) * half, q, half, buf);
#pragma unroll
    for (int u = 0; u < LK_PER_LANE; ++u)
      if (u == i) score[u] = x;
  }
  return beam_of_scores(score, side, beam, sc);
}

__global__ void __launch_bounds__(128)
product_key_lookup_kernel(const float* __restrict__ left_approx, const float* __restrict__ right_approx, const float* __restrict__ query,
                          long long ld_q, const float* __restrict__ left_keys, const float* __restrict__ right_keys,
                          const float* __restrict__ norms /* largest of either side */, int64_t* __restrict__ out, int tokens, int side, int half,
                          int top_k, int beam, int* __restrict__ status) {
  pdl_begin();
  extern __shared__ __align__(16) float lk_smem[];
  __shared__ TopkScratch scratch[4];
  __shared__ int cands[4][2][64];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int token = blockIdx.x * 4 + w;
  if (token >= tokens) return;
  TopkScratch& sc = scratch[w];
  float* q = lk_smem + w * (2 * half + 32 * LK_LD);
  float* buf = q + 2 * half;
  float squares[2] = {0.f, 0.f};
  for (int c = lane * 4; c < 2 * half; c += 128) {
    const float4 x = *reinterpret_cast<const float4*>(query + (size_t)token * ld_q + c);
    *reinterpret_cast<float4*>(q + c) = x;
    const float t = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
    if (c < half) squares[0] += t; else squares[1] += t;
  }
  int (*cand)[64] = cands[w];
  int count[2];
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    const float qn = sqrtf(warp_sum(squares[sd])), kn = norms[sd], s = qn * kn;
    const bool within = qn >= 1e-18f && kn >= 1e-18f && s >= 1e-30f && s <= 1e37f;  // (false for NaN)
    const float band = 2.f * s * (5.4e-7f * (float)half + 3.2e-5f);
    count[sd] = within ? find_candidates((sd ? right_approx : left_approx) + (size_t)token * side, side, beam, band, cand[sd], sc) : -1;
  }
  int more[2] = {max(0, count[0] - 32), max(0, count[1] - 32)};  // beyond a warp's lanes
  if (more[0] + more[1] > 32) {
    count[more[0] > more[1] ? 0 : 1] = -1;
    more[more[0] > more[1] ? 0 : 1] = 0;
  }
  unsigned long long v[2][2];  // [side]: the first 32 candidates, the rest
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    v[sd][0] = v[sd][1] = 0ull;
    if (count[sd] < 0) continue;
    const int mine = lane < count[sd] ? cand[sd][lane] : 0;
    const float x = exact_score(lane < count[sd] ? (sd ? right_keys : left_keys) + (size_t)mine * half : nullptr, q + sd * half, half, buf);
    if (lane < count[sd]) v[sd][0] = ((unsigned long long)okey(x) << 32) | (0xffffffffu - (unsigned)mine);
  }
  if (more[0] + more[1] > 0) {  // both sides' in one go
    const int sd = lane < more[0] ? 0 : 1, at = sd ? lane - more[0] : lane;
    const bool real = lane < more[0] + more[1];
    const int mine = real ? cand[sd][32 + at] : 0;
    const float x = exact_score(real ? (sd ? right_keys : left_keys) + (size_t)mine * half : nullptr, q + sd * half, half, buf);
    const unsigned long long e = ((unsigned long long)okey(x) << 32) | (0xffffffffu - (unsigned)mine);
    if (real && sd == 0) v[0][1] = e;
    if (real && sd == 1) v[1][1] = e;
  }
  unsigned long long beams[2];
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    if (count[sd] < 0) {
      beams[sd] = exact_beam(sd ? right_keys : left_keys, q + sd * half, side, half, beam, buf, sc);
      continue;
    }
    if (more[sd] > 0) {
      sort_lanes(v[sd]);
      unsigned long long best[1] = {upper_half(v[sd][0], v[sd][1])};
      merge_lanes(best);
      beams[sd] = best[0];
    } else {
      unsigned long long one[1] = {v[sd][0]};
      sort_lanes(one);
      beams[sd] = one[0];
    }
    if (lane >= beam) beams[sd] = 0ull;
  }
  pick_pairs(beams[0], beams[1], out + (size_t)token * top_k, nullptr, side, top_k, beam, sc, status);
}

// Operands of the approximate scores.  Queries: row [hi left | lo left | hi right | lo right]; half keys: row [hi | hi | lo], the left
// table's rows, then the right one's, and the largest norm of either table.
__global__ void __launch_bounds__(256)
query_pieces_kernel(const float* __restrict__ query, long long ld_q, __nv_bfloat16* __restrict__ out, int tokens, int half) {
  pdl_begin();
  const int per_row = half / 4;  // groups of eight in a row
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  const long long t = i / per_row;
  if (t >= tokens) return;
  const int c = (int)(i - t * per_row) * 8, sd = c >= half;
  float x[8];
  const float4 a = *reinterpret_cast<const float4*>(query + t * ld_q + c), b = *reinterpret_cast<const float4*>(query + t * ld_q + c + 4);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  uint4 piece[3];
  split8_bf16(x, piece);
  __nv_bfloat16* to = out + t * 4 * half + sd * 2 * half + (c - sd * half);
  *reinterpret_cast<uint4*>(to) = piece[0];
  *reinterpret_cast<uint4*>(to + half) = piece[1];
}
__global__ void __launch_bounds__(256)
key_pieces_kernel(const float* __restrict__ left, const float* __restrict__ right, __nv_bfloat16* __restrict__ out, int* __restrict__ norm_bits,
                  int side, int half) {
  pdl_begin();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= 2 * side) return;
  const float* key = row < side ? left + (size_t)row * half : right + (size_t)(row - side) * half;
  float squares = 0.f;
  for (int c = lane * 8; c < half; c += 256) {
    float x[8];
    const float4 a = __ldg(reinterpret_cast<const float4*>(key + c)), b = __ldg(reinterpret_cast<const float4*>(key + c + 4));
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
#pragma unroll
    for (int e = 0; e < 8; ++e) squares += x[e] * x[e];
    uint4 piece[3];
    split8_bf16(x, piece);
    __nv_bfloat16* to = out + (size_t)row * 3 * half + c;
    *reinterpret_cast<uint4*>(to) = piece[0];
    *reinterpret_cast<uint4*>(to + half) = piece[0];
    *reinterpret_cast<uint4*>(to + 2 * half) = piece[1];
  }
  squares = warp_sum(squares);
  const float norm = sqrtf(squares);
  if (lane == 0) atomicMax(norm_bits + (row >= side), norm == norm ? __float_as_int(norm) : 0x7fffffff);  // (a NaN stays one)
}

__global__ void split_rows_kernel(const int64_t* __restrict__ rows, int64_t* __restrict__ left, int64_t* __restrict__ right,
                                  long long n, int side) {
  pdl_begin();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long r = rows[i];
  left[i] = r / side;
  right[i] = r % side;
}

// Sums over the warp's lanes of eight values a lane: value 4 b4 + 2 b3 + b2 in the lanes whose bits 4, 3 and 2 are these (a lane keeps
// the half of its values that its bit names and gives the other half away: 9 exchanges instead of 40).
__device__ __forceinline__ double sum8_over_lanes(double (&v)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 16, n = 4; n >= 1; d >>= 1, n >>= 1) {
    const bool upper = (lane & d) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const double send = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}
__device__ __forceinline__ int sum8_index() { return (threadIdx.x & 31) >> 2; }  // which of the eight a lane holds then

// The kernels that gather table rows (selected scores and weighted value, forward and backward) are bound by how many rows are on
// their way: by L2 for many tokens (16384 tokens of 32 rows of 2 KB: 50 to 100 us a kernel), and for few by latency, since with a warp
// a token, a row after the other, 2048 tokens keep a tenth of the memory busy.  So a warp asks for eight pieces of rows at a time, and where
// columns do not meet, for a few of a row's pieces only (by_pieces).  Scores, their gradient and value of 32 slots of 512 columns at 2048
// tokens 21, 25 and 18 -> 13, 9 and 10 us, at 16384 tokens 100, 77 and 72 -> 64, 53 and 57.
constexpr int GATHER = 8;
__device__ __forceinline__ float4 row_piece(const float* table, long long row, int dim, int piece, bool on) {
  return on && row >= 0 ? __ldg(reinterpret_cast<const float4*>(table + (size_t)row * dim) + piece) : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ void add_scaled(float4& acc, float w, const float4& v) {
  acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
}
// launch(pieces of a row a lane has): as many as leave a warp several rows on their way, and more where a token has a slot or two, so
// that as many bytes are asked for.  Value of 16384 tokens of 512 columns, one, two, four pieces, us: 1 slot 18.8, 10.4, 8.0, 8 slots 23.4,
// 17.9, 17.7, 32 slots 65, 57, 57; 2048 tokens of 32 slots 13.1, 10.2, 10.3; 64 tokens 5.6, 4.1, 6.1.
template <typename F> void by_pieces(int top_k, int dim, F launch) {
  if (dim <= 128) launch(std::integral_constant<int, 1>{});
  else if (dim <= 256 || top_k > 2) launch(std::integral_constant<int, 2>{});
  else launch(std::integral_constant<int, 4>{});
}

// ---- selected scores: score[t,k] = q_L . K_L[idx/side] + q_R . K_R[idx%side]  (src/tensor.rs:3593-3769).
// Product-key form, key_dim up to 128 U, sixteen-byte rows: one, two or four warps a token, eight slots each at a time (a CTA a token left
// three of its warps idle for up to eight slots: 2048 tokens of 8 slots of 512 columns 14.4 us, 10.0 before that); the query sits in registers.  A lane's share (at most 4 U products) is summed in f32, the 32 shares in f64: f64 multiply-adds run at a
// fraction of the f32 rate.
template <int U>
__global__ void __launch_bounds__(128)
selected_scores_rows_kernel(const int64_t* __restrict__ idx, const float* __restrict__ query, long long ld_q,
                            const float* __restrict__ left, const float* __restrict__ right, float* __restrict__ scores, int tokens,
                            int top_k, int side, int key_dim, int slots, int log_warps, int* __restrict__ status) {
  pdl_begin();
  const int lane = threadIdx.x & 31, w = (int)blockIdx.x * 4 + (int)(threadIdx.x >> 5);
  if (w >> log_warps >= tokens) return;
  const size_t token = w >> log_warps;
  const int first = (w & ((1 << log_warps) - 1)) * GATHER, step = GATHER << log_warps;
  const int half = key_dim / 2, groups = key_dim / 4, half_groups = half / 4;
  float4 qv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int gi = u * 32 + lane;
    qv[u] = gi < groups ? *reinterpret_cast<const float4*>(query + token * ld_q + gi * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int k0 = first; k0 < top_k; k0 += step) {
    int my_li = -1, my_ri = 0;
    if (lane < GATHER && k0 + lane < top_k) {
      const long long slot = idx[token * top_k + k0 + lane];
      if (slot >= 0 && slot < slots) {
        my_li = (int)((unsigned)slot / (unsigned)side);
        my_ri = (int)((unsigned)slot % (unsigned)side);
      } else {
        atomicExch(status + ST_BAD_INDEX, 1);
      }
    }
    double part[GATHER];
#pragma unroll
    for (int k = 0; k < GATHER; ++k) {
      const int li = __shfl_sync(0xffffffffu, my_li, k), ri = __shfl_sync(0xffffffffu, my_ri, k);
      float acc = 0.f;
      if (li >= 0) {
        const float4* lrow = reinterpret_cast<const float4*>(left + (size_t)li * half);
        const float4* rrow = reinterpret_cast<const float4*>(right + (size_t)ri * half);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int gi = u * 32 + lane;
          if (gi < groups) {
            const float4 kv = gi < half_groups ? __ldg(lrow + gi) : __ldg(rrow + (gi - half_groups));
            acc = fmaf(qv[u].x, kv.x, acc); acc = fmaf(qv[u].y, kv.y, acc);
            acc = fmaf(qv[u].z, kv.z, acc); acc = fmaf(qv[u].w, kv.w, acc);
          }
        }
      }
      part[k] = (double)acc;
    }
    const double sum = sum8_over_lanes(part);
    const int k = k0 + sum8_index();
    if ((lane & 3) == 0 && k < top_k) scores[token * top_k + k] = (float)sum;
  }
}

// The same for any sizes, and in `exact` mode (side == 0): score = q . K[idx] over key_dim (src/tensor.rs:3465-3548).  A warp a token.
__global__ void selected_scores_fwd_kernel(const int64_t* __restrict__ idx, const float* __restrict__ query, long long ld_q,
                                           const float* __restrict__ left, const float* __restrict__ right,
                                           float* __restrict__ scores, int tokens, int top_k, int side, int key_dim,
                                           int slots, int* __restrict__ status) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= tokens) return;
  const int half = side > 0 ? key_dim / 2 : key_dim;
  const float* q = query + (size_t)token * ld_q;
  for (int k = 0; k < top_k; ++k) {
    const long long slot = idx[(size_t)token * top_k + k];
    if (slot < 0 || slot >= slots) {
      if (lane == 0) { atomicExch(status + ST_BAD_INDEX, 1); scores[(size_t)token * top_k + k] = 0.f; }
      continue;
    }
    double acc = 0.0;
    if (side > 0) {
      const unsigned s32 = (unsigned)slot, side32 = (unsigned)side;
      const float* kl = left + (size_t)(s32 / side32) * half;
      const float* kr = right + (size_t)(s32 % side32) * half;
      for (int j = lane; j < half; j += 32) acc += (double)q[j] * (double)kl[j] + (double)q[half + j] * (double)kr[j];
    } else {
      const float* kr = left + (size_t)slot * key_dim;
      for (int j = lane; j < key_dim; j += 32) acc += (double)q[j] * (double)kr[j];
    }
    acc = warp_sum(acc);
    if (lane == 0) scores[(size_t)token * top_k + k] = (float)acc;
  }
}

// dq[t,:] = sum_k g[t,k] * [K_L[li]; K_R[ri]] of the product-key form, sixteen-byte rows: a warp a token and 128 U columns.
template <int U>
__global__ void __launch_bounds__(128)
selected_query_gradient_kernel(const int64_t* __restrict__ idx, const float* __restrict__ left, const float* __restrict__ right,
                               const float* __restrict__ grad_scores, float* __restrict__ dq, long long ld_dq, int tokens, int top_k,
                               int side, int key_dim, int slots, int* __restrict__ clear) {
  pdl_begin();
  if (clear && blockIdx.x == 0 && threadIdx.x == 0) *clear = 0;  // a word that the kernels behind this one set and read
  constexpr int ROWS = GATHER / U;
  const int lane = threadIdx.x & 31, slices = (key_dim + 128 * U - 1) / (128 * U), w = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int token = w / slices, g0 = (w - token * slices) * 32 * U + lane, half = key_dim / 2, groups = key_dim / 4, half_groups = half / 4;
  if (token >= tokens) return;
  float4 acc[U];
#pragma unroll
  for (int u = 0; u < U; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < top_k; k0 += 32) {
    int my_li = -1, my_ri = -1;
    float my_g = 0.f;
    if (k0 + lane < top_k) {
      const long long slot = idx[(size_t)token * top_k + k0 + lane];
      if (slot >= 0 && slot < slots) {
        my_li = (int)((unsigned)slot / (unsigned)side);
        my_ri = (int)((unsigned)slot % (unsigned)side);
        my_g = grad_scores[(size_t)token * top_k + k0 + lane];
      }
    }
    for (int k = 0; k < min(32, top_k - k0); k += ROWS) {
      float4 v[ROWS][U];
      float g[ROWS];
      bool there[ROWS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        const int li = __shfl_sync(0xffffffffu, my_li, k + j), ri = __shfl_sync(0xffffffffu, my_ri, k + j);
        g[j] = __shfl_sync(0xffffffffu, my_g, k + j);
        there[j] = li >= 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int gi = g0 + u * 32;
          const bool in_left = gi < half_groups;
          v[j][u] = row_piece(in_left ? left : right, in_left ? li : ri, half, in_left ? gi : gi - half_groups, gi < groups);
        }
      }
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
        if (there[j])
#pragma unroll
          for (int u = 0; u < U; ++u) add_scaled(acc[u], g[j], v[j][u]);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (g0 + u * 32 < groups) *reinterpret_cast<float4*>(dq + (size_t)token * ld_dq + (g0 + u * 32) * 4) = acc[u];
}

// The same for any sizes, and in `exact` mode with dK[idx,:] += g[t,k] q[t]
// (src/tensor/autograd.rs:2386-2494).  Those key gradients use f32 atomics like the reference.
__global__ void selected_scores_bwd_kernel(const int64_t* __restrict__ idx, const float* __restrict__ query, long long ld_q,
                                           const float* __restrict__ left, const float* __restrict__ right,
                                           const float* __restrict__ grad_scores, float* __restrict__ dq, long long ld_dq,
                                           float* __restrict__ dleft, float* __restrict__ dright, int tokens, int top_k,
                                           int side, int key_dim, int slots, int* __restrict__ clear) {
  pdl_begin();
  if (clear && blockIdx.x == 0 && threadIdx.x == 0) *clear = 0;  // a word that the kernels behind this one set and read
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= tokens) return;
  const int half = side > 0 ? key_dim / 2 : key_dim;
  const float* q = query + (size_t)token * ld_q;
  if (dq) {
    for (int j = lane; j < key_dim; j += 32) {
      double acc = 0.0;
      for (int k = 0; k < top_k; ++k) {
        const long long slot = idx[(size_t)token * top_k + k];
        if (slot < 0 || slot >= slots) continue;
        const double g = (double)grad_scores[(size_t)token * top_k + k];
        float kv;
        if (side > 0) kv = j < half ? left[(size_t)(slot / side) * half + j] : right[(size_t)(slot % side) * half + (j - half)];
        else kv = left[(size_t)slot * key_dim + j];
        acc += g * (double)kv;
      }
      dq[(size_t)token * ld_dq + j] = (float)acc;
    }
  }
  if (side > 0) return;  // the half-key gradients of the product-key form come from product_key_dkeys_kernel
  for (int k = 0; k < top_k; ++k) {
    const long long slot = idx[(size_t)token * top_k + k];
    if (slot < 0 || slot >= slots) continue;
    const float g = grad_scores[(size_t)token * top_k + k];
    if (dleft) {
      float* dk = dleft + (size_t)slot * key_dim;
      for (int j = lane; j < key_dim; j += 32) atomicAdd(dk + j, g * q[j]);
    }
  }
}

// Half-key gradients of the product-key form: dK_L[li,:] += g[t,k] q_L[t,:], dK_R[ri,:] += g[t,k] q_R[t,:] over the
// selected slots.  With only `side` rows per table every row collects about tokens*top_k/side terms, so atomics
// (global or shared) would pile onto a few addresses.  The sum is therefore run as a dense product
// dK = Wᵀ·Q with W[t, row] = sum of the g[t,k] whose slot maps to `row`: a CTA owns a block of tokens, 256 rows
// and 64 columns of one table; per slice of 32 tokens it builds W in shared memory (one warp per token, its
// duplicates added in slot order), multiplies with an 8 x 8 register tile per thread (two CTAs per SM), and clears the entries it
// set.  The slots and queries of the next slice are fetched during the product (read where they were needed, the building took
// two thirds of the time: 16384 tokens, 32 of 2 x 512 rows of 256: 386 us).  From 2048 tokens on key_gradient_run (memory_keys.cu)
// takes its place where it can.  The CTA's tile goes out as a partial result that fold_key_partials_kernel adds up in block order, so the
// result does not depend on scheduling.
constexpr int DK_COLS = 64;    // columns per CTA
constexpr int DK_ROWS = 256;   // table rows per CTA
constexpr int DK_TOKENS = 32;  // tokens per slice
__global__ void __launch_bounds__(256, 2)
product_key_dkeys_kernel(const int64_t* __restrict__ idx, const float* __restrict__ query, long long ld_q,
                         const float* __restrict__ grad_scores, float* __restrict__ partial, int tokens, int top_k,
                         int side, int half, int slots, int tokens_per_block, int col_blocks) {
  pdl_begin();
  extern __shared__ __align__(16) float dk_smem[];
  float* w_tile = dk_smem;                          // [DK_TOKENS][DK_ROWS]
  float* q_tile = dk_smem + DK_TOKENS * DK_ROWS;    // [DK_TOKENS][DK_COLS]
  const int table = blockIdx.z;                     // 0 left, 1 right
  const int c0 = (blockIdx.y % col_blocks) * DK_COLS;
  const int r0 = (blockIdx.y / col_blocks) * DK_ROWS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tr = threadIdx.x >> 3;  // 32 row groups of 8 rows
  const int tc = threadIdx.x & 7;   // 8 column groups of 8 columns
  float2 acc[8][4];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = both(0.f);
  for (int i = threadIdx.x; i < DK_TOKENS * DK_ROWS; i += 256) w_tile[i] = 0.f;
  const int t_begin = blockIdx.x * tokens_per_block, t_end = min(tokens, t_begin + tokens_per_block);
  // What a slice is built from travels while the slice before it is multiplied: eight query values a thread, and of each of
  // its warp's four tokens one selected slot a lane (more than 32 slots: the rest is read when it is needed).
  constexpr int TW = DK_TOKENS / 8, QV = DK_TOKENS * DK_COLS / 256;
  float next_q[QV], next_g[TW];
  int next_row[TW];
  const unsigned side32 = (unsigned)side;
  auto row_of = [&](long long slot) -> int {  // within this CTA's rows, -1 outside
    if (slot < 0 || slot >= slots) return -1;
    const unsigned s32 = (unsigned)slot;
    const int row = (int)(table ? s32 % side32 : s32 / side32) - r0;
    return row < 0 || row >= DK_ROWS ? -1 : row;
  };
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < QV; ++i) {
      const int t = (i * 256 + (int)threadIdx.x) / DK_COLS, c = (int)threadIdx.x % DK_COLS;
      next_q[i] = (t0 + t < t_end && c0 + c < half) ? query[(size_t)(t0 + t) * ld_q + (table ? half : 0) + c0 + c] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < TW; ++i) {
      const int t = t0 + warp + i * 8;
      const bool in = t < t_end && lane < top_k;
      next_row[i] = row_of(in ? idx[(size_t)t * top_k + lane] : -1);
      next_g[i] = in ? grad_scores[(size_t)t * top_k + lane] : 0.f;
    }
  };
  // Lanes whose slots share a table row add their gradients one after the other in slot order (round r = the lane's rank among
  // its duplicates), so a row's sum is formed in the same order on every run.
  auto add_row = [&](int t, int row, float g) {
    const unsigned same = __match_any_sync(0xffffffffu, row);
    const int rank = row < 0 ? -1 : __popc(same & ((1u << lane) - 1u));
    const int rounds = __reduce_max_sync(0xffffffffu, rank) + 1;
    for (int r = 0; r < rounds; ++r) {
      if (rank == r) w_tile[t * DK_ROWS + row] += g;
      __syncwarp();
    }
  };
  fetch(t_begin);
  for (int t0 = t_begin; t0 < t_end; t0 += DK_TOKENS) {
    __syncthreads();  // the previous slice's product is done and its entries are cleared (first time: the tile is zero)
    int rows_set[TW];
#pragma unroll
    for (int i = 0; i < QV; ++i) q_tile[i * 256 + threadIdx.x] = next_q[i];
#pragma unroll
    for (int i = 0; i < TW; ++i) {
      rows_set[i] = next_row[i];
      add_row(warp + i * 8, next_row[i], next_g[i]);
    }
    if (top_k > 32)
      for (int t = warp; t < DK_TOKENS && t0 + t < t_end; t += 8)
        for (int k = 32 + lane; k - lane < top_k; k += 32) {
          const bool in = k < top_k;
          add_row(t, row_of(in ? idx[(size_t)(t0 + t) * top_k + k] : -1), in ? grad_scores[(size_t)(t0 + t) * top_k + k] : 0.f);
        }
    if (t0 + DK_TOKENS < t_end) fetch(t0 + DK_TOKENS);
    __syncthreads();
    const int tn = min(DK_TOKENS, t_end - t0);
    for (int t = 0; t < tn; ++t) {
      float wv[8];
      float2 qv[4];
#pragma unroll
      for (int a = 0; a < 8; a += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&w_tile[t * DK_ROWS + tr * 8 + a]);
        wv[a] = x.x; wv[a + 1] = x.y; wv[a + 2] = x.z; wv[a + 3] = x.w;
      }
#pragma unroll
      for (int b = 0; b < 8; b += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&q_tile[t * DK_COLS + tc * 8 + b]);
        qv[b / 2] = make_float2(x.x, x.y);
        qv[b / 2 + 1] = make_float2(x.z, x.w);
      }
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fma2(both(wv[a]), qv[b], acc[a][b]);
    }
    __syncthreads();
    // clear what this slice set
#pragma unroll
    for (int i = 0; i < TW; ++i)
      if (rows_set[i] >= 0) w_tile[(warp + i * 8) * DK_ROWS + rows_set[i]] = 0.f;
    if (top_k > 32)
      for (int t = warp; t < DK_TOKENS && t0 + t < t_end; t += 8)
        for (int k = 32 + lane; k < top_k; k += 32) {
          const int row = row_of(idx[(size_t)(t0 + t) * top_k + k]);
          if (row >= 0) w_tile[t * DK_ROWS + row] = 0.f;
        }
  }
  // partial[block][table][side][half]
  float* dst = partial + ((size_t)blockIdx.x * 2 + table) * side * half;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int row = r0 + tr * 8 + a;
    if (row >= side) continue;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int c = c0 + tc * 8 + b;
      if (c < half) dst[(size_t)row * half + c] = (b & 1) ? acc[a][b / 2].y : acc[a][b / 2].x;
    }
  }
}

__global__ void fold_key_partials_kernel(const float* __restrict__ partial, float* __restrict__ dleft,
                                         float* __restrict__ dright, int blocks, int side, int half) {
  pdl_begin();
  const size_t per_table = (size_t)side * half;
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= 2 * per_table) return;
  const int table = i >= per_table;
  const size_t e = i - table * per_table;
  float* dst = table ? dright : dleft;
  if (!dst) return;
  float s = 0.f;
  for (int b = 0; b < blocks; ++b) s += partial[((size_t)b * 2 + table) * per_table + e];
  dst[e] += s;  // the tables are shared by every memory block of the model: gradients accumulate
}

// ---- row softmax over a few columns (top-k weights), src/tensor.rs:4521-4602 / autograd.rs:2512-2543 ----
__global__ void softmax_rows_kernel(const float* __restrict__ x, float* __restrict__ y, int rows, int cols) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const float* xr = x + (size_t)row * cols;
  double mx = -INFINITY;
  for (int c = lane; c < cols; c += 32) mx = max(mx, (double)xr[c]);
  mx = warp_max(mx);
  double s = 0.0;
  for (int c = lane; c < cols; c += 32) s += exp((double)xr[c] - mx);
  s = warp_sum(s);
  for (int c = lane; c < cols; c += 32) y[(size_t)row * cols + c] = (float)(exp((double)xr[c] - mx) / s);
}

__global__ void softmax_rows_bwd_kernel(const float* __restrict__ y, const float* __restrict__ gy, float* __restrict__ gx,
                                        int rows, int cols) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  double dot = 0.0;
  for (int c = lane; c < cols; c += 32) dot += (double)y[(size_t)row * cols + c] * (double)gy[(size_t)row * cols + c];
  dot = warp_sum(dot);
  for (int c = lane; c < cols; c += 32) {
    const size_t i = (size_t)row * cols + c;
    gx[i] = (float)((double)y[i] * ((double)gy[i] - dot));
  }
}

// ---- weighted value: out[t,:] = sum_k w[t,k] V[idx[t,k],:] (* gate[t,:] when given)  (src/tensor.rs:3771-3900).
// A warp a token and 128 U columns; at most top_k products a column in f32 (f64 multiply-adds run at a fraction of the f32 rate).
template <int U>
__global__ void __launch_bounds__(128)
weighted_value_rows_kernel(const int64_t* __restrict__ idx, const float* __restrict__ weights, const float* __restrict__ values,
                           float* __restrict__ out, int tokens, int top_k, int rows, int dim, int* __restrict__ status) {
  pdl_begin();
  constexpr int ROWS = GATHER / U;
  const int lane = threadIdx.x & 31, slices = (dim + 128 * U - 1) / (128 * U), w = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int token = w / slices, g0 = (w - token * slices) * 32 * U + lane, groups = dim / 4;
  if (token >= tokens) return;
  float4 acc[U];
#pragma unroll
  for (int u = 0; u < U; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < top_k; k0 += 32) {
    int my_row = -1;
    float my_w = 0.f;
    if (k0 + lane < top_k) {
      const long long r = idx[(size_t)token * top_k + k0 + lane];
      my_w = weights[(size_t)token * top_k + k0 + lane];
      if (r < 0 || r >= rows) atomicExch(status + ST_BAD_INDEX, 1);
      else my_row = (int)r;
    }
    for (int k = 0; k < min(32, top_k - k0); k += ROWS) {
      float4 v[ROWS][U];
      float wt[ROWS];
      bool there[ROWS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        const int r = __shfl_sync(0xffffffffu, my_row, k + j);
        wt[j] = __shfl_sync(0xffffffffu, my_w, k + j);
        there[j] = r >= 0;
#pragma unroll
        for (int u = 0; u < U; ++u) v[j][u] = row_piece(values, r, dim, g0 + u * 32, g0 + u * 32 < groups);
      }
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
        if (there[j])
#pragma unroll
          for (int u = 0; u < U; ++u) add_scaled(acc[u], wt[j], v[j][u]);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (g0 + u * 32 < groups) reinterpret_cast<float4*>(out + (size_t)token * dim)[g0 + u * 32] = acc[u];
}

// The same for rows of more than 1024.
__global__ void weighted_value_fwd_kernel(const int64_t* __restrict__ idx, const float* __restrict__ weights,
                                          const float* __restrict__ values, float* __restrict__ out, int tokens, int top_k,
                                          int rows, int dim, int* __restrict__ status) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= tokens) return;
  for (int c = lane * 4; c < dim; c += 128) {
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    for (int k = 0; k < top_k; ++k) {
      const long long r = idx[(size_t)token * top_k + k];
      if (r < 0 || r >= rows) { if (lane == 0 && c == 0) atomicExch(status + ST_BAD_INDEX, 1); continue; }
      const double w = (double)weights[(size_t)token * top_k + k];
      const float4 v = __ldg(reinterpret_cast<const float4*>(values + (size_t)r * dim + c));
      a0 += w * v.x; a1 += w * v.y; a2 += w * v.z; a3 += w * v.w;
    }
    *reinterpret_cast<float4*>(out + (size_t)token * dim + c) = make_float4((float)a0, (float)a1, (float)a2, (float)a3);
  }
}

// dw[t,k] = dout[t] . V[idx[t,k]];  dV[idx[t,k],:] += w[t,k] dout[t,:] (f32 atomics, repeats accumulate)
// (src/tensor/autograd.rs:2263-2323).  Rows of up to 1024: a warp a token and 128 columns, the warps of a token in one CTA, which adds
// up their parts of dw; f64 sums.
constexpr int VB_WARPS = 8;  // rows of up to 1024
__global__ void weighted_value_bwd_rows_kernel(const int64_t* __restrict__ idx, const float* __restrict__ weights,
                                               const float* __restrict__ values, const float* __restrict__ grad_out,
                                               float* __restrict__ dweights, float* __restrict__ dvalues, int top_k, int rows, int dim) {
  pdl_begin();
  __shared__ double parts[VB_WARPS][32];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, slices = blockDim.x >> 5, gi = slice * 32 + lane;
  const size_t token = blockIdx.x;
  const bool on = gi < dim / 4;
  const float4 g = on ? reinterpret_cast<const float4*>(grad_out + token * dim)[gi] : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < top_k; k0 += 32) {
    int my_row = -1;
    float my_w = 0.f;
    if (k0 + lane < top_k) {
      const long long r = idx[token * top_k + k0 + lane];
      my_w = weights[token * top_k + k0 + lane];
      if (r >= 0 && r < rows) my_row = (int)r;
    }
    const int n = min(32, top_k - k0);
    for (int k = 0; k < n; k += GATHER) {
      float4 v[GATHER];
      int row[GATHER];
#pragma unroll
      for (int j = 0; j < GATHER; ++j) {
        row[j] = __shfl_sync(0xffffffffu, my_row, k + j);
        if (dweights) v[j] = row_piece(values, row[j], dim, gi, on);
      }
      if (dvalues)
#pragma unroll
        for (int j = 0; j < GATHER; ++j) {
          const float w = __shfl_sync(0xffffffffu, my_w, k + j);
          if (on && row[j] >= 0)
            atomicAdd(reinterpret_cast<float4*>(dvalues + (size_t)row[j] * dim) + gi, make_float4(w * g.x, w * g.y, w * g.z, w * g.w));
        }
      if (dweights) {
        double dot[GATHER];
#pragma unroll
        for (int j = 0; j < GATHER; ++j) dot[j] = (double)g.x * v[j].x + (double)g.y * v[j].y + (double)g.z * v[j].z + (double)g.w * v[j].w;
        const double sum = sum8_over_lanes(dot);
        if ((lane & 3) == 0) parts[slice][k + sum8_index()] = sum;
      }
    }
    if (dweights) {
      __syncthreads();
      if (slice == 0 && lane < n && my_row >= 0) {
        double sum = 0.0;
        for (int i = 0; i < slices; ++i) sum += parts[i][lane];
        dweights[token * top_k + k0 + lane] = (float)sum;
      }
      __syncthreads();
    }
  }
}
// The same for longer rows, and for tokens of few slots: a warp a token.
__global__ void weighted_value_bwd_kernel(const int64_t* __restrict__ idx, const float* __restrict__ weights,
                                          const float* __restrict__ values, const float* __restrict__ grad_out,
                                          float* __restrict__ dweights, float* __restrict__ dvalues, int tokens, int top_k,
                                          int rows, int dim) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= tokens) return;
  const float* go = grad_out + (size_t)token * dim;
  for (int k = 0; k < top_k; ++k) {
    const long long r = idx[(size_t)token * top_k + k];
    if (r < 0 || r >= rows) continue;
    const float w = weights[(size_t)token * top_k + k];
    double dot = 0.0;
    for (int c = lane * 4; c < dim; c += 128) {
      const float4 g = *reinterpret_cast<const float4*>(go + c);
      if (dweights) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(values + (size_t)r * dim + c));
        dot += (double)g.x * v.x + (double)g.y * v.y + (double)g.z * v.z + (double)g.w * v.w;
      }
      if (dvalues) atomicAdd(reinterpret_cast<float4*>(dvalues + (size_t)r * dim + c), make_float4(w * g.x, w * g.y, w * g.z, w * g.w));
    }
    if (dweights) {
      dot = warp_sum(dot);
      if (lane == 0) dweights[(size_t)token * top_k + k] = (float)dot;
    }
  }
}

// ---- weighted value backward in row order ---------------------------------------------------------------------
// With many more (token, slot) events than distinct rows (about 26 events per row at the memory-transformer size),
// per-event 16-byte atomics pile onto hot rows in L2.  Events are therefore sorted by row (radix sort over as many key
// bits as the row count needs); a warp takes 32 consecutive sorted events, keeps the value row of the current run and
// the run's gradient sum in registers, and issues one set of atomics per run (and per chunk boundary).  The weight
// gradients, dot(grad_out[token], values[row]), come from the same pass: one 2 KB read of grad_out per event is all
// the traffic that does not stay in registers.
__global__ void value_event_keys_kernel(const int64_t* __restrict__ idx, long long n, int rows, int* __restrict__ keys,
                                        int* __restrict__ events, float* __restrict__ dweights, int* __restrict__ status) {
  pdl_begin();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long r = idx[i];
  const bool bad = r < 0 || r >= rows;
  keys[i] = bad ? rows : (int)r;  // out-of-range slots sort behind every row and are skipped by the row walk,
  events[i] = (int)i;
  if (bad) {                      // so they are reported and their weight gradient is written here
    atomicExch(status + ST_BAD_INDEX, 1);
    if (dweights) dweights[i] = 0.f;
  }
}

// ---- stable radix sort of (row key, event) pairs, eight bits a pass --------------------------------------------
// The row-ordered value backward needs the step's (token, slot) events grouped by table row, events of a row in
// ascending order (that order fixes the f32 summation order of a row's gradient).  Three kernels a pass:
// digit histograms per tile of 2048 keys, an exclusive scan of every digit's row of the digit-major histogram array
// (one block per digit; the scatter adds the scan over the 256 digit totals itself), and a scatter in which every
// warp walks its 256 keys in order, ranking equal digits with warp matches, so the sort is stable.
constexpr int RS_BITS = 8, RS_DIGITS = 1 << RS_BITS, RS_WARPS = 8, RS_THREADS = RS_WARPS * 32;
constexpr int RS_PER_WARP = 256, RS_TILE = RS_WARPS * RS_PER_WARP;

// Digit counts of each warp's keys in shared memory: lanes with equal digits are found with a warp match, the
// lowest of them adds the group's size.
__device__ __forceinline__ void rs_count_tile(const int* __restrict__ keys, long long n, int shift,
                                              int (*wc)[RS_DIGITS]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < RS_WARPS * RS_DIGITS; i += RS_THREADS) (&wc[0][0])[i] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * RS_TILE + (long long)warp * RS_PER_WARP;
  for (int r = 0; r < RS_PER_WARP / 32; ++r) {
    const long long i = base + r * 32 + lane;
    const bool in = i < n;
    const unsigned alive = __ballot_sync(0xffffffffu, in);
    if (in) {
      const int d = (keys[i] >> shift) & (RS_DIGITS - 1);
      const unsigned peers = __match_any_sync(alive, d);
      if (lane == __ffs(peers) - 1) wc[warp][d] += __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
}

__global__ void __launch_bounds__(RS_THREADS)
radix_hist_kernel(const int* __restrict__ keys, long long n, int shift, int* __restrict__ hist, int n_tiles) {
  pdl_begin();
  __shared__ int wc[RS_WARPS][RS_DIGITS];
  rs_count_tile(keys, n, shift, wc);
  for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS) {
    int t = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) t += wc[w][d];
    hist[(size_t)d * n_tiles + blockIdx.x] = t;  // digit-major: a scan over the array gives every (digit, tile) its start
  }
}

// Block d scans row d of the digit-major histogram in place (exclusive) and writes the row's total.
__global__ void __launch_bounds__(RS_THREADS)
radix_scan_rows_kernel(int* __restrict__ hist, int n_tiles, int* __restrict__ totals) {
  pdl_begin();
  __shared__ int warp_sums[RS_WARPS];
  __shared__ int carry;
  int* row = hist + (size_t)blockIdx.x * n_tiles;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n_tiles; base += RS_THREADS) {
    const int i = base + threadIdx.x;
    const int v = i < n_tiles ? row[i] : 0;
    int inc = v;  // inclusive scan within the warp
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += t;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; ++w) before += warp_sums[w];
    if (i < n_tiles) row[i] = before + inc - v;
    __syncthreads();
    if (threadIdx.x == RS_THREADS - 1) carry = before + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(RS_THREADS)
radix_scatter_kernel(const int* __restrict__ keys, const int* __restrict__ vals, int* __restrict__ keys_out,
                     int* __restrict__ vals_out, long long n, int shift, const int* __restrict__ starts,
                     const int* __restrict__ totals, int n_tiles) {
  pdl_begin();
  __shared__ int wc[RS_WARPS][RS_DIGITS];  // counts, then the running output position of each (warp, digit)
  __shared__ int dbase[RS_DIGITS];         // keys with a smaller digit, over all tiles
  __shared__ int wsum[RS_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  static_assert(RS_DIGITS == RS_THREADS, "one thread per digit");
  {
    const int v = totals[threadIdx.x];
    int inc = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    dbase[threadIdx.x] = before + inc - v;
  }
  rs_count_tile(keys, n, shift, wc);
  for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS) {
    int run = dbase[d] + starts[(size_t)d * n_tiles + blockIdx.x];
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      const int c = wc[w][d];
      wc[w][d] = run;
      run += c;
    }
  }
  __syncthreads();
  const long long base = (long long)blockIdx.x * RS_TILE + (long long)warp * RS_PER_WARP;
  for (int r = 0; r < RS_PER_WARP / 32; ++r) {
    const long long i = base + r * 32 + lane;
    const bool in = i < n;
    const unsigned alive = __ballot_sync(0xffffffffu, in);
    if (in) {
      const int key = keys[i];
      const int d = (key >> shift) & (RS_DIGITS - 1);
      const unsigned peers = __match_any_sync(alive, d);
      const int leader = __ffs(peers) - 1;
      int first = 0;
      if (lane == leader) {
        first = wc[warp][d];
        wc[warp][d] = first + __popc(peers);
      }
      first = __shfl_sync(peers, first, leader);
      const int pos = first + __popc(peers & ((1u << lane) - 1u));  // earlier lanes hold earlier keys
      keys_out[pos] = key;
      vals_out[pos] = vals[i];
    }
    __syncwarp();
  }
}

// A warp a chunk of CHUNK events, VPL 16-byte pieces of a row a lane (dim <= VPL * 128).  Columns shared by several warps, as above, were
// slower here (16384 tokens of 32 slots 105 -> 220 us): what a run of equal rows costs to follow is paid by each.
template <int VPL, int CHUNK>
__global__ void __launch_bounds__(128)
weighted_value_bwd_sorted_kernel(const int* __restrict__ keys, const int* __restrict__ events,
                                 const float* __restrict__ weights, const float* __restrict__ values,
                                 const float* __restrict__ grad_out, float* __restrict__ dweights,
                                 float* __restrict__ dvalues, long long n, int top_k, int rows, int dim) {
  // Short chunks are thousands of CTAs: a successor that came in beside them would sit where they ran and leave other SMs empty (the sort of
  // a next call of 65536 events of 512 columns 95 -> 62 us a call; long chunks gain from it: 32 and 131072 events of 64 columns 87 -> 72).
  pdl_begin(CHUNK < 32);
  const int lane = threadIdx.x & 31;
  const long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * CHUNK;
  if (base >= n) return;
  const int groups = dim / 4;
  int my_key = rows, my_event = 0;
  float my_w = 0.f;
  if (lane < CHUNK && base + lane < n) {
    my_key = keys[base + lane];
    my_event = events[base + lane];
    if (my_key < rows) my_w = weights[my_event];
  }
  const int my_token = my_event / top_k;
  float4 acc[VPL], vrow[VPL];
#pragma unroll
  for (int u = 0; u < VPL; ++u) acc[u] = vrow[u] = make_float4(0.f, 0.f, 0.f, 0.f);
  int cur = -1;
  auto flush = [&]() {
    if (cur < 0 || !dvalues) return;
#pragma unroll
    for (int u = 0; u < VPL; ++u) {
      const int gi = u * 32 + lane;
      if (gi < groups) atomicAdd(reinterpret_cast<float4*>(dvalues + (size_t)cur * dim) + gi, acc[u]);
      acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  for (int i0 = 0; i0 < CHUNK; i0 += GATHER) {
    if (__shfl_sync(0xffffffffu, my_key, i0) >= rows) break;  // sorted: nothing valid follows
    double dot[GATHER];
#pragma unroll
    for (int j = 0; j < GATHER; ++j) {
      const int key = __shfl_sync(0xffffffffu, my_key, i0 + j), token = __shfl_sync(0xffffffffu, my_token, i0 + j);
      const float w = __shfl_sync(0xffffffffu, my_w, i0 + j);
      dot[j] = 0.0;
      if (key >= rows) continue;
      if (key != cur) {
        flush();
        cur = key;
        if (dweights) {
#pragma unroll
          for (int u = 0; u < VPL; ++u) vrow[u] = row_piece(values, key, dim, u * 32 + lane, u * 32 + lane < groups);
        }
      }
      float share = 0.f;  // this lane's part of the dot product in f32, the 32 parts are summed in f64
#pragma unroll
      for (int u = 0; u < VPL; ++u) {
        const float4 g = row_piece(grad_out, token, dim, u * 32 + lane, u * 32 + lane < groups);
        share = fmaf(g.x, vrow[u].x, share); share = fmaf(g.y, vrow[u].y, share);
        share = fmaf(g.z, vrow[u].z, share); share = fmaf(g.w, vrow[u].w, share);
        acc[u].x = fmaf(w, g.x, acc[u].x); acc[u].y = fmaf(w, g.y, acc[u].y);
        acc[u].z = fmaf(w, g.z, acc[u].z); acc[u].w = fmaf(w, g.w, acc[u].w);
      }
      dot[j] = (double)share;
    }
    if (dweights) {
      const double sum = sum8_over_lanes(dot);
      const int at = i0 + sum8_index();
      const int event = __shfl_sync(0xffffffffu, my_event, at), key = __shfl_sync(0xffffffffu, my_key, at);
      if ((lane & 3) == 0 && key < rows) dweights[event] = (float)sum;
    }
  }
  flush();
}

// ---- access counts: counts[r] += occurrences of r among the selected rows (kernels.ptx:813-886) ---------------
__global__ void access_count_rows_kernel(const int64_t* __restrict__ selected, long long n, int rows,
                                         unsigned long long* __restrict__ counts, int* __restrict__ status) {
  pdl_begin();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const long long r = selected[i];
    if (r < 0 || r >= rows) { atomicExch(status + ST_BAD_INDEX, 1); continue; }
    atomicAdd(counts + r, 1ull);
  }
}

// ---- row-set AdamW (src/nn.rs:2256-2323, :2899-2939; kernels.ptx:537-811) -----------------------------------
__global__ void mark_rows_kernel(const int64_t* __restrict__ selected, long long n, unsigned char* __restrict__ flags,
                                 const unsigned char* __restrict__ row_mask, int rows, int* __restrict__ status) {
  pdl_begin();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long r = selected[i];
  if (r < 0 || r >= rows) { atomicExch(status + ST_BAD_INDEX, 1); return; }
  if (row_mask == nullptr || row_mask[r]) flags[r] = 1;
}

__device__ __forceinline__ void adamw_one(float& p, float g, float& m, float& v, const hl_adamw_params& hp) {
  const float gd = __fadd_rn(__fmul_rn(g, hp.clip_scale), __fmul_rn(p, hp.weight_decay));
  m = __fadd_rn(__fmul_rn(hp.beta1, m), __fmul_rn(__fsub_rn(1.0f, hp.beta1), gd));
  v = __fadd_rn(__fmul_rn(hp.beta2, v), __fmul_rn(__fsub_rn(1.0f, hp.beta2), __fmul_rn(gd, gd)));
  const float upd = __fdiv_rn(__fdiv_rn(m, hp.bias_correction1), __fadd_rn(__fsqrt_rn(__fdiv_rn(v, hp.bias_correction2)), hp.eps));
  p = __fsub_rn(p, __fmul_rn(hp.lr, upd));
}

// One warp per flagged row; clears the flag and (optionally) the gradient row it consumed.
__global__ void sparse_adamw_rows_kernel(float* __restrict__ param, float* __restrict__ grad, float* __restrict__ m,
                                         float* __restrict__ v, unsigned char* __restrict__ flags, int rows, int row_dim,
                                         const hl_adamw_params hp, int zero_grad_rows) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows || !flags[row]) return;
  const size_t base = (size_t)row * row_dim;
  for (int c = lane; c < row_dim; c += 32) {
    float p = param[base + c], mm = m[base + c], vv = v[base + c];
    adamw_one(p, grad[base + c], mm, vv, hp);
    param[base + c] = p; m[base + c] = mm; v[base + c] = vv;
    if (zero_grad_rows) grad[base + c] = 0.f;
  }
  __syncwarp();
  if (lane == 0) flags[row] = 0;
}

// Sum of squares of the flagged gradient rows (a set: a row counts once however often it was selected); one warp per flagged
// row, flags cleared on the way out.  A block walks many rows and adds once: an f64 addition to the one result per row took longer
// than reading the rows (262144 rows of 512, a third of them flagged: 62 us).
__global__ void __launch_bounds__(256)
flagged_rows_sum_squares_kernel(const float* __restrict__ grad, unsigned char* __restrict__ flags, int rows, int row_dim, bool vec,
                                double* __restrict__ out) {
  pdl_begin();
  __shared__ double sm[32];
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  double s = 0.0;
  for (int row = blockIdx.x * warps + (threadIdx.x >> 5); row < rows; row += gridDim.x * warps) {
    if (!flags[row]) continue;
    const float* g = grad + (size_t)row * row_dim;
    if (vec) {
#pragma unroll 4
      for (int c = lane * 4; c < row_dim; c += 128) {
        const float4 x = *reinterpret_cast<const float4*>(g + c);
        s += ((double)x.x * (double)x.x + (double)x.y * (double)x.y) + ((double)x.z * (double)x.z + (double)x.w * (double)x.w);
      }
    } else {
      for (int c = lane; c < row_dim; c += 32) s += (double)g[c] * (double)g[c];
    }
    __syncwarp();
    if (lane == 0) flags[row] = 0;
  }
  s = block_sum(s, sm);
  if (threadIdx.x == 0 && s != 0.0) atomicAdd(out, s);
}

// Ascending indices of the non-zero bytes of a mask, and their count.  One CTA: every thread counts a contiguous
// span, an exclusive scan over the spans gives its write position.
__global__ void __launch_bounds__(1024)
mask_to_indices_kernel(const unsigned char* __restrict__ mask, int rows, int64_t* __restrict__ out, int* __restrict__ count) {
  pdl_begin();
  __shared__ int span_start[1025];
  const int per = (rows + 1023) / 1024;
  const int lo = min(rows, (int)threadIdx.x * per), hi = min(rows, lo + per);
  int mine = 0;
  for (int r = lo; r < hi; ++r) mine += mask[r] != 0;
  span_start[threadIdx.x + 1] = mine;
  if (threadIdx.x == 0) span_start[0] = 0;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i <= 1024; ++i) span_start[i] += span_start[i - 1];
  __syncthreads();
  int at = span_start[threadIdx.x];
  for (int r = lo; r < hi; ++r)
    if (mask[r]) out[at++] = r;
  if (threadIdx.x == 0) *count = span_start[1024];
}

// dst[i,:] = src[idx[i],:] (gather) or dst[idx[i],:] = src[i,:] (scatter); one warp per row, 16-byte accesses.
__global__ void move_rows_kernel(const float* __restrict__ src, const int64_t* __restrict__ idx, const int* __restrict__ count_dev,
                                 int n_max, int dim, float* __restrict__ dst, int scatter) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int n = count_dev ? min(*count_dev, n_max) : n_max;
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += gridDim.x * (blockDim.x >> 5)) {
    const size_t row = (size_t)idx[i];
    const float4* s4 = reinterpret_cast<const float4*>(src + (scatter ? (size_t)i : row) * dim);
    float4* d4 = reinterpret_cast<float4*>(dst + (scatter ? row : (size_t)i) * dim);
    for (int c = lane; c < dim / 4; c += 32) d4[c] = s4[c];
  }
}

// Half-table rows and a row of queries (or their gradient) `ld` apart that the sixteen-byte forms take.
bool rows_of_16_bytes(int key_dim, long long ld, const void* query, const void* left, const void* right) {
  return key_dim % 8 == 0 && key_dim <= 1024 && ld % 4 == 0 &&
         ((reinterpret_cast<uintptr_t>(query) | reinterpret_cast<uintptr_t>(left) | reinterpret_cast<uintptr_t>(right)) & 15) == 0;
}

int check_memory_dims(int tokens, int top_k, int dim, const char* who) {
  HL_REQUIRE(tokens > 0 && top_k > 0 && dim > 0, std::string(who) + ": requires non-zero tokens/top_k/dim");
  return HL_OK;
}

}  // namespace
}  // namespace hl

using namespace hl;

namespace hl {
int product_key_topk_impl(hl_ctx* ctx, const float* left_scores, const float* right_scores, int64_t* out, int tokens, int side, int top_k,
                          int beam, int64_t* kept, const long long* kept_row) {
  HL_REQUIRE(ctx && left_scores && right_scores && out, "hl_product_key_topk_from_side_scores: null argument");
  HL_REQUIRE(tokens > 0 && side > 0, "hl_product_key_topk_from_side_scores: requires non-zero tokens/side");
  HL_REQUIRE(side <= 2048, "hl_product_key_topk_from_side_scores: side must be at most 2048");
  HL_REQUIRE(beam > 0 && beam <= 32 && beam <= side, "hl_product_key_topk_from_side_scores: beam must be in [1, min(32, side)]");
  HL_REQUIRE(top_k > 0 && top_k <= beam * beam, "hl_product_key_topk_from_side_scores: top_k must be in [1, beam^2]");
  if (side <= 512)
    pdl(product_key_topk_kernel<16>, ceil_div(tokens, 4), 128, 0, ctx->stream)(left_scores, right_scores, out, tokens, side,
                                                                              top_k, beam, ctx->status_dev, kept, kept_row);
  else
    pdl(product_key_topk_kernel<PK_MAX_PER_LANE>, ceil_div(tokens, 4), 128, 0, ctx->stream)(
        left_scores, right_scores, out, tokens, side, top_k, beam, ctx->status_dev, kept, kept_row);
  HL_LAUNCH_CHECK("product_key_topk_kernel");
  count_launch(ctx);
  return HL_OK;
}

bool product_key_lookup_takes(int side, int key_dim, int beam) {
  return side % 8 == 0 && side <= 32 * LK_PER_LANE && key_dim % 64 == 0 && key_dim <= 1024 && beam <= 32;
}
size_t product_key_pieces_bytes(int side, int key_dim) { return (size_t)3 * side * key_dim * sizeof(__nv_bfloat16) + 256; }
int product_key_pieces(hl_ctx* ctx, const float* left_keys, const float* right_keys, int side, int key_dim, void* pieces) {
  int* norms = static_cast<int*>(pieces);
  HL_CUDA(cudaMemsetAsync(norms, 0, 2 * sizeof(int), ctx->stream));
  pdl(key_pieces_kernel, ceil_div(2 * side, 8), 256, 0, ctx->stream)(left_keys, right_keys,
                                                                    reinterpret_cast<__nv_bfloat16*>(static_cast<uint8_t*>(pieces) + 256), norms,
                                                                    side, key_dim / 2);
  HL_LAUNCH_CHECK("key_pieces_kernel");
  count_launch(ctx);
  return HL_OK;
}
int product_key_lookup(hl_ctx* ctx, const float* query, const float* left_keys, const float* right_keys, const void* pieces,
                       __nv_bfloat16* query_pieces, float* left_approx, float* right_approx, int64_t* out, int tokens, int side, int key_dim,
                       int top_k, int beam) {
  const int half = key_dim / 2;
  pdl(query_pieces_kernel, (unsigned)ceil_div_ll((long long)tokens * (half / 4), 256), 256, 0, ctx->stream)(query, key_dim, query_pieces, tokens, half);
  HL_LAUNCH_CHECK("query_pieces_kernel");
  const __nv_bfloat16* keys = reinterpret_cast<const __nv_bfloat16*>(static_cast<const uint8_t*>(pieces) + 256);
  hl_gemm_desc d{};
  d.m = tokens; d.n = side; d.k = 3 * half;
  d.a_layout = d.b_layout = HL_K_MAJOR;
  d.lda = 4 * half; d.ldb = 3 * half; d.ldc = side;
  d.out_dtype = HL_F32;
  d.a_k_period = 2 * half;
  for (int sd = 0; sd < 2; ++sd) {
    const int rc = gemm_bf16_ctx(ctx, &d, query_pieces + sd * 2 * half, keys + (size_t)sd * side * 3 * half, sd ? right_approx : left_approx, nullptr,
                                 nullptr, nullptr);
    if (rc != HL_OK) return rc;
  }
  const size_t smem = sizeof(float) * 4 * (size_t)(2 * half + 32 * LK_LD);
  HL_ALLOW_SHARED(ctx, sizeof(float) * 4 * (2 * 512 + 32 * LK_LD), product_key_lookup_kernel);
  pdl(product_key_lookup_kernel, ceil_div(tokens, 4), 128, smem, ctx->stream)(left_approx, right_approx, query, key_dim, left_keys, right_keys,
                                                                             static_cast<const float*>(pieces), out, tokens, side, half, top_k,
                                                                             beam, ctx->status_dev);
  HL_LAUNCH_CHECK("product_key_lookup_kernel");
  count_launch(ctx, 2);
  return HL_OK;
}
}  // namespace hl

extern "C" {

int hl_topk_rows_f32(hl_ctx* ctx, const float* scores, int64_t* out, int rows, int cols, int k) {
  HL_REQUIRE(ctx && scores && out, "hl_topk_rows_f32: null argument");
  HL_REQUIRE(rows > 0 && cols > 0, "hl_topk_rows_f32: requires non-zero rows/cols");
  HL_REQUIRE(k > 0 && k <= cols, "hl_topk_rows_f32: k must be in [1, cols]");
  HL_REQUIRE(cols <= 2048, "hl_topk_rows_f32: at most 2048 columns");
  pdl(topk_rows_kernel, ceil_div(rows, 4), 128, 0, ctx->stream)(scores, out, rows, cols, k);
  HL_LAUNCH_CHECK("topk_rows_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_product_key_side_scores_f32(hl_ctx* ctx, const float* query, long long ld_query, const float* left_keys,
                                   const float* right_keys, float* left_scores, float* right_scores, int tokens, int side,
                                   int key_dim) {
  HL_REQUIRE(ctx && query && left_keys && right_keys && left_scores && right_scores, "hl_product_key_side_scores_f32: null argument");
  HL_REQUIRE(tokens > 0 && side > 0 && key_dim > 0, "hl_product_key_side_scores_f32: requires non-zero sizes");
  HL_REQUIRE(key_dim % 2 == 0, "product-key memory lookup requires even memory_key_dim, got " + std::to_string(key_dim));
  HL_REQUIRE(ld_query >= key_dim, "hl_product_key_side_scores_f32: query row stride smaller than key_dim");
  const int half = key_dim / 2;
  // Both tables in one launch: a second one would come in while the first runs, and its blocks, four to an SM, would sit on the few
  // SMs that the first one leaves over (2048 tokens: 72 us a table instead of 43).
  dim3 grid(ceil_div(side, SS_K), ceil_div(tokens, SS_T), 2);
  pdl(side_scores_kernel, grid, 256, 0, ctx->stream)(query, ld_query, left_keys, right_keys, left_scores, right_scores, tokens, side,
                                                     half, -0.0f);
  HL_LAUNCH_CHECK("side_scores_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_product_key_lookup(hl_ctx* ctx, const float* query, const float* left_keys, const float* right_keys, void* pieces, void* query_pieces,
                          float* left_approx, float* right_approx, int64_t* out, int tokens, int side, int key_dim, int top_k, int beam) {
  HL_REQUIRE(ctx && query && left_keys && right_keys && pieces && query_pieces && left_approx && right_approx && out,
             "hl_product_key_lookup: null argument");
  HL_REQUIRE(tokens > 0 && side > 0 && key_dim > 0, "hl_product_key_lookup: requires non-zero sizes");
  HL_REQUIRE(beam > 0 && beam <= 32 && beam <= side, "hl_product_key_lookup: beam must be in [1, min(32, side)]");
  HL_REQUIRE(top_k > 0 && top_k <= beam * beam, "hl_product_key_lookup: top_k must be in [1, beam^2]");
  HL_REQUIRE(product_key_lookup_takes(side, key_dim, beam),
             "hl_product_key_lookup: side must be a multiple of 8 up to 512, key_dim a multiple of 64 up to 1024");
  HL_REQUIRE(((reinterpret_cast<uintptr_t>(query) | reinterpret_cast<uintptr_t>(left_keys) | reinterpret_cast<uintptr_t>(right_keys) |
               reinterpret_cast<uintptr_t>(pieces) | reinterpret_cast<uintptr_t>(query_pieces) | reinterpret_cast<uintptr_t>(left_approx) |
               reinterpret_cast<uintptr_t>(right_approx)) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0,
             "hl_product_key_lookup: pointers must be 16-byte aligned");
  const int rc = product_key_pieces(ctx, left_keys, right_keys, side, key_dim, pieces);
  if (rc != HL_OK) return rc;
  return product_key_lookup(ctx, query, left_keys, right_keys, pieces, static_cast<__nv_bfloat16*>(query_pieces), left_approx, right_approx, out,
                            tokens, side, key_dim, top_k, beam);
}

int hl_product_key_topk_from_side_scores(hl_ctx* ctx, const float* left_scores, const float* right_scores, int64_t* out,
                                         int tokens, int side, int top_k, int beam) {
  return hl::product_key_topk_impl(ctx, left_scores, right_scores, out, tokens, side, top_k, beam, nullptr, nullptr);
}

int hl_product_key_split_rows(hl_ctx* ctx, const int64_t* rows, int64_t* left, int64_t* right, long long n, int side) {
  HL_REQUIRE(ctx && rows && left && right, "hl_product_key_split_rows: null argument");
  HL_REQUIRE(n > 0 && side > 0, "hl_product_key_split_rows: requires non-zero rows/side");
  pdl(split_rows_kernel, (unsigned)ceil_div_ll(n, 256), 256, 0, ctx->stream)(rows, left, right, n, side);
  HL_LAUNCH_CHECK("split_rows_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_memory_selected_scores_forward(hl_ctx* ctx, const int64_t* indices, const float* query, long long ld_query,
                                      const float* left_or_keys, const float* right_keys, float* scores, int tokens,
                                      int top_k, int side, int key_dim, int slots) {
  HL_REQUIRE(ctx && indices && query && left_or_keys && scores, "hl_memory_selected_scores_forward: null argument");
  int rc = check_memory_dims(tokens, top_k, key_dim, "hl_memory_selected_scores_forward");
  if (rc != HL_OK) return rc;
  HL_REQUIRE(side == 0 || (right_keys && key_dim % 2 == 0 && (long long)side * side == slots),
             "hl_memory_selected_scores_forward: product-key mode needs both half tables, even key_dim and square slots");
  if (side > 0 && rows_of_16_bytes(key_dim, ld_query, query, left_or_keys, right_keys)) {
    auto launch = [&](auto kern) {
      const int log_warps = top_k <= GATHER ? 0 : top_k <= 2 * GATHER ? 1 : 2;  // a token's
      pdl(kern, (unsigned)ceil_div_ll((long long)tokens << log_warps, 4), 128, 0, ctx->stream).streaming(4.0 * tokens * top_k * key_dim)(
          indices, query, ld_query, left_or_keys, right_keys, scores, tokens, top_k, side, key_dim, slots, log_warps, ctx->status_dev);
    };
    if (key_dim <= 128) launch(selected_scores_rows_kernel<1>);
    else if (key_dim <= 256) launch(selected_scores_rows_kernel<2>);
    else if (key_dim <= 512) launch(selected_scores_rows_kernel<4>);
    else launch(selected_scores_rows_kernel<8>);
  } else {
    pdl(selected_scores_fwd_kernel, ceil_div(tokens, 4), 128, 0, ctx->stream).streaming(4.0 * tokens * top_k * key_dim)(
        indices, query, ld_query, left_or_keys, right_keys, scores, tokens, top_k, side, key_dim, slots, ctx->status_dev);
  }
  HL_LAUNCH_CHECK("selected_scores_fwd_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_memory_selected_scores_backward(hl_ctx* ctx, const int64_t* indices, const float* query, long long ld_query,
                                       const float* left_or_keys, const float* right_keys, const float* grad_scores,
                                       float* grad_query, long long ld_grad_query, float* grad_left_or_keys,
                                       float* grad_right_keys, int tokens, int top_k, int side, int key_dim, int slots) {
  HL_REQUIRE(ctx && indices && query && left_or_keys && grad_scores, "hl_memory_selected_scores_backward: null argument");
  int rc = check_memory_dims(tokens, top_k, key_dim, "hl_memory_selected_scores_backward");
  if (rc != HL_OK) return rc;
  HL_REQUIRE(side == 0 || (right_keys && key_dim % 2 == 0), "hl_memory_selected_scores_backward: product-key mode needs both half tables");
  const int half = key_dim / 2;
  const KeyGradient keys{indices, query, ld_query, grad_scores, tokens, top_k, side, half, slots};
  const bool half_keys = side > 0 && (grad_left_or_keys || grad_right_keys);
  int token_blocks = half_keys ? key_gradient_shares(ctx, keys) : 0;
  // the tensor-core form's scratch holds the queries' pieces as well: where the device has no room for them, the f32 form
  const bool tensor = token_blocks > 0 && try_workspace(ctx, key_gradient_bytes(keys, token_blocks));
  int* clear = tensor ? static_cast<int*>(ctx->workspace) : nullptr;
  const bool alone = side > 0 && !grad_query;  // the tables' gradients, whose kernels come below
  if (side > 0 && !alone && rows_of_16_bytes(key_dim, ld_grad_query, grad_query, left_or_keys, right_keys)) {
    by_pieces(top_k, key_dim, [&](auto pieces) {
      constexpr int U = decltype(pieces)::value;
      pdl(selected_query_gradient_kernel<U>, (unsigned)ceil_div_ll((long long)tokens * ceil_div(key_dim, 128 * U), 4), 128, 0, ctx->stream)(
          indices, left_or_keys, right_keys, grad_scores, grad_query, ld_grad_query, tokens, top_k, side, key_dim, slots, clear);
    });
    HL_LAUNCH_CHECK("selected_query_gradient_kernel");
    count_launch(ctx);
  } else if (!alone || clear) {  // `alone`: a block that clears the word (a memset in front of dependent launches: 2320 us a step of sparse fine-tuning, 2275)
    pdl(selected_scores_bwd_kernel, alone ? 1 : ceil_div(tokens, 4), 128, 0, ctx->stream)(
        indices, query, ld_query, left_or_keys, right_keys, grad_scores, grad_query, ld_grad_query, grad_left_or_keys,
        grad_right_keys, tokens, top_k, side, key_dim, slots, clear);
    HL_LAUNCH_CHECK("selected_scores_bwd_kernel");
    count_launch(ctx);
  }
  if (half_keys) {
    const int col_blocks = ceil_div(half, DK_COLS), row_blocks = ceil_div(side, DK_ROWS);
    if (!tensor) {
      token_blocks = std::max(1, std::min(ceil_div(tokens, 64), std::max(1, (2 * ctx->sm_count) / (2 * col_blocks * row_blocks))));
      rc = ensure_workspace(ctx, sizeof(float) * (size_t)token_blocks * 2 * side * half);
      if (rc != HL_OK) return rc;
    }
    float* partial = reinterpret_cast<float*>(ctx->workspace);
    if (tensor) {
      rc = key_gradient_run(ctx, keys, token_blocks, ctx->workspace, &partial);
      if (rc != HL_OK) return rc;
    } else {
      const size_t smem = sizeof(float) * (size_t)DK_TOKENS * (DK_ROWS + DK_COLS);
      HL_ALLOW_SHARED(ctx, smem, product_key_dkeys_kernel);
      pdl(product_key_dkeys_kernel, dim3(token_blocks, col_blocks * row_blocks, 2), 256, smem, ctx->stream)(
          indices, query, ld_query, grad_scores, partial, tokens, top_k, side, half, slots, ceil_div(tokens, token_blocks), col_blocks);
      HL_LAUNCH_CHECK("product_key_dkeys_kernel");
      count_launch(ctx);
    }
    const size_t total = 2 * (size_t)side * half;
    pdl(fold_key_partials_kernel, (unsigned)((total + 255) / 256), 256, 0, ctx->stream)(partial, grad_left_or_keys, grad_right_keys,
                                                                                       token_blocks, side, half);
    HL_LAUNCH_CHECK("fold_key_partials_kernel");
    count_launch(ctx);
  }
  return HL_OK;
}

int hl_softmax_rows_f32(hl_ctx* ctx, const float* x, float* y, int rows, int cols) {
  HL_REQUIRE(ctx && x && y, "hl_softmax_rows_f32: null argument");
  HL_REQUIRE(rows > 0 && cols > 0, "hl_softmax_rows_f32: requires non-zero rows/cols");
  pdl(softmax_rows_kernel, ceil_div(rows, 4), 128, 0, ctx->stream)(x, y, rows, cols);
  HL_LAUNCH_CHECK("softmax_rows_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_softmax_rows_backward_f32(hl_ctx* ctx, const float* y, const float* grad_y, float* grad_x, int rows, int cols) {
  HL_REQUIRE(ctx && y && grad_y && grad_x, "hl_softmax_rows_backward_f32: null argument");
  HL_REQUIRE(rows > 0 && cols > 0, "hl_softmax_rows_backward_f32: requires non-zero rows/cols");
  pdl(softmax_rows_bwd_kernel, ceil_div(rows, 4), 128, 0, ctx->stream)(y, grad_y, grad_x, rows, cols);
  HL_LAUNCH_CHECK("softmax_rows_bwd_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_memory_weighted_value_forward(hl_ctx* ctx, const int64_t* indices, const float* weights, const float* values,
                                     float* out, int tokens, int top_k, int rows, int dim) {
  HL_REQUIRE(ctx && indices && weights && values && out, "hl_memory_weighted_value_forward: null argument");
  int rc = check_memory_dims(tokens, top_k, dim, "hl_memory_weighted_value_forward");
  if (rc != HL_OK) return rc;
  HL_REQUIRE(rows > 0 && dim % 4 == 0, "hl_memory_weighted_value_forward: non-zero rows/row_dim, row_dim a multiple of 4");
  if (dim <= 1024)
    by_pieces(top_k, dim, [&](auto pieces) {
      constexpr int U = decltype(pieces)::value;
      pdl(weighted_value_rows_kernel<U>, (unsigned)ceil_div_ll((long long)tokens * ceil_div(dim, 128 * U), 4), 128, 0, ctx->stream)(
          indices, weights, values, out, tokens, top_k, rows, dim, ctx->status_dev);
    });
  else
    pdl(weighted_value_fwd_kernel, ceil_div(tokens, 4), 128, 0, ctx->stream)(indices, weights, values, out, tokens, top_k, rows, dim,
                                                                            ctx->status_dev);
  HL_LAUNCH_CHECK("weighted_value_fwd_kernel");
  count_launch(ctx);
  return HL_OK;
}

}  // extern "C" (reopened below)

namespace hl {
// Row order of a step's (token, slot) events (see weighted_value_bwd_sorted_kernel).
bool value_events_ordered(long long n, int rows, int dim) { return n >= 32768 && n < (1ll << 31) - 64 && dim <= 1024 && rows < (1 << 30); }
static size_t value_array_bytes(long long n) { return ((size_t)n * sizeof(int) + 255) & ~size_t(255); }
size_t value_sort_bytes(long long n) { return 2 * value_array_bytes(n); }
size_t value_order_scratch_bytes(long long n) {  // keys and events of every other pass; digit counts of every tile, then their totals
  return 2 * value_array_bytes(n) + (((size_t)RS_DIGITS * ((size_t)ceil_div_ll(n, RS_TILE) + 1) * sizeof(int) + 255) & ~size_t(255));
}
int value_sort(hl_ctx* ctx, const int64_t* indices, long long n, int rows, int* keys, int* events, void* scratch, float* grad_weights) {
  uint8_t* ws = static_cast<uint8_t*>(scratch);
  const size_t arr = value_array_bytes(n);
  int *keys_a = keys, *ev_a = events, *keys_b = reinterpret_cast<int*>(ws), *ev_b = reinterpret_cast<int*>(ws + arr);
  int* hist = reinterpret_cast<int*>(ws + 2 * arr);
  const int n_tiles = (int)ceil_div_ll(n, RS_TILE);
  int end_bit = 1;
  while ((1ll << end_bit) <= rows) ++end_bit;  // the sentinel key `rows` must sort last
  const int passes = ceil_div(end_bit, RS_BITS);
  if (passes & 1) {  // so that the last pass writes where the caller wants it
    std::swap(keys_a, keys_b);
    std::swap(ev_a, ev_b);
  }
  pdl(value_event_keys_kernel, (unsigned)ceil_div_ll(n, 256), 256, 0, ctx->stream)(indices, n, rows, keys_a, ev_a, grad_weights, ctx->status_dev);
  HL_LAUNCH_CHECK("value_event_keys_kernel");
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * RS_BITS;
    pdl(radix_hist_kernel, n_tiles, RS_THREADS, 0, ctx->stream)(keys_a, n, shift, hist, n_tiles);
    HL_LAUNCH_CHECK("radix_hist_kernel");
    int* totals = hist + (size_t)RS_DIGITS * n_tiles;
    pdl(radix_scan_rows_kernel, RS_DIGITS, RS_THREADS, 0, ctx->stream)(hist, n_tiles, totals);
    HL_LAUNCH_CHECK("radix_scan_rows_kernel");
    pdl(radix_scatter_kernel, n_tiles, RS_THREADS, 0, ctx->stream)(keys_a, ev_a, keys_b, ev_b, n, shift, hist, totals, n_tiles);
    HL_LAUNCH_CHECK("radix_scatter_kernel");
    std::swap(keys_a, keys_b);
    std::swap(ev_a, ev_b);
  }
  count_launch(ctx, 1 + 3 * passes);
  return HL_OK;
}
int weighted_value_backward_ordered(hl_ctx* ctx, const int* keys, const int* events, const float* weights, const float* values,
                                    const float* grad_out, float* grad_weights, float* grad_values, long long n, int top_k, int rows, int dim) {
  auto launch = [&](auto kern, int chunk) {
    pdl(kern, (unsigned)ceil_div_ll(ceil_div_ll(n, chunk), 4), 128, 0, ctx->stream)(keys, events, weights, values, grad_out, grad_weights,
                                                                                    grad_values, n, top_k, rows, dim);
  };
  // Short chunks where the warps of long ones would not fill the chip, us a call with its sort, long / short: 65536 events of 512 columns
  // 118 / 60 and 72 / 50 (many and few distinct rows), 131072 132 / 104 and 73 / 82, of 64 columns 72 / 98 and 61 / 75, 262144 90 / 146 and 80 / 114
  // (256 columns); rows of 1024 columns: 32768 events 96 / 74 and 59 / 55, 65536 135 / 135 and 80 / 77 to 138 / 153 and 80 / 81.
  const bool few = n < (dim > 512 ? 50000 : 100000);
  if (dim <= 512) few ? launch(weighted_value_bwd_sorted_kernel<4, 8>, 8) : launch(weighted_value_bwd_sorted_kernel<4, 32>, 32);
  else few ? launch(weighted_value_bwd_sorted_kernel<8, 8>, 8) : launch(weighted_value_bwd_sorted_kernel<8, 32>, 32);
  HL_LAUNCH_CHECK("weighted_value_bwd_sorted_kernel");
  count_launch(ctx);
  return HL_OK;
}
}  // namespace hl

extern "C" {

int hl_memory_weighted_value_backward(hl_ctx* ctx, const int64_t* indices, const float* weights, const float* values,
                                      const float* grad_out, float* grad_weights, float* grad_values, int tokens,
                                      int top_k, int rows, int dim) {
  HL_REQUIRE(ctx && indices && weights && values && grad_out, "hl_memory_weighted_value_backward: null argument");
  int rc = check_memory_dims(tokens, top_k, dim, "hl_memory_weighted_value_backward");
  if (rc != HL_OK) return rc;
  HL_REQUIRE(rows > 0 && dim % 4 == 0, "hl_memory_weighted_value_backward: non-zero rows/row_dim, row_dim a multiple of 4");
  const long long n = (long long)tokens * top_k;
  if (grad_values && value_events_ordered(n, rows, dim)) {
    rc = ensure_workspace(ctx, value_sort_bytes(n) + value_order_scratch_bytes(n));
    if (rc != HL_OK) return rc;
    uint8_t* ws = reinterpret_cast<uint8_t*>(ctx->workspace);
    int *keys = reinterpret_cast<int*>(ws), *events = reinterpret_cast<int*>(ws + value_sort_bytes(n) / 2);
    rc = value_sort(ctx, indices, n, rows, keys, events, ws + value_sort_bytes(n), grad_weights);
    if (rc != HL_OK) return rc;
    return weighted_value_backward_ordered(ctx, keys, events, weights, values, grad_out, grad_weights, grad_values, n, top_k, rows, dim);
  }
  // A CTA a token pays from a few slots on; us, a warp a token / a CTA a token: 16384 tokens of 1 slot of 512 columns 11.4 / 36, 8192 of 3
  // 14.9 / 20.7, 2048 of 2 5.8 / 6.3, of 3 7.7 / 6.8, 1024 of 2 4.0 / 4.0, 512 of 3 4.7 / 3.4, 64 of 2 3.5 / 2.6.
  const bool by_warp = dim > 1024 || top_k == 1 || (top_k <= 3 && tokens >= 64 << (2 * top_k));
  if (!by_warp)
    pdl(weighted_value_bwd_rows_kernel, tokens, 32 * ceil_div(dim, 128), 0, ctx->stream)(indices, weights, values, grad_out, grad_weights,
                                                                                        grad_values, top_k, rows, dim);
  else
    pdl(weighted_value_bwd_kernel, ceil_div(tokens, 4), 128, 0, ctx->stream)(indices, weights, values, grad_out, grad_weights, grad_values,
                                                                            tokens, top_k, rows, dim);
  HL_LAUNCH_CHECK("weighted_value_bwd_kernel");
  count_launch(ctx);
  return HL_OK;
}

}  // extern "C" (reopened below)

namespace hl {
// Stream-explicit forms, used by the data-parallel row exchange on the collective stream.
int mark_rows_on(hl_ctx* ctx, cudaStream_t stream, const int64_t* selected_rows, long long n_selected, const unsigned char* row_mask,
                 unsigned char* flags, int rows) {
  if (n_selected <= 0) return HL_OK;
  pdl(mark_rows_kernel, (unsigned)ceil_div_ll(n_selected, 256), 256, 0, stream)(selected_rows, n_selected, flags, row_mask, rows,
                                                                             ctx->status_dev);
  HL_LAUNCH_CHECK("mark_rows_kernel");
  count_launch(ctx);
  return HL_OK;
}
int mask_to_indices_on(hl_ctx* ctx, cudaStream_t stream, const unsigned char* mask, int rows, int64_t* out, int* count_dev) {
  pdl(mask_to_indices_kernel, 1, 1024, 0, stream)(mask, rows, out, count_dev);
  HL_LAUNCH_CHECK("mask_to_indices_kernel");
  count_launch(ctx);
  return HL_OK;
}
int move_rows_on(hl_ctx* ctx, cudaStream_t stream, const float* src, const int64_t* idx, const int* count_dev, int n_max, int dim,
                 float* dst, bool scatter) {
  if (n_max <= 0) return HL_OK;
  const int blocks = std::min(ceil_div(n_max, 8), ctx->sm_count * 8);
  pdl(move_rows_kernel, blocks, 256, 0, stream)(src, idx, count_dev, n_max, dim, dst, scatter ? 1 : 0);
  HL_LAUNCH_CHECK("move_rows_kernel");
  count_launch(ctx);
  return HL_OK;
}
}  // namespace hl

extern "C" {

int hl_memory_access_count_rows_i64_u64(hl_ctx* ctx, const int64_t* selected_rows, long long n_selected, int slots,
                                        unsigned long long* counts) {
  HL_REQUIRE(ctx && counts, "hl_memory_access_count_rows_i64_u64: null argument");
  HL_REQUIRE(slots > 0, "memory_access_count_rows_i64_u64 requires non-zero memory_slots");
  HL_REQUIRE(n_selected >= 0 && (n_selected == 0 || selected_rows), "hl_memory_access_count_rows_i64_u64: null selected rows");
  if (n_selected == 0) return HL_OK;
  const unsigned blocks = (unsigned)std::min<long long>(ceil_div_ll(n_selected, 256), (long long)ctx->sm_count * 16);
  pdl(access_count_rows_kernel, blocks, 256, 0, ctx->stream)(selected_rows, n_selected, slots, counts, ctx->status_dev);
  HL_LAUNCH_CHECK("access_count_rows_kernel");
  count_launch(ctx);
  return HL_OK;
}

int hl_mark_rows_u8(hl_ctx* ctx, const int64_t* selected_rows, long long n_selected, const unsigned char* row_mask,
                    unsigned char* flags, int rows) {
  HL_REQUIRE(ctx && selected_rows && flags, "hl_mark_rows_u8: null argument");
  HL_REQUIRE(rows > 0, "hl_mark_rows_u8: requires non-zero rows");
  return mark_rows_on(ctx, ctx->stream, selected_rows, n_selected, row_mask, flags, rows);
}

int hl_mask_to_indices_u8(hl_ctx* ctx, const unsigned char* mask, int rows, int64_t* out_indices, int* count_dev) {
  HL_REQUIRE(ctx && mask && out_indices && count_dev, "hl_mask_to_indices_u8: null argument");
  HL_REQUIRE(rows > 0, "hl_mask_to_indices_u8: requires non-zero rows");
  return mask_to_indices_on(ctx, ctx->stream, mask, rows, out_indices, count_dev);
}

int hl_gather_rows_f32(hl_ctx* ctx, const float* src, const int64_t* indices, int n, int dim, float* dst) {
  HL_REQUIRE(ctx && src && indices && dst, "hl_gather_rows_f32: null argument");
  HL_REQUIRE(n >= 0 && dim > 0 && dim % 4 == 0, "hl_gather_rows_f32: row_dim must be a positive multiple of 4");
  return move_rows_on(ctx, ctx->stream, src, indices, nullptr, n, dim, dst, false);
}

int hl_scatter_rows_f32(hl_ctx* ctx, const float* src, const int64_t* indices, int n, int dim, float* dst) {
  HL_REQUIRE(ctx && src && indices && dst, "hl_scatter_rows_f32: null argument");
  HL_REQUIRE(n >= 0 && dim > 0 && dim % 4 == 0, "hl_scatter_rows_f32: row_dim must be a positive multiple of 4");
  return move_rows_on(ctx, ctx->stream, src, indices, nullptr, n, dim, dst, true);
}

int hl_sparse_rows_sum_squares_f32(hl_ctx* ctx, const float* grad, const int64_t* selected_rows, long long n_selected,
                                   const unsigned char* row_mask, unsigned char* row_flags, int rows, int row_dim,
                                   double* sum_dev) {
  HL_REQUIRE(ctx && grad && selected_rows && row_flags && sum_dev, "hl_sparse_rows_sum_squares_f32: null argument");
  HL_REQUIRE(rows > 0 && row_dim > 0, "hl_sparse_rows_sum_squares_f32: requires non-zero rows/row_dim");
  if (n_selected <= 0) return HL_OK;
  pdl(mark_rows_kernel, (unsigned)ceil_div_ll(n_selected, 256), 256, 0, ctx->stream)(selected_rows, n_selected, row_flags,
                                                                                  row_mask, rows, ctx->status_dev);
  HL_LAUNCH_CHECK("mark_rows_kernel");
  const bool vec = row_dim % 4 == 0 && (reinterpret_cast<uintptr_t>(grad) & 15) == 0;
  pdl(flagged_rows_sum_squares_kernel, std::min(ceil_div(rows, 8), ctx->sm_count * 8), 256, 0, ctx->stream)(grad, row_flags, rows, row_dim,
                                                                                                           vec, sum_dev);
  HL_LAUNCH_CHECK("flagged_rows_sum_squares_kernel");
  count_launch(ctx, 2);
  return HL_OK;
}

int hl_sparse_adamw_rows_f32(hl_ctx* ctx, float* param, float* grad, float* m, float* v, const int64_t* selected_rows,
                             long long n_selected, const unsigned char* row_mask, unsigned char* row_flags, int rows,
                             int row_dim, const hl_adamw_params* hp, int zero_grad_rows) {
  HL_REQUIRE(ctx && param && grad && m && v && selected_rows && row_flags && hp, "hl_sparse_adamw_rows_f32: null argument");
  HL_REQUIRE(rows > 0 && row_dim > 0, "hl_sparse_adamw_rows_f32: requires non-zero rows/row_dim");
  HL_REQUIRE(hp->bias_correction1 > 0.f && hp->bias_correction2 > 0.f, "hl_sparse_adamw_rows_f32: bias corrections must be positive");
  if (n_selected <= 0) return HL_OK;
  pdl(mark_rows_kernel, (unsigned)ceil_div_ll(n_selected, 256), 256, 0, ctx->stream)(selected_rows, n_selected, row_flags,
                                                                                  row_mask, rows, ctx->status_dev);
  HL_LAUNCH_CHECK("mark_rows_kernel");
  pdl(sparse_adamw_rows_kernel, ceil_div(rows, 8), 256, 0, ctx->stream)(param, grad, m, v, row_flags, rows, row_dim, *hp,
                                                                       zero_grad_rows);
  HL_LAUNCH_CHECK("sparse_adamw_rows_kernel");
  count_launch(ctx, 2);
  return HL_OK;
}

}  // extern "C"
