// One position through a block of the decoder in two kernels, and through the head in a third.
//
// What bounds a one-token step is how often one kernel waits for another: a kernel's end, seen by its dependent, and the input row
// out of L2 are two microseconds, whatever the kernel does.  A block took five kernels (q/k/v, attention, its projection, and the
// two products of the feed-forward), 20 us for the GPT-sized model.  Here a cluster keeps what stays within it in shared memory:
// the eight CTAs of a head form its q, k and v, attend, and multiply the head's channels into every output of the projection; the
// eight CTAs of a slice of the hidden units do the same for the feed-forward.  What crosses clusters is a sum over them of such
// partial rows, taken by every cluster of the next kernel, an eighth of the channels a CTA, in the clusters' order.  All weights, and
// the keys and values but the newest, are on their way into shared memory before a kernel waits for its predecessor.
//
// Within a kernel a chain of a dozen short phases is left, 400 to 1500 cycles each: shared-memory reads, dependent steps, barriers, and
// code that runs once (an unrolled loop is slower than a rolled one).  A product by lanes that multiply and add reads the input row
// again for every row of weights (24 rows of 768: 2700 cycles); on the matrix instruction the row is the second operand, the same in
// all of its columns, and the warps share the contraction (1100).
//
// A one-token step of the GPT-sized model at 500 positions: 271 -> 211 us (attention kernel 9.8, feed-forward 5.6, head 19, the choice
// 7.6); generation of 8 tokens behind a prefix of 500 2690 -> 2215 us, of 32 with four f32 blocks of 128 channels (24 one-token steps)
// 3550 -> 3010.
#include "decode.cuh"
#include "tc05.cuh"

namespace hl {
namespace {

constexpr int DB_CTAS = 8;        // a cluster
constexpr int DB_THREADS = 512;
constexpr int DB_WARPS = DB_THREADS / 32;
constexpr int DB_SLOTS = DB_THREADS / 8;  // keys at a time: eight lanes take one, sixteen bytes each
constexpr int DB_KEY_TURNS = 2;           // keys a thread sees at most: contexts of up to 8 * 2 * 64
constexpr int DB_PARTS = 16;              // partial rows whose loads a thread has in flight
constexpr int DB_MAX_PARTS = 32;
constexpr size_t DB_MAX_SHARED = 220 * 1024;

__device__ __forceinline__ void cp_async4(void* shared, const void* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(shared)), "l"(global) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T> __device__ __forceinline__ float rounded(float x) { return sizeof(T) == 2 ? bf16_round(x) : x; }
template <typename T> __device__ __forceinline__ T stored(float x) {
  if constexpr (sizeof(T) == 2) return to_bf16(x); else return x;
}

template <typename T> constexpr int row_pad = 16 / (int)sizeof(T);  // elements behind a row of weights, so that rows side by side touch all banks

// Sixteen rows of bf16 weights times sixteen values of a vector, which stands in all columns of the second operand: every column of the
// result is the same, and lane 4 r holds rows r and r + 8.
struct RowMma {
  static constexpr int M = 16, K = 16;
  float c[4] = {};
  // `w`: the tile's first element, rows `pitch` elements apart, `last` the last of its rows that there is
  __device__ __forceinline__ void step(const __nv_bfloat16* w, int pitch, int last, const __nv_bfloat16* x) {
    const int lane = threadIdx.x & 31;
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(w + min(lane & 15, last) * pitch + (lane >> 4) * 8);
    uint32_t a0, a1, a2, a3;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "r"(at) : "memory");
    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(x + (lane & 3) * 2), b1 = *reinterpret_cast<const uint32_t*>(x + 8 + (lane & 3) * 2);
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
  // put(row, value) for the rows that there are
  template <typename F> __device__ __forceinline__ void rows(int last, F put) const {
    const int r = (threadIdx.x & 31) >> 2;
    if ((threadIdx.x & 3) == 0) {
      if (r <= last) put(r, c[0]);
      if (r + 8 <= last) put(r + 8, c[2]);
    }
  }
};

template <typename Acc>
__device__ __forceinline__ Acc sum_of_warps(const Acc* red, int rows, int r) {
  Acc s = 0;
#pragma unroll
  for (int w = 0; w < DB_WARPS; ++w) s += red[w * rows + r];
  return s;
}

// Rows of weights times x, both in shared memory.  bf16: the warps share the contraction, red[warp][row] is left for product_of_row
// behind a barrier; k a multiple of 16.  f64 sums: a warp a row (the f64 matrix instruction, four values a step, took longer).
__device__ __forceinline__ void multiply_rows(const __nv_bfloat16* w, int pitch, int rows, const __nv_bfloat16* x, int k, float* red) {
  const int warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int m = 0; m < rows; m += RowMma::M) {
    RowMma t;
#pragma unroll 1
    for (int at = warp * RowMma::K; at < k; at += DB_WARPS * RowMma::K) t.step(w + m * pitch + at, pitch, rows - 1 - m, x + at);
    t.rows(rows - 1 - m, [&](int r, float v) { red[warp * rows + m + r] = v; });
  }
}
__device__ __forceinline__ float product_of_row(const float* red, int rows, int r) { return sum_of_warps(red, rows, r); }
__device__ __forceinline__ void multiply_rows(const float* w, int pitch, int rows, const float* x, int k, double* red) {
#pragma unroll 1
  for (int r = threadIdx.x >> 5; r < rows; r += DB_WARPS) {
    double acc = 0;
#pragma unroll 1
    for (int c = (threadIdx.x & 31) * 4; c < k; c += 128) {
      float v[4], y[4];
      load_x(w + r * pitch + c, v);
      load_x(x + c, y);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc += (double)v[e] * (double)y[e];
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[r] = acc;
  }
}
__device__ __forceinline__ double product_of_row(const double* red, int, int r) { return red[r]; }

// Many rows times a few values (k at most a few dozen): put(row, value) for each.
template <typename F>
__device__ __forceinline__ void multiply_columns(const __nv_bfloat16* w, int pitch, int rows, const __nv_bfloat16* x, int k, F put) {
  const int warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int m = warp * RowMma::M; m < rows; m += DB_WARPS * RowMma::M) {
    RowMma t;
#pragma unroll 1
    for (int s = 0; s < k; s += RowMma::K) t.step(w + m * pitch + s, pitch, rows - 1 - m, x + s);
    t.rows(rows - 1 - m, [&](int r, float v) { put(m + r, v); });
  }
}
template <typename F>
__device__ __forceinline__ void multiply_columns(const float* w, int pitch, int rows, const float* x, int k, F put) {
#pragma unroll 1
  for (int r = threadIdx.x; r < rows; r += DB_THREADS) {
    double acc = 0;
#pragma unroll 1
    for (int c = 0; c < k; c += 4) {
      float v[4], y[4];
      load_x(w + r * pitch + c, v);
      load_x(x + c, y);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc += (double)v[e] * (double)y[e];
    }
    put(r, acc);
  }
}

// What the peers of a cluster send arrives on barriers that count its bytes: a barrier of the cluster behind the stores cost a release,
// that is, waiting for every store's answer, and the barrier's own way there and back.
struct Mail {
  uint64_t arrived[2];
  int abort_flag;
  __device__ __forceinline__ void open(int bytes0, int bytes1) {  // by one thread, before the cluster meets
    tc05::mbar_init(&arrived[0], 1);
    tc05::mbar_init(&arrived[1], 1);
    abort_flag = 0;
    tc05::fence_barrier_init();
    if (bytes0) tc05::mbar_arrive_expect_tx(&arrived[0], bytes0);
    if (bytes1) tc05::mbar_arrive_expect_tx(&arrived[1], bytes1);
  }
  __device__ __forceinline__ bool wait(int i, unsigned long long limit_ns, int* status) {
    const bool all = tc05::mbar_wait(&arrived[i], 0, &abort_flag, limit_ns);
    if (!all) *status = 1;
    return all;
  }
};
// At the end of a kernel whose wait ran out.  The thread, and with it its CTA, stays until the peers, whose waits are bounded as well, have left
// or are here too, and then until what they sent has landed: a peer may be late and not lost.
__device__ __noinline__ void outstay_peers() {
  tc05::cluster_meet();
  for (int k = 0; k < 2000; ++k) __nanosleep(100);
}
// `bytes` (whole sixteens) of this CTA's shared memory into a peer's, by one warp.  A store to a peer takes its turn whatever its width:
// 96 of 32 bytes held a kernel up for 3300 cycles.
__device__ __forceinline__ void push(uint64_t* arrived, void* to, const void* from, int bytes, int peer) {
  const uint32_t there = tc05::cluster_map_shared(to, peer), bar = tc05::cluster_map_shared(arrived, peer);
#pragma unroll 1
  for (int b = (threadIdx.x & 31) * 16; b < bytes; b += 32 * 16) {
    const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const char*>(from) + b);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(there + b), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w), "r"(bar) : "memory");
  }
}

// The residual stream's row, rounded where the full-window kernels round it, and its layer norm.  Every CTA forms it for itself, a
// thread channels 2 i and 2 i + 1; block 0 keeps the row.  (A share of the channels each and exchanged within the cluster, with the
// means and squares of groups of channels: 3 % less for a step of 768 channels, 4 to 8 % more from 64 to 512.)
template <typename T, typename Acc>
struct Row {
  float2 bias, gamma, beta;
  Acc per_row;
  __device__ __forceinline__ Row(const DecodeRow& r, const float* g, const float* b, int d) {  // nothing here is the predecessor's
    const int c = threadIdx.x * 2;
    per_row = (Acc)1 / (Acc)d;
    bias = gamma = beta = make_float2(0.f, 0.f);
    if (c < d) {
      if (r.n) bias = __ldg(reinterpret_cast<const float2*>(r.bias + c));
      gamma = __ldg(reinterpret_cast<const float2*>(g + c));
      beta = __ldg(reinterpret_cast<const float2*>(b + c));
    }
  }
  __device__ __forceinline__ static Acc sum_of_block(Acc v, Acc* red) {
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    v = warp_sum(v);
    if (lane == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    return warp_sum(lane < warps ? red[lane] : (Acc)0);
  }
  // out [d] and red (two values a warp): shared memory.  Ends without a barrier behind `out`.
  __device__ __forceinline__ void form(const DecodeRow& r, int d, Acc* red, T* out) const {
    struct alignas(2 * sizeof(Acc)) Pair { Acc x, y; };
    const int c = threadIdx.x * 2;
    const T* base = static_cast<const T*>(r.base);
    float x = 0.f, y = 0.f;
    if (c < d) {
      if (base) { x = as_f32(__ldcg(base + c)); y = as_f32(__ldcg(base + c + 1)); }
      if (r.n) {
        const Acc* parts = static_cast<const Acc*>(r.parts) + c;
        Pair s{0, 0};
#pragma unroll 1
        for (int i0 = 0; i0 < r.n; i0 += DB_PARTS) {
          Pair v[DB_PARTS];
#pragma unroll
          for (int j = 0; j < DB_PARTS; ++j) v[j] = i0 + j < r.n ? load_pair(reinterpret_cast<const Pair*>(parts + (i0 + j) * d)) : Pair{0, 0};
#pragma unroll
          for (int j = 0; j < DB_PARTS; ++j) { s.x += v[j].x; s.y += v[j].y; }
        }
        x = rounded<T>(x + rounded<T>((float)s.x + bias.x));
        y = rounded<T>(y + rounded<T>((float)s.y + bias.y));
      } else if (!base) {
        const float *a = r.table + r.state[1] * d + c, *b = r.positions + r.state[0] * d + c;
        x = rounded<T>(rounded<T>(a[0]) + rounded<T>(b[0]));
        y = rounded<T>(rounded<T>(a[1]) + rounded<T>(b[1]));
      }
      if (r.keep && blockIdx.x == 0) { static_cast<T*>(r.keep)[c] = stored<T>(x); static_cast<T*>(r.keep)[c + 1] = stored<T>(y); }
    }
    const Acc mean = sum_of_block((Acc)x + (Acc)y, red) * per_row;
    const Acc dx = c < d ? (Acc)x - mean : (Acc)0, dy = c < d ? (Acc)y - mean : (Acc)0;
    const Acc rstd = (Acc)1 / sqrt(sum_of_block(dx * dx + dy * dy, red + (blockDim.x >> 5)) * per_row + (Acc)1e-5f);
    if (c < d) {
      out[c] = stored<T>((float)(dx * rstd * (Acc)gamma.x + (Acc)beta.x));
      out[c + 1] = stored<T>((float)(dy * rstd * (Acc)gamma.y + (Acc)beta.y));
    }
  }

 private:
  template <typename Pair> __device__ __forceinline__ static Pair load_pair(const Pair* p) {
    if constexpr (sizeof(Pair) == 8) {
      const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
      return Pair{v.x, v.y};
    } else {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
      return Pair{v.x, v.y};
    }
  }
};

// `rows` rows of `bytes` bytes, `stride` bytes apart, into shared memory, `pitch` bytes apart: a warp a row, or eight lanes where it is short.
__device__ __forceinline__ void stage_rows(void* shared, int pitch, const void* global, size_t stride, int rows, int bytes) {
  const int group = bytes < 512 ? 8 : 32;
#pragma unroll 1
  for (int r = threadIdx.x / group; r < rows; r += DB_THREADS / group)
#pragma unroll 1
    for (int b = threadIdx.x % group * 16; b < bytes; b += group * 16)
      cp_async16(static_cast<char*>(shared) + r * pitch + b, static_cast<const char*>(global) + r * stride + b);
}

// Layer norm, q/k/v, attention over rows 0 .. *position and the head's share of the projection: cluster h is head h.  With
// `window` the q/k/v rows are all there, left by the predecessor: only attention and projection.
template <typename T, typename Acc>
struct AttentionLayout {  // shared memory, bytes
  int wqkv, wo, kv, bias, row, red, fresh, q, part, all, pitch_all, att, total;
  __host__ __device__ AttentionLayout(int d, int hd, int cap, bool window) {
    const int sz = sizeof(T), rows = 3 * (hd / DB_CTAS);
    int at = 0;
    auto take = [&](int bytes) { const int here = at; at += (bytes + 15) & ~15; return here; };
    wqkv = take(window ? 0 : rows * (d + row_pad<T>) * sz);
    wo = take(d / DB_CTAS * (hd + row_pad<T>) * sz);
    kv = take(2 * cap * hd * sz);
    bias = take(rows * 4);
    row = take(window ? 0 : d * sz);
    red = take(DB_WARPS * rows * (int)sizeof(Acc));
    fresh = take(DB_CTAS * ((rows + 3) & ~3) * 4);
    q = take(hd * 4);
    part = take(DB_WARPS * hd * (int)sizeof(Acc));
    pitch_all = (hd + 2 + 3) & ~3;  // elements
    all = take(DB_CTAS * pitch_all * (int)sizeof(Acc));
    att = take(hd * sz);
    total = at;
  }
};
struct AttentionArgs {
  DecodeRow x;
  const float *gamma, *beta;
  const void* wqkv;
  const float* bqkv;
  void* qkv;
  const long long* state;
  const void* wo;
  void* parts;  // [heads][d]
  int d, hd, cap;
  bool window;
  int* status;
  unsigned long long wait_limit_ns;
  int withheld;  // test hook: bytes that are waited for and never sent
};

template <typename T, typename Acc>
__global__ void __launch_bounds__(DB_THREADS, 2) decode_attention_block_kernel(const __grid_constant__ AttentionArgs a) {
  extern __shared__ __align__(16) unsigned char db_smem[];
  __shared__ Acc norm[2 * DB_WARPS], red_max[DB_WARPS], red_sum[DB_WARPS];
  __shared__ Mail mail;
  constexpr int PN = Pack<T>::N, PAD = row_pad<T>;
  const int d = a.d, hd = a.hd, cpc = hd / DB_CTAS, opc = d / DB_CTAS, rows = 3 * cpc;
  const AttentionLayout<T, Acc> at(d, hd, a.cap, a.window);
  T* wqkv = reinterpret_cast<T*>(db_smem + at.wqkv);    // [3][cpc][d]
  T* wo = reinterpret_cast<T*>(db_smem + at.wo);        // [opc][hd]
  T* kept = reinterpret_cast<T*>(db_smem + at.kv);      // [2][cap][hd]
  float* bias = reinterpret_cast<float*>(db_smem + at.bias);
  T* row = reinterpret_cast<T*>(db_smem + at.row);
  Acc* red = reinterpret_cast<Acc*>(db_smem + at.red);
  // [CTAs][3][cpc] this position's q, k and v
  float* fresh = reinterpret_cast<float*>(db_smem + at.fresh);
  const int pitch_fresh = (rows + 3) & ~3, pitch_all = at.pitch_all;
  float* q = reinterpret_cast<float*>(db_smem + at.q);
  Acc* part = reinterpret_cast<Acc*>(db_smem + at.part);        // [warps][hd]
  Acc* all = reinterpret_cast<Acc*>(db_smem + at.all);          // [CTAs][pitch_all] values, maximum, sum
  T* att = reinterpret_cast<T*>(db_smem + at.att);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = (int)(blockIdx.x % DB_CTAS), h = (int)(blockIdx.x / DB_CTAS);
  const long long ld = 3 * d;
  T* qkv = static_cast<T*>(a.qkv) + h * hd;
  pdl_trigger();
  if (threadIdx.x == 0) mail.open(a.window ? 0 : (DB_CTAS - 1) * pitch_fresh * 4 + a.withheld, (DB_CTAS - 1) * pitch_all * (int)sizeof(Acc) + a.withheld);
  // The position was copied here before the first kernel of the sequence started.
  const int t = (int)a.state[0], keys = t + 1, chunk = (keys + DB_CTAS - 1) / DB_CTAS;
  const int k0 = min(keys, rank * chunk), k1 = min(keys, k0 + chunk);
  auto stage_keys = [&](int n) {
#pragma unroll 1
    for (int i = 0; i < 2; ++i)
      stage_rows(kept + (size_t)i * a.cap * hd, hd * sizeof(T), qkv + (long long)k0 * ld + (1 + i) * d, ld * sizeof(T), n, hd * sizeof(T));
  };
  if (!a.window) {
#pragma unroll 1
    for (int i = 0; i < 3; ++i)
      stage_rows(wqkv + i * cpc * (d + PAD), (d + PAD) * sizeof(T), static_cast<const T*>(a.wqkv) + ((size_t)i * d + h * hd + rank * cpc) * d,
                 d * sizeof(T), cpc, d * sizeof(T));
    if ((int)threadIdx.x < rows) cp_async4(bias + threadIdx.x, a.bqkv + threadIdx.x / cpc * d + h * hd + rank * cpc + threadIdx.x % cpc);
    cp_async_commit();
    stage_keys(min(k1, t) - min(k0, t));
  }
  stage_rows(wo, (hd + PAD) * sizeof(T), static_cast<const T*>(a.wo) + (size_t)rank * opc * d + h * hd, d * sizeof(T), opc, hd * sizeof(T));
  cp_async_commit();
  const Row<T, Acc> in(a.x, a.gamma, a.beta, a.window ? 0 : d);
  const Acc scale = (Acc)1 / sqrt((Acc)hd);
  const int fresh_at = (int)threadIdx.x / cpc * pitch_fresh + (int)threadIdx.x % cpc;
  bool answered = true;
  tc05::cluster_meet();  // the peers have started: their shared memory may be written
  pdl_wait();
  if (a.window) {
    stage_keys(k1 - k0);
    for (int c = threadIdx.x; c < hd; c += DB_THREADS) q[c] = as_f32(__ldcg(qkv + (long long)t * ld + c));
    cp_async_wait_all();
  } else {
    in.form(a.x, d, norm, row);
    cp_async_wait<1>();
    __syncthreads();
    multiply_rows(wqkv, d + PAD, rows, row, d, red);
    __syncthreads();
    float* own = fresh + rank * pitch_fresh;
    float y = 0.f;
    if (const int i = threadIdx.x; i < rows) own[i] = y = rounded<T>((float)product_of_row(red, rows, i) + bias[i]);
    __syncthreads();
    if (warp < DB_CTAS && warp != rank) push(&mail.arrived[0], own, own, pitch_fresh * 4, warp);
    cp_async_wait_all();
    answered = mail.wait(0, a.wait_limit_ns, a.status);
    if (const int i = threadIdx.x; i < rows) {  // (nobody waits for these)
      const int which = i < cpc ? 0 : i < 2 * cpc ? 1 : 2;
      qkv[(long long)t * ld + which * d + rank * cpc + i - which * cpc] = stored<T>(y);
    }
    if (const int c = threadIdx.x; c < hd) {
      const float* f = fresh + fresh_at;
      q[c] = f[0];
      if (k0 <= t && t < k1) {
        kept[(t - k0) * hd + c] = stored<T>(f[cpc]);
        kept[(a.cap + t - k0) * hd + c] = stored<T>(f[2 * cpc]);
      }
    }
  }
  __syncthreads();
  const int sub = threadIdx.x & 7, slot = threadIdx.x >> 3;
  Acc w[DB_KEY_TURNS], mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < DB_KEY_TURNS; ++i) {
    const int key = k0 + slot + i * DB_SLOTS;
    w[i] = 0;
    if (k0 + i * DB_SLOTS >= k1) continue;  // (the same for every thread)
    if (key < k1)
#pragma unroll 1
      for (int c = sub * PN; c < hd; c += 8 * PN) {
        float v[PN], qv[PN];
        Pack<T>::unpack(*reinterpret_cast<const uint4*>(kept + (key - k0) * hd + c), v);
        load_x(q + c, qv);
#pragma unroll
        for (int e = 0; e < PN; ++e) w[i] += (Acc)qv[e] * (Acc)v[e];
      }
    w[i] += __shfl_xor_sync(0xffffffffu, w[i], 1);
    w[i] += __shfl_xor_sync(0xffffffffu, w[i], 2);
    w[i] += __shfl_xor_sync(0xffffffffu, w[i], 4);
    w[i] *= scale;
    if (key < k1) mx = max(mx, w[i]);
  }
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
  if (lane == 0) red_max[warp] = mx;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < DB_WARPS; ++i) mx = max(mx, red_max[i]);
  Acc weights = 0;
#pragma unroll
  for (int i = 0; i < DB_KEY_TURNS; ++i) {
    w[i] = k0 + slot + i * DB_SLOTS < k1 ? exp(w[i] - mx) : (Acc)0;
    weights += w[i];
  }
  weights += __shfl_xor_sync(0xffffffffu, weights, 8);
  weights += __shfl_xor_sync(0xffffffffu, weights, 16);
  if (lane == 0) red_sum[warp] = weights;
#pragma unroll 1
  for (int c0 = 0; c0 < hd; c0 += 8 * PN) {
    const int c = c0 + sub * PN;
    Acc acc[PN];
#pragma unroll
    for (int e = 0; e < PN; ++e) acc[e] = 0;
#pragma unroll
    for (int i = 0; i < DB_KEY_TURNS; ++i)
      if (const int key = k0 + slot + i * DB_SLOTS; key < k1 && c < hd) {
        float v[PN];
        Pack<T>::unpack(*reinterpret_cast<const uint4*>(kept + (a.cap + key - k0) * hd + c), v);
#pragma unroll
        for (int e = 0; e < PN; ++e) acc[e] += w[i] * (Acc)v[e];
      }
#pragma unroll
    for (int e = 0; e < PN; ++e) {
      acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 8);
      acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 16);
    }
    if (lane < 8 && c < hd) {
#pragma unroll
      for (int e = 0; e < PN; ++e) part[warp * hd + c + e] = acc[e];
    }
  }
  __syncthreads();
  Acc* own = all + rank * pitch_all;
  if (const int c = threadIdx.x; c < hd + 2) own[c] = c == hd ? mx : sum_of_warps(c < hd ? part : red_sum, c < hd ? hd : 1, c < hd ? c : 0);
  __syncthreads();
  if (warp < DB_CTAS && warp != rank) push(&mail.arrived[1], own, own, pitch_all * sizeof(Acc), warp);
  answered &= mail.wait(1, a.wait_limit_ns, a.status);
  {
    const Acc* mine = all + (lane & 7) * pitch_all + hd;
    const Acc m = mine[0];
    Acc top = m;
#pragma unroll
    for (int o = 1; o < DB_CTAS; o *= 2) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    const Acc f = m == (Acc)-INFINITY ? (Acc)0 : exp(m - top);
    Acc l = f * mine[1];
#pragma unroll
    for (int o = 1; o < DB_CTAS; o *= 2) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (const int c = threadIdx.x; warp * 32 < hd) {
      Acc v = 0;
#pragma unroll
      for (int r = 0; r < DB_CTAS; ++r) {
        const Acc fr = __shfl_sync(0xffffffffu, f, r);
        if (c < hd) v += fr * all[r * pitch_all + c];
      }
      if (c < hd) att[c] = stored<T>((float)(v / l));
    }
  }
  __syncthreads();
  Acc* out = static_cast<Acc*>(a.parts) + (size_t)h * d + rank * opc;
  multiply_columns(wo, hd + PAD, opc, att, hd, [&](int o, Acc v) { out[o] = v; });
  if (!answered) outstay_peers();
}

// Layer norm, the hidden units of a CTA and their share of every output; the shares of a cluster are added up within it.
template <typename T, typename Acc>
struct FeedForwardLayout {
  int w1, w2, pitch2, bias, row, red, hidden, outputs, sums, pitch_sums, total;
  __host__ __device__ FeedForwardLayout(int d, int units) {
    const int sz = sizeof(T);
    int at = 0;
    auto take = [&](int bytes) { const int here = at; at += (bytes + 15) & ~15; return here; };
    pitch2 = units * sz % 32 ? units : units + row_pad<T>;  // elements; an odd number of sixteen bytes
    w1 = take(units * (d + row_pad<T>) * sz);
    w2 = take(d * pitch2 * sz);
    bias = take(units * 4);
    row = take(d * sz);
    red = take(DB_WARPS * units * (int)sizeof(Acc));
    hidden = take(units * sz);
    pitch_sums = (d / DB_CTAS + 3) & ~3;  // elements
    outputs = take(DB_CTAS * pitch_sums * (int)sizeof(Acc));
    sums = take(DB_CTAS * pitch_sums * (int)sizeof(Acc));
    total = at;
  }
};
struct FeedForwardArgs {
  DecodeRow x;
  const float *gamma, *beta;
  const void* w1;
  const float* b1;
  const void* w2;
  void* parts;  // [clusters][d]
  int d, hidden, units;  // units: hidden units a CTA
  int* status;
  unsigned long long wait_limit_ns;
  int withheld;  // as above
};

template <typename T, typename Acc>
__global__ void __launch_bounds__(DB_THREADS, 2) decode_feed_forward_kernel(const __grid_constant__ FeedForwardArgs a) {
  extern __shared__ __align__(16) unsigned char db_smem[];
  __shared__ Acc norm[2 * DB_WARPS];
  __shared__ Mail mail;
  constexpr int PAD = row_pad<T>;
  const int d = a.d, opc = d / DB_CTAS, units = a.units;
  const FeedForwardLayout<T, Acc> at(d, units);
  T* w1 = reinterpret_cast<T*>(db_smem + at.w1);  // [units][d]
  T* w2 = reinterpret_cast<T*>(db_smem + at.w2);  // [d][units]
  float* bias = reinterpret_cast<float*>(db_smem + at.bias);
  T* row = reinterpret_cast<T*>(db_smem + at.row);
  Acc* red = reinterpret_cast<Acc*>(db_smem + at.red);
  T* hidden = reinterpret_cast<T*>(db_smem + at.hidden);
  const int pitch_sums = at.pitch_sums;
  Acc* outputs = reinterpret_cast<Acc*>(db_smem + at.outputs);  // [CTAs][pitch_sums] this CTA's part of every output, a peer's together
  Acc* sums = reinterpret_cast<Acc*>(db_smem + at.sums);        // [CTAs][pitch_sums] the peers' parts of this CTA's outputs
  const int warp = threadIdx.x >> 5, rank = (int)(blockIdx.x % DB_CTAS);
  const int first = min(a.hidden, (int)blockIdx.x * units), n = min(units, a.hidden - first);  // n may be 0
  pdl_trigger();
  if (threadIdx.x == 0) mail.open(DB_CTAS * pitch_sums * (int)sizeof(Acc) + a.withheld, 0);
  stage_rows(w1, (d + PAD) * sizeof(T), static_cast<const T*>(a.w1) + (size_t)first * d, d * sizeof(T), n, d * sizeof(T));
  if ((int)threadIdx.x < n) cp_async4(bias + threadIdx.x, a.b1 + first + threadIdx.x);
  cp_async_commit();
  stage_rows(w2, at.pitch2 * sizeof(T), static_cast<const T*>(a.w2) + first, (size_t)a.hidden * sizeof(T), d, n * sizeof(T));
  cp_async_commit();
  if (n < units)  // units that do not exist weigh nothing
    for (int i = threadIdx.x; i < d * (units - n); i += DB_THREADS) w2[i / (units - n) * at.pitch2 + n + i % (units - n)] = T(0.f);
  const Row<T, Acc> in(a.x, a.gamma, a.beta, d);
  const unsigned per_share = ((1u << 20) + opc - 1) / opc;  // c / opc = c * per_share >> 20 for c < 1024, opc <= 128
  tc05::cluster_meet();  // the peers have started
  pdl_wait();
  in.form(a.x, d, norm, row);
  cp_async_wait<1>();
  __syncthreads();
  multiply_rows(w1, d + PAD, n, row, d, red);
  cp_async_wait_all();
  __syncthreads();
  if (const int u = threadIdx.x; u < units) {
    float y = 0.f;
    if (u < n) {
      y = (float)product_of_row(red, n, u) + bias[u];
      y = sizeof(T) == 2 ? gelu_fwd_fast(bf16_round(y)) : (float)gelu_fwd<double>((double)y);
    }
    hidden[u] = stored<T>(y);
  }
  __syncthreads();
  multiply_columns(w2, at.pitch2, d, hidden, units, [&](int c, Acc v) {
    const int owner = (int)(c * per_share >> 20);
    outputs[owner * pitch_sums + c - owner * opc] = v;
  });
  __syncthreads();
  if (warp < DB_CTAS) push(&mail.arrived[0], sums + rank * pitch_sums, outputs + warp * pitch_sums, pitch_sums * sizeof(Acc), warp);
  const bool answered = mail.wait(0, a.wait_limit_ns, a.status);
  Acc* out = static_cast<Acc*>(a.parts) + (size_t)(blockIdx.x / DB_CTAS) * d + rank * opc;
  if (const int c = threadIdx.x; c < opc) {
    Acc s = 0;
#pragma unroll
    for (int r = 0; r < DB_CTAS; ++r) s += sums[r * pitch_sums + c];
    out[c] = s;
  }
  if (!answered) outstay_peers();
}

// The row itself, for kernels that read it.
template <typename T, typename Acc>
__global__ void __launch_bounds__(256) decode_row_kernel(const __grid_constant__ DecodeRow r, int d) {
  pdl_trigger();
  const int c = blockIdx.x * 256 + threadIdx.x;
  const float bias = c < d ? __ldg(r.bias + c) : 0.f;
  pdl_wait();
  if (c >= d) return;
  Acc s = 0;
#pragma unroll 8
  for (int i = 0; i < r.n; ++i) s += __ldcg(static_cast<const Acc*>(r.parts) + i * d + c);
  static_cast<T*>(r.keep)[c] = stored<T>(as_f32(__ldcg(static_cast<const T*>(r.base) + c)) + rounded<T>((float)s + bias));
}

// Final layer norm and head: out[v] = W[v] · row + bias[v].  Bound by the weights' bytes (77 MB for 50304 x 768).  A warp keeps
// DEPTH rows of weights, and their biases, on their way in a ring of its own, and its lanes the row in registers.
constexpr int DH_WARPS = 16;
constexpr int DH_THREADS = DH_WARPS * 32;
struct HeadArgs {
  DecodeRow x;
  const float *gamma, *beta;
  const void* w;
  const float* bias;
  float* out;
  int n, d;
};
template <typename T> __host__ __device__ constexpr int head_slot(int d) { return d * (int)sizeof(T) + 16; }
template <typename T, typename Acc, int DEPTH>
__global__ void __launch_bounds__(DH_THREADS) decode_head_kernel(const __grid_constant__ HeadArgs a) {
  extern __shared__ __align__(16) unsigned char db_smem[];
  __shared__ Acc norm[2 * DH_WARPS];
  constexpr int PN = Pack<T>::N, U = GV_SPAN / (32 * PN);
  const int d = a.d, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot = head_slot<T>(d);
  T* row = reinterpret_cast<T*>(db_smem);
  unsigned char* ring = db_smem + d * sizeof(T) + (size_t)warp * DEPTH * slot;
  const int step = gridDim.x * DH_WARPS;
  int fetch = blockIdx.x + warp * gridDim.x, fetch_slot = 0;
  auto request = [&]() {
    if (fetch < a.n) {
      unsigned char* to = ring + fetch_slot * slot;
      const T* w = static_cast<const T*>(a.w) + (size_t)fetch * d;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (const int c = u * 32 * PN + lane * PN; c < d) cp_async16(to + c * sizeof(T), w + c);
      if (lane == 0) cp_async4(to + d * sizeof(T), a.bias + fetch);
    }
    cp_async_commit();
    fetch += step;
    fetch_slot = fetch_slot + 1 == DEPTH ? 0 : fetch_slot + 1;
  };
  pdl_trigger();
#pragma unroll 1
  for (int i = 0; i < DEPTH; ++i) request();
  const Row<T, Acc> in(a.x, a.gamma, a.beta, d);
  pdl_wait();
  in.form(a.x, d, norm, row);
  __syncthreads();
  float xv[U][PN];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int c = u * 32 * PN + lane * PN;
    if (c < d) {
      load_x(row + c, xv[u]);
    } else {
#pragma unroll
      for (int e = 0; e < PN; ++e) xv[u][e] = 0.f;
    }
  }
  int now = 0;
  for (int v = blockIdx.x + warp * gridDim.x; v < a.n; v += step) {
    cp_async_wait<DEPTH - 1>();
    __syncwarp();
    const unsigned char* at = ring + now * slot;
    Acc acc = 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (const int c = u * 32 * PN + lane * PN; c < d) {
        float y[PN];
        Pack<T>::unpack(*reinterpret_cast<const uint4*>(at + c * sizeof(T)), y);
#pragma unroll
        for (int e = 0; e < PN; ++e) acc += (Acc)y[e] * (Acc)xv[u][e];
      }
    acc = warp_sum(acc);
    if (lane == 0) a.out[v] = (float)acc + *reinterpret_cast<const float*>(at + d * sizeof(T));
    __syncwarp();
    request();
    now = now + 1 == DEPTH ? 0 : now + 1;
  }
}

// Hidden units a CTA: sixteen or a multiple (f64 sums: eight), so that at most sixteen clusters' rows are left to add.
template <typename T> int feed_forward_units(int hidden) {
  const int least = sizeof(T) == 2 ? 16 : 8;
  return least * ceil_div(hidden, least * DB_CTAS * 16);
}

template <typename T, typename Acc>
bool block_fits(int d, int heads, int hidden, int context) {
  const int hd = d / heads;
  // contractions in whole steps of the matrix instruction, rows of weights and slices of them on sixteen bytes
  if (d > GV_SPAN || d % 16 || hd % (DB_CTAS * 2) || hidden % 8 || heads > DB_MAX_PARTS) return false;
  if (ceil_div(context, DB_CTAS) > DB_KEY_TURNS * DB_SLOTS) return false;
  if (feed_forward_units<T>(hidden) > DB_THREADS) return false;  // a thread a hidden unit
  return AttentionLayout<T, Acc>(d, hd, ceil_div(context, DB_CTAS), false).total <= (int)DB_MAX_SHARED && 3 * hd <= DB_THREADS &&
         FeedForwardLayout<T, Acc>(d, feed_forward_units<T>(hidden)).total <= (int)DB_MAX_SHARED;
}

unsigned long long wait_limit(const hl_ctx* ctx) { return ctx->wait_limit_ns ? ctx->wait_limit_ns : tc05::kWaitLimitNs; }
int withheld(const hl_ctx* ctx) { return ctx->gemm_skip_kblock >= 0 ? 16 : 0; }

template <typename T, typename Acc>
int run_attention(hl_ctx* ctx, const DecodeBlock& b) {
  AttentionArgs a{b.x, b.ln1_gamma, b.ln1_beta, b.wqkv, b.bqkv, b.qkv, b.state, b.wo, b.attention_parts, b.d, b.d / b.heads,
                  ceil_div(b.context, DB_CTAS), b.window, ctx->status_dev + ST_WAIT_EXPIRED, wait_limit(ctx), withheld(ctx)};
  const AttentionLayout<T, Acc> at(a.d, a.hd, a.cap, a.window);
  auto kern = decode_attention_block_kernel<T, Acc>;
  HL_ALLOW_SHARED(ctx, DB_MAX_SHARED, kern);
  HL_CUDA(launch_pdl(kern, b.heads * DB_CTAS, DB_THREADS, at.total, ctx->stream, DB_CTAS, a));
  count_launch(ctx);
  return HL_OK;
}

template <typename T, typename Acc>
int run_feed_forward(hl_ctx* ctx, const DecodeBlock& b, const DecodeRow& x, int units, int clusters) {
  FeedForwardArgs a{x, b.ln2_gamma, b.ln2_beta, b.w1, b.b1, b.w2, b.feed_forward_parts, b.d, b.hidden, units, ctx->status_dev + ST_WAIT_EXPIRED, wait_limit(ctx),
                    withheld(ctx)};
  const FeedForwardLayout<T, Acc> at(a.d, units);
  auto kern = decode_feed_forward_kernel<T, Acc>;
  HL_ALLOW_SHARED(ctx, DB_MAX_SHARED, kern);
  HL_CUDA(launch_pdl(kern, clusters * DB_CTAS, DB_THREADS, at.total, ctx->stream, DB_CTAS, a));
  count_launch(ctx);
  return HL_OK;
}

template <typename T, typename Acc, int DEPTH>
int run_head(hl_ctx* ctx, const HeadArgs& a) {
  auto kern = decode_head_kernel<T, Acc, DEPTH>;
  HL_ALLOW_SHARED(ctx, DB_MAX_SHARED, kern);
  const size_t smem = a.d * (int)sizeof(T) + (size_t)DH_WARPS * DEPTH * head_slot<T>(a.d);
  HL_CUDA(launch_pdl(kern, std::min(ceil_div(a.n, DH_WARPS), ctx->sm_count), DH_THREADS, smem, ctx->stream, 1, a));
  count_launch(ctx);
  return HL_OK;
}

template <typename T, typename Acc>
int run_head(hl_ctx* ctx, const HeadArgs& a) {
  const int row = DH_WARPS * head_slot<T>(a.d), room = (int)DB_MAX_SHARED - a.d * (int)sizeof(T);
  if (8 * row <= room) return run_head<T, Acc, 8>(ctx, a);
  if (4 * row <= room) return run_head<T, Acc, 4>(ctx, a);
  return run_head<T, Acc, 2>(ctx, a);
}

}  // namespace

bool decode_block_applies(int dtype, int d, int heads, int hidden, int context) {
  return dtype == HL_BF16 ? block_fits<__nv_bfloat16, float>(d, heads, hidden, context) : block_fits<float, double>(d, heads, hidden, context);
}

size_t decode_block_parts_bytes(int d) { return (size_t)DB_MAX_PARTS * d * sizeof(double); }

int decode_attention_block(hl_ctx* ctx, const DecodeBlock& b, DecodeRow* after) {
  const int rc = b.dtype == HL_BF16 ? run_attention<__nv_bfloat16, float>(ctx, b) : run_attention<float, double>(ctx, b);
  if (rc != HL_OK) return rc;
  *after = DecodeRow{};
  after->base = b.x.n || !b.x.base ? b.x.keep : b.x.base;
  after->parts = b.attention_parts;
  after->n = b.heads;
  after->bias = b.bo;
  return HL_OK;
}

int decode_feed_forward(hl_ctx* ctx, const DecodeBlock& b, const DecodeRow& x, DecodeRow* after) {
  const int units = b.dtype == HL_BF16 ? feed_forward_units<__nv_bfloat16>(b.hidden) : feed_forward_units<float>(b.hidden), clusters = ceil_div(b.hidden, units * DB_CTAS);
  const int rc = b.dtype == HL_BF16 ? run_feed_forward<__nv_bfloat16, float>(ctx, b, x, units, clusters)
                                    : run_feed_forward<float, double>(ctx, b, x, units, clusters);
  if (rc != HL_OK) return rc;
  *after = DecodeRow{};
  after->base = x.keep;
  after->parts = b.feed_forward_parts;
  after->n = clusters;
  after->bias = b.b2;
  return HL_OK;
}

int decode_row(hl_ctx* ctx, const DecodeRow& r, int dtype, int d) {
  const int grid = ceil_div(d, 256);
  if (dtype == HL_BF16) HL_CUDA(launch_pdl(decode_row_kernel<__nv_bfloat16, float>, grid, 256, 0, ctx->stream, 1, r, d));
  else HL_CUDA(launch_pdl(decode_row_kernel<float, double>, grid, 256, 0, ctx->stream, 1, r, d));
  count_launch(ctx);
  return HL_OK;
}

int decode_head_row(hl_ctx* ctx, const DecodeRow& x, int dtype, const float* gamma, const float* beta, const void* w, const float* bias,
                    float* out, int n, int d) {
  const HeadArgs a{x, gamma, beta, w, bias, out, n, d};
  return dtype == HL_BF16 ? run_head<__nv_bfloat16, float>(ctx, a) : run_head<float, double>(ctx, a);
}

}  // namespace hl
