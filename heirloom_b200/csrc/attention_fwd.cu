// Causal flash attention forward on tcgen05: S = Q·Kᵀ and O += P·V are tensor-memory
// accumulators, K/V tiles stream in by TMA, the online softmax runs in registers and P goes
// back to the tensor cores through tensor memory.
//
// Replaces the reference's attention forward family — materialised [B,H,T,T] scores
// (src/tensor.rs:4459-4472, tensor_core.ptx:1785-2283) and the mma.sync flash forward that
// recomputes the same QK tile in every one of its hd/8 CTAs (tensor_core.ptx:2284-2981,
// heirloom-kernels/src/cuda.rs:5338-5359).  Saves the per-row log-sum-exp instead of
// row_max/row_denom.
//
// Layout: q, k, v are bf16 row-major [B*T, *] views with heads interleaved along the channel
// dimension (column h*hd + j, as src/tensor.rs:5156-5177), so they may live side by side in
// one fused [B*T, 3C] projection buffer.  A work item is 128 query rows of one (batch, head).
//
// Key tiles of 64; S, P (bf16) and the O accumulator in tensor memory.  Softmax warps (one per tensor-memory lane group, a thread per
// query row) work on tile j while the tensor cores run P·V of tile j-1 and Q·Kᵀ of tile j+1.  P is formed against a reference maximum
// that a row raises only when its maximum has grown by more than 2^8; the row then rescales its O in place (tensor-memory load,
// multiply, store) between two P·V products.  P goes to the tensor cores out of tensor memory: through shared memory it was a third
// of that memory's traffic, which was three quarters of what an SM can do (heads of 128: B4 H12 T4096 211.7 us with it, now 200.5).
//
// Work items go round persistent streams without a gap, several of them on an SM, so that one's tensor work and waits lie under
// another's exponentials: two streams, a CTA each (192 threads, 56 or 112 KB of shared memory, 256 tensor-memory columns), or, for heads of
// 64 in many items, three in one CTA (below).  With a CTA per item (heads of 64, B16 H12 T1024: 69 us) 29 us were starts and ends.
#include <type_traits>

#include "common.cuh"
#include "tc05.cuh"

namespace hl {
namespace {

constexpr int FA_BM = 128;   // query rows per item
constexpr int FA_BN = 64;    // keys per tile
constexpr int FA_SOFTMAX_WARPS = 4;
constexpr int FA_THREADS = (FA_SOFTMAX_WARPS + 2) * 32;  // + TMA warp + MMA warp
constexpr int FA_TMEM_COLS = 256;  // S: 2 x 64 columns, O: head_dim columns (allocations are powers of two)

// A CTA with one stream of items.  Operands wider than one 128-byte swizzle row are kept as blocks of 64 channels side by side: a Q
// block is [128 rows x 128 bytes], a K or V block [64 keys x 128 bytes].
constexpr int FA_K_STAGES = 3, FA_V_STAGES = 2;
constexpr int FA_Q_BLOCK = FA_BM * 128, FA_KV_BLOCK = FA_BN * 128;
template <int HD>
struct FaShape {
  static constexpr int BLOCKS = HD / 64, Q_BYTES = BLOCKS * FA_Q_BLOCK, KV_BYTES = BLOCKS * FA_KV_BLOCK;
  static constexpr int DATA = Q_BYTES + (FA_K_STAGES + FA_V_STAGES) * KV_BYTES;  // 56 or 112 KB
  static constexpr int SMEM = DATA + 256;                                        // barriers behind the tiles
  static_assert(2 * (SMEM + 1024) <= 228 * 1024, "shared memory per SM");
  static_assert(2 * FA_BN + HD <= FA_TMEM_COLS, "tensor memory columns");
};

struct FaShared {
  uint64_t q_full, q_empty;
  uint64_t k_full[FA_K_STAGES], k_empty[FA_K_STAGES];
  uint64_t v_full[FA_V_STAGES], v_empty[FA_V_STAGES];
  uint64_t s_full[2], p_full[2], o_full[2];  // by tile
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(FaShared) <= 256, "barriers outgrow their place");

struct FaParams {
  int B, T, H;
  float* lse;
  QuickDiv by_heads, by_h;  // all heads, a batch entry's
  float scale_log2;  // softmax scale times log2(e)
  int* status;
};

// The items of a CTA, longest walks first; rounds over the CTAs alternate direction, which evens out their totals.  Every warp
// role advances an identical copy.
struct FaItem {
  int local, q0, b, h, n_tiles;  // n_tiles: key tiles of 64 up to and including the diagonal; 0: no more items
};
__device__ __forceinline__ FaItem fa_item(int local, const FaParams& p, int cta, int grid) {
  const int nq = (p.T + FA_BM - 1) / FA_BM, heads = p.B * p.H;
  const int item = local * grid + ((local & 1) ? grid - 1 - cta : cta);
  FaItem it{local, 0, 0, 0, 0};
  if (item >= nq * heads) return it;
  const int round = p.by_heads(item), qi = nq - 1 - round, bh = item - round * heads;
  it.q0 = qi * FA_BM;
  it.b = p.by_h(bh);
  it.h = bh - it.b * p.H;
  it.n_tiles = 2 * (qi + 1);
  return it;
}

__device__ __forceinline__ FaItem fa_item(int local, const FaParams& p) { return fa_item(local, p, (int)blockIdx.x, (int)gridDim.x); }

template <int HD>
__global__ void __launch_bounds__(FA_THREADS, 2)
flash_attention_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                           const FaParams p) {
  using Z = FaShape<HD>;
  extern __shared__ __align__(1024) uint8_t fa_smem[];  // swizzled tiles want 1024 bytes; checked below
  uint8_t* sq = fa_smem;
  uint8_t* sk = sq + Z::Q_BYTES;
  uint8_t* sv = sk + FA_K_STAGES * Z::KV_BYTES;
  FaShared* sh = reinterpret_cast<FaShared*>(fa_smem + Z::DATA);
  const bool layout_ok = (tc05::smem_u32(fa_smem) & 1023u) == 0;
  volatile int* abort_flag = &sh->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < FA_K_STAGES; ++s) {
      tc05::mbar_init(&sh->k_full[s], 1);
      tc05::mbar_init(&sh->k_empty[s], 1);
    }
    for (int s = 0; s < FA_V_STAGES; ++s) {
      tc05::mbar_init(&sh->v_full[s], 1);
      tc05::mbar_init(&sh->v_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc05::mbar_init(&sh->s_full[i], 1);
      tc05::mbar_init(&sh->p_full[i], FA_SOFTMAX_WARPS);
      tc05::mbar_init(&sh->o_full[i], 1);
    }
    tc05::mbar_init(&sh->q_full, 1);
    tc05::mbar_init(&sh->q_empty, FA_SOFTMAX_WARPS);
    sh->abort_flag = layout_ok ? 0 : 1;
    tc05::fence_barrier_init();
  }
  if (warp == FA_SOFTMAX_WARPS + 1) {
    tc05::tmem_alloc(&sh->tmem_base, FA_TMEM_COLS);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  tc05::tc_fence_after_sync();
  const uint32_t tmem_s0 = sh->tmem_base;         // S buffers at +0 and +64, P over the S it is formed from
  const uint32_t tmem_o0 = tmem_s0 + 2 * FA_BN;   // O at +128
  pdl_begin();  // everything above touches nothing a predecessor wrote

  if (warp == FA_SOFTMAX_WARPS) {
    // -------------------------------------------------------------------------- TMA producer
    if (tc05::elect_one() && !*abort_flag) {
      tc05::tma_prefetch_desc(&map_q);
      tc05::tma_prefetch_desc(&map_k);
      tc05::tma_prefetch_desc(&map_v);
      bool ok = true;
      int g = 0;  // key tiles loaded so far
      for (FaItem it = fa_item(0, p); ok && it.n_tiles > 0; it = fa_item(it.local + 1, p)) {
        if (!tc05::mbar_wait(&sh->q_empty, ((uint32_t)it.local & 1u) ^ 1u, abort_flag)) break;
        tc05::mbar_arrive_expect_tx(&sh->q_full, Z::Q_BYTES);
#pragma unroll
        for (int blk = 0; blk < Z::BLOCKS; ++blk)
          tc05::tma_load_3d(sq + blk * FA_Q_BLOCK, &map_q, &sh->q_full, it.h * HD + blk * 64, it.q0, it.b);
        for (int j = 0; j < it.n_tiles; ++j, ++g) {
          const int s = g % FA_K_STAGES, vs = g % FA_V_STAGES;
          ok = tc05::mbar_wait(&sh->k_empty[s], ((uint32_t)(g / FA_K_STAGES) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          tc05::mbar_arrive_expect_tx(&sh->k_full[s], Z::KV_BYTES);
#pragma unroll
          for (int blk = 0; blk < Z::BLOCKS; ++blk)
            tc05::tma_load_3d(sk + s * Z::KV_BYTES + blk * FA_KV_BLOCK, &map_k, &sh->k_full[s], it.h * HD + blk * 64,
                              j * FA_BN, it.b);
          ok = tc05::mbar_wait(&sh->v_empty[vs], ((uint32_t)(g / FA_V_STAGES) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          tc05::mbar_arrive_expect_tx(&sh->v_full[vs], Z::KV_BYTES);
#pragma unroll
          for (int blk = 0; blk < Z::BLOCKS; ++blk)
            tc05::tma_load_3d(sv + vs * Z::KV_BYTES + blk * FA_KV_BLOCK, &map_v, &sh->v_full[vs], it.h * HD + blk * 64,
                              j * FA_BN, it.b);
        }
      }
    }
  } else if (warp == FA_SOFTMAX_WARPS + 1) {
    // -------------------------------------------------------------------------- MMA issuer
    if (tc05::elect_one() && !*abort_flag) {
      constexpr uint32_t idesc_qk = tc05::instr_desc_bf16_f32(FA_BM, FA_BN, false, false);
      constexpr uint32_t idesc_pv = tc05::instr_desc_bf16_f32(FA_BM, HD, false, true);
      // Q·Kᵀ runs two tiles ahead of P·V, into the next item where this one ends.
      FaItem qi = fa_item(0, p);
      int qj = 0, qg = 0;  // the next scores: tile of the item, tile of the CTA
      auto issue_qk = [&]() -> bool {  // S[qg & 1] = Q · K(qj)ᵀ
        if (qi.n_tiles == 0) return true;
        const int s = qg % FA_K_STAGES;
        if (qj == 0 && !tc05::mbar_wait(&sh->q_full, (uint32_t)qi.local & 1u, abort_flag)) return false;
        if (!tc05::mbar_wait(&sh->k_full[s], (uint32_t)(qg / FA_K_STAGES) & 1u, abort_flag)) return false;
        // P·V of two tiles before reads the P that stands here: products of other sizes are not kept in order
        if (qg >= 2 && !tc05::mbar_wait(&sh->o_full[qg & 1], (uint32_t)((qg - 2) >> 1) & 1u, abort_flag)) return false;
        tc05::tc_fence_after_sync();
        const uint32_t aq = tc05::smem_u32(sq), ak = tc05::smem_u32(sk + s * Z::KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)  // 16 channels a step; four steps per 64-channel block
          tc05::umma_ss(tmem_s0 + (uint32_t)((qg & 1) * FA_BN),
                        tc05::smem_desc_sw128(aq + (ks / 4) * FA_Q_BLOCK + (ks % 4) * 32, 16, 1024),
                        tc05::smem_desc_sw128(ak + (ks / 4) * FA_KV_BLOCK + (ks % 4) * 32, 16, 1024), idesc_qk,
                        ks > 0 ? 1u : 0u);
        tc05::umma_commit(&sh->k_empty[s]);
        tc05::umma_commit(&sh->s_full[qg & 1]);
        ++qg;
        if (++qj == qi.n_tiles) {
          qi = fa_item(qi.local + 1, p);
          qj = 0;
        }
        return true;
      };
      bool ok = issue_qk();
      // Q is overwritten once the item's result has left through its place, which the softmax warps do after the last P·V: the scores of
      // the next item wait until those have been issued.
      auto may_run_ahead = [&]() { return qj > 0; };
      int ahead = 1;  // scores issued beyond the tile at hand
      int g = 0;
      for (FaItem it = fa_item(0, p); ok && it.n_tiles > 0; it = fa_item(it.local + 1, p)) {
        for (int j = 0; j < it.n_tiles && ok; ++j, ++g) {
          while (ok && ahead < 2 && qi.n_tiles > 0 && may_run_ahead()) {
            ok = issue_qk();
            ++ahead;
          }
          if (!ok) break;
          // P(g) stands in S(g)'s columns and, in an item's first tile, the last item's O has been read
          if (!tc05::mbar_wait(&sh->p_full[g & 1], (uint32_t)(g >> 1) & 1u, abort_flag)) { ok = false; break; }
          tc05::tc_fence_after_sync();
          const int s = g % FA_V_STAGES;
          if (!tc05::mbar_wait(&sh->v_full[s], (uint32_t)(g / FA_V_STAGES) & 1u, abort_flag)) { ok = false; break; }
          tc05::tc_fence_after_sync();
          const uint32_t av = tc05::smem_u32(sv + s * Z::KV_BYTES);
#pragma unroll
          for (int ks = 0; ks < FA_BN / 16; ++ks) {
            // A = P, two keys a column; B = V: rows are keys (MN-major), 16 keys per step, channel blocks FA_KV_BLOCK apart
            const uint64_t db = tc05::smem_desc_sw128(av + ks * (16 * 128), FA_KV_BLOCK, 1024);
            tc05::umma_ts(tmem_o0, tmem_s0 + (uint32_t)((g & 1) * FA_BN + ks * 8), db, idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
          }
          tc05::umma_commit(&sh->v_empty[s]);
          tc05::umma_commit(&sh->o_full[g & 1]);
          --ahead;
          if (ahead < 1 && qi.n_tiles > 0) {  // at the end of an item
            ok = issue_qk();
            ++ahead;
          }
        }
      }
    }
  } else {
    // -------------------------------------------------------------------------- softmax warps
    const int r = warp * 32 + lane;     // query row within the tile == tensor-memory lane
    const uint32_t lane_sel = (uint32_t)(warp * 32) << 16;
    // O accumulates in tensor memory against a reference maximum m_ref that is only raised when a row's maximum has
    // grown by more than 2^8 since: P = 2^(s - m_ref) then stays below 256, which costs bf16 nothing (same relative
    // precision) and f32 sums nothing, and O is rescaled in place a few times per row instead of once per tile.
    constexpr float kRaise = 8.0f;
    bool ok = !*abort_flag;
    int g = 0;            // key tiles done so far

    for (FaItem it = fa_item(0, p); ok && it.n_tiles > 0; it = fa_item(it.local + 1, p)) {
    const int n_tiles = it.n_tiles, t = it.q0 + r;  // query position within the batch
    float m_ref = -INFINITY;   // reference maximum, in log2 units
    float l_run = 0.f;         // row sum, scaled to m_ref
    for (int j = 0; j < n_tiles && ok; ++j, ++g) {
      if (!tc05::mbar_wait(&sh->s_full[g & 1], (uint32_t)(g >> 1) & 1u, abort_flag)) { ok = false; break; }
      tc05::tc_fence_after_sync();
      const bool diag = (j >= n_tiles - 2);  // the two tiles that hold keys q0 .. q0+127
      const int key0 = j * FA_BN;
      uint32_t sb[FA_BN];
      tc05::tmem_ld_32x32b_x32(tmem_s0 + (uint32_t)((g & 1) * FA_BN) + lane_sel, *reinterpret_cast<uint32_t(*)[32]>(&sb[0]));
      tc05::tmem_ld_32x32b_x32(tmem_s0 + (uint32_t)((g & 1) * FA_BN) + lane_sel + 32, *reinterpret_cast<uint32_t(*)[32]>(&sb[32]));
      tc05::tmem_ld_wait();
      // maximum of the raw scores (the scale is positive); masked entries become -inf
      float m_tile = -INFINITY;
      if (diag) {
#pragma unroll
        for (int i = 0; i < FA_BN; ++i)
          if (key0 + i > t) sb[i] = 0xff800000u;
      }
      {  // eight independent running maxima, so that the 64 comparisons are not one dependent chain
        float mx[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) mx[u] = __uint_as_float(sb[u]);
#pragma unroll
        for (int i = 8; i < FA_BN; ++i) mx[i & 7] = fmaxf(mx[i & 7], __uint_as_float(sb[i]));
        m_tile = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
      }
      const float m_new = m_tile * p.scale_log2;  // finite in tile 0: key 0 is visible to every row
      const bool raise = m_new > m_ref + kRaise;  // always true in tile 0 (m_ref = -inf)
      if (j == 0) {
        m_ref = m_new;
      } else if (__any_sync(0xffffffffu, raise)) {
        // rows of this warp rescale their O in place; P·V of tile j-1 must have landed, and P·V of tile j is not
        // issued before this warp has handed over P(j)
        if (!tc05::mbar_wait(&sh->o_full[(g - 1) & 1], (uint32_t)((g - 1) >> 1) & 1u, abort_flag)) { ok = false; break; }
        tc05::tc_fence_after_sync();
        const float a = raise ? ex2_fast(m_ref - m_new) : 1.0f;
        if (raise) m_ref = m_new;
        l_run *= a;
#pragma unroll
        for (int hb = 0; hb < HD / 32; ++hb) {
          uint32_t ob[32];
          tc05::tmem_ld_32x32b_x32(tmem_o0 + lane_sel + hb * 32, ob);
          tc05::tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 32; ++k) ob[k] = __float_as_uint(__uint_as_float(ob[k]) * a);
          tc05::tmem_st_32x32b_x32(tmem_o0 + lane_sel + hb * 32, ob);
        }
        tc05::tmem_st_wait();
      }
      const float neg_m = -m_ref;
      const uint32_t tp = tmem_s0 + (uint32_t)((g & 1) * FA_BN) + lane_sel;
      float l_tile = 0.f;  // key after key, as ever: the results are the same bits
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // sixteen keys
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float2 x = fma2(make_float2(__uint_as_float(sb[q * 16 + 2 * e]), __uint_as_float(sb[q * 16 + 2 * e + 1])),
                                both(p.scale_log2), both(neg_m));
          const float2 pr = make_float2(ex2_fast(x.x), ex2_fast(x.y));
          l_tile += pr.x + pr.y;
          w[e] = pack_bf16x2(pr.x, pr.y);
        }
        tc05::tmem_st_32x32b_x8(tp + q * 8, w);
      }
      l_run += l_tile;
      tc05::tmem_st_wait();
      tc05::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&sh->p_full[g & 1]);
    }
    if (!ok) break;
    ok = tc05::mbar_wait(&sh->o_full[(g - 1) & 1], (uint32_t)((g - 1) >> 1) & 1u, abort_flag);  // the last P·V
    tc05::tc_fence_after_sync();
    if (ok) {
      // O leaves through the Q tile's shared memory (every product that read Q has finished): a warp stages its 32
      // rows per 64-channel block (128-byte rows, 128-byte swizzle) and its lane 0 sends them with one TMA store, whole
      // 128-byte row segments instead of 16-byte stores that each touch 32 different lines.  Rows past T are clipped by
      // the tensor map.
      const float inv = 1.0f / l_run;
#pragma unroll
      for (int hb = 0; hb < HD / 32; ++hb) {
        uint32_t ob[32];
        tc05::tmem_ld_32x32b_x32(tmem_o0 + lane_sel + hb * 32, ob);
        tc05::tmem_ld_wait();
        uint8_t* line = sq + (hb / 2) * FA_Q_BLOCK + r * 128;
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(ob[i]) * inv, __uint_as_float(ob[i + 1]) * inv);
          o.y = pack_bf16x2(__uint_as_float(ob[i + 2]) * inv, __uint_as_float(ob[i + 3]) * inv);
          o.z = pack_bf16x2(__uint_as_float(ob[i + 4]) * inv, __uint_as_float(ob[i + 5]) * inv);
          o.w = pack_bf16x2(__uint_as_float(ob[i + 6]) * inv, __uint_as_float(ob[i + 7]) * inv);
          const int chunk = (hb & 1) * 4 + i / 8;  // 16-byte chunk of the 128-byte row
          *reinterpret_cast<uint4*>(line + ((chunk ^ (r & 7)) << 4)) = o;
        }
      }
      tc05::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (int blk = 0; blk < Z::BLOCKS; ++blk)
          tc05::tma_store_3d(&map_o, sq + blk * FA_Q_BLOCK + warp * (32 * 128), it.h * HD + blk * 64, it.q0 + warp * 32, it.b);
        tc05::tma_store_commit();
        tc05::tma_store_wait_read();  // the next item's Q waits for it
        tc05::mbar_arrive(&sh->q_empty);
      }
    }
    if (ok && t < p.T) {
      // natural-log log-sum-exp of the scaled scores
      p.lse[((size_t)it.b * p.H + it.h) * p.T + t] = (m_ref + log2f(l_run)) * 0.6931471805599453f;
    }
    }
    if (lane == 0) tc05::tma_store_wait_all();  // the results have landed before shared memory goes
  }

  tc05::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (threadIdx.x == 0) atomicExch(p.status + (layout_ok ? ST_WAIT_EXPIRED : ST_BAD_ARGUMENT), 1);
  }
  if (warp == FA_SOFTMAX_WARPS + 1) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc(tmem_s0, FA_TMEM_COLS);
  }
}

// ---- heads of 64 channels, many items ---------------------------------------------------------------------------------------
// What bounds these is the softmax: 64 exponentials a row and tile are 512 cycles of a scheduler's, the products 256.  A warp's chain (scores,
// maximum, exponentials, hand-over) takes three times that, so that three warps share a scheduler: one CTA an SM walks three streams
// of items side by side, each with its own tiles, four softmax warps and a warp whose elected thread queues both loads and products
// (B16 H12 T1024: two CTAs of four softmax warps 62.8 us, three streams 58.3, P in tensor memory and its place waited for
// when half of P has been formed 54.9; B4 H12 T4096 175.5, 176.5, 167).
// That thread waits for scores that have been read and P that has been written, and for nothing else: when S(g) has been read, Q·K(g)
// is done and K(g) can be replaced; when P(g) has been written, P·V(g-1) is done and V(g-1) can.
// A stream has S, P and O in tensor memory (160 columns), and Q, a place for the result, three K and two V in shared memory: 72 KB.
constexpr int F3_STREAMS = 3;
constexpr int F3_THREADS = F3_STREAMS * 5 * 32;
constexpr int F3_K_STAGES = 3, F3_V_STAGES = 2;
constexpr int F3_TMEM_COLS = FA_BN + FA_BN / 2 + 64;  // S, P in bf16, O
static_assert(F3_STREAMS * F3_TMEM_COLS <= 512, "tensor memory columns");
constexpr int F3_Q_BYTES = FA_BM * 128, F3_KV_BYTES = FA_BN * 128;
constexpr int F3_O_BYTES = F3_Q_BYTES;
constexpr int F3_STREAM_BYTES = F3_Q_BYTES + F3_O_BYTES + (F3_K_STAGES + F3_V_STAGES) * F3_KV_BYTES;
struct F3Shared {
  uint64_t q_full, k_full[F3_K_STAGES], v_full[F3_V_STAGES], s_full, s_empty, p_full, o_full;
};
constexpr int F3_SMEM = F3_STREAMS * F3_STREAM_BYTES + 512;
static_assert(F3_STREAMS * sizeof(F3Shared) + 8 <= 512 && F3_SMEM <= 227 * 1024, "shared memory budget");

__global__ void __launch_bounds__(F3_THREADS, 1)
flash_attention_fwd64_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                             const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o, const FaParams p) {
  extern __shared__ __align__(1024) uint8_t fa_smem[];  // swizzled tiles want 1024 bytes; checked below
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool control = warp >= F3_STREAMS * 4;
  const int stream = control ? warp - F3_STREAMS * 4 : warp >> 2;
  uint8_t* sq = fa_smem + stream * F3_STREAM_BYTES;
  uint8_t* so = sq + F3_Q_BYTES;
  uint8_t* sk = so + F3_O_BYTES;
  uint8_t* sv = sk + F3_K_STAGES * F3_KV_BYTES;
  F3Shared* all = reinterpret_cast<F3Shared*>(fa_smem + F3_STREAMS * F3_STREAM_BYTES);
  F3Shared* sh = all + stream;
  uint32_t* tmem_base = reinterpret_cast<uint32_t*>(all + F3_STREAMS);
  int* abort_word = reinterpret_cast<int*>(tmem_base + 1);
  volatile int* abort_flag = abort_word;
  const bool layout_ok = (tc05::smem_u32(fa_smem) & 1023u) == 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < F3_STREAMS; ++i) {
      tc05::mbar_init(&all[i].q_full, 1);
      for (int s = 0; s < F3_K_STAGES; ++s) tc05::mbar_init(&all[i].k_full[s], 1);
      for (int s = 0; s < F3_V_STAGES; ++s) tc05::mbar_init(&all[i].v_full[s], 1);
      tc05::mbar_init(&all[i].s_full, 1);
      tc05::mbar_init(&all[i].s_empty, 4);
      tc05::mbar_init(&all[i].p_full, 4);
      tc05::mbar_init(&all[i].o_full, 1);
    }
    *abort_word = layout_ok ? 0 : 1;
    tc05::fence_barrier_init();
  }
  if (warp == F3_STREAMS * 4) {
    tc05::tmem_alloc(tmem_base, 512);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  tc05::tc_fence_after_sync();
  const uint32_t tmem_s = *tmem_base + (uint32_t)(stream * F3_TMEM_COLS), tmem_p = tmem_s + FA_BN, tmem_o = tmem_p + FA_BN / 2;
  pdl_begin();  // everything above touches nothing a predecessor wrote

  const int grid = F3_STREAMS * (int)gridDim.x, cta = stream * (int)gridDim.x + (int)blockIdx.x;
  auto item = [&](int local) { return fa_item(local, p, cta, grid); };
  if (control) {
    // -------------------------------------------------------------------------- loads and products of one stream
    if (tc05::elect_one() && !*abort_flag) {
      tc05::tma_prefetch_desc(&map_q);
      tc05::tma_prefetch_desc(&map_k);
      tc05::tma_prefetch_desc(&map_v);
      constexpr uint32_t idesc_qk = tc05::instr_desc_bf16_f32(FA_BM, FA_BN, false, false);
      constexpr uint32_t idesc_pv = tc05::instr_desc_bf16_f32(FA_BM, 64, false, true);
      // the next tile to load (K, V) or to score, each with its item, its place in the item and its number in the stream
      struct Cursor {
        FaItem it;
        int j, g;
      };
      auto advance = [&](Cursor& c) {
        ++c.g;
        if (++c.j == c.it.n_tiles) {
          c.it = item(c.it.local + 1);
          c.j = 0;
        }
      };
      const FaItem first = item(0);
      Cursor ck{first, 0, 0}, cv{first, 0, 0}, cs{first, 0, 0};
      auto load_q = [&](const FaItem& it) {
        if (it.n_tiles == 0) return;
        tc05::mbar_arrive_expect_tx(&sh->q_full, F3_Q_BYTES);
        tc05::tma_load_3d(sq, &map_q, &sh->q_full, it.h * 64, it.q0, it.b);
      };
      auto load_k = [&]() {
        if (ck.it.n_tiles == 0) return;
        const int s = ck.g % F3_K_STAGES;
        tc05::mbar_arrive_expect_tx(&sh->k_full[s], F3_KV_BYTES);
        tc05::tma_load_3d(sk + s * F3_KV_BYTES, &map_k, &sh->k_full[s], ck.it.h * 64, ck.j * FA_BN, ck.it.b);
        advance(ck);
      };
      auto load_v = [&]() {
        if (cv.it.n_tiles == 0) return;
        const int s = cv.g % F3_V_STAGES;
        tc05::mbar_arrive_expect_tx(&sh->v_full[s], F3_KV_BYTES);
        tc05::tma_load_3d(sv + s * F3_KV_BYTES, &map_v, &sh->v_full[s], cv.it.h * 64, cv.j * FA_BN, cv.it.b);
        advance(cv);
      };
      auto scores = [&]() -> bool {  // S = Q · Kᵀ of the next tile
        if (cs.it.n_tiles == 0) return true;
        if (cs.j == 0 && !tc05::mbar_wait(&sh->q_full, (uint32_t)cs.it.local & 1u, abort_flag)) return false;
        const int s = cs.g % F3_K_STAGES;
        if (!tc05::mbar_wait(&sh->k_full[s], (uint32_t)(cs.g / F3_K_STAGES) & 1u, abort_flag)) return false;
        tc05::tc_fence_after_sync();
        const uint32_t aq = tc05::smem_u32(sq), ak = tc05::smem_u32(sk + s * F3_KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          tc05::umma_ss(tmem_s, tc05::smem_desc_sw128(aq + ks * 32, 16, 1024), tc05::smem_desc_sw128(ak + ks * 32, 16, 1024), idesc_qk, ks > 0 ? 1u : 0u);
        tc05::umma_commit(&sh->s_full);
        advance(cs);
        return true;
      };
      load_q(first);
      load_k();
      load_v();
#pragma unroll 1
      for (int i = 1; i < F3_K_STAGES; ++i) load_k();
#pragma unroll 1
      for (int i = 1; i < F3_V_STAGES; ++i) load_v();
      bool ok = scores();
      int g = 0;
      for (FaItem it = first; ok && it.n_tiles > 0; it = item(it.local + 1)) {
        for (int j = 0; j < it.n_tiles; ++j, ++g) {
          ok = tc05::mbar_wait(&sh->s_empty, (uint32_t)g & 1u, abort_flag);  // S(g) has been read
          if (!ok) break;
          load_k();
          if (j + 1 == it.n_tiles) load_q(item(it.local + 1));
          ok = scores();
          if (!ok) break;
          // P(g) has been written and, in an item's first tile, the last item's O read
          ok = tc05::mbar_wait(&sh->p_full, (uint32_t)g & 1u, abort_flag);
          if (!ok) break;
          if (g > 0) load_v();  // in the place of V(g - 1)
          const int s = g % F3_V_STAGES;
          ok = tc05::mbar_wait(&sh->v_full[s], (uint32_t)(g / F3_V_STAGES) & 1u, abort_flag);
          if (!ok) break;
          tc05::tc_fence_after_sync();
          const uint32_t av = tc05::smem_u32(sv + s * F3_KV_BYTES);
#pragma unroll
          for (int ks = 0; ks < FA_BN / 16; ++ks)  // A = P, two keys a column; B = V: rows are keys (MN-major), 16 keys per step
            tc05::umma_ts(tmem_o, tmem_p + ks * 8, tc05::smem_desc_sw128(av + ks * (16 * 128), F3_KV_BYTES, 1024), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
          tc05::umma_commit(&sh->o_full);
        }
      }
    }
  } else {
    // -------------------------------------------------------------------------- softmax warps
    const int rows = warp & 3;          // tensor-memory lanes and query rows of this warp
    const int r = rows * 32 + lane;     // query row within the tile
    const uint32_t lane_sel = (uint32_t)(rows * 32) << 16;
    uint8_t* line = so + r * 128;
    constexpr float kRaise = 8.0f;      // as above
    bool ok = !*abort_flag, stored = false;  // stored: this warp has staged rows of an item
    int g = 0;
    for (FaItem it = item(0); ok && it.n_tiles > 0; it = item(it.local + 1)) {
      const int t = it.q0 + r;
      float m_ref = -INFINITY, l_run = 0.f;
      for (int j = 0; j < it.n_tiles; ++j, ++g) {
        const int key0 = j * FA_BN, last_row = it.q0 + rows * 32 + 31;
        const int halves = key0 > last_row ? 0 : key0 + 32 > last_row ? 1 : 2;  // halves of the tile that any of this warp's rows sees
        ok = tc05::mbar_wait(&sh->s_full, (uint32_t)g & 1u, abort_flag);
        if (!ok) break;
        tc05::tc_fence_after_sync();
        uint32_t sb[FA_BN];
        if (halves > 0) tc05::tmem_ld_32x32b_x32(tmem_s + lane_sel, *reinterpret_cast<uint32_t(*)[32]>(&sb[0]));
        if (halves > 1) tc05::tmem_ld_32x32b_x32(tmem_s + lane_sel + 32, *reinterpret_cast<uint32_t(*)[32]>(&sb[32]));
        tc05::tmem_ld_wait();
        tc05::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) tc05::mbar_arrive(&sh->s_empty);
        tc05::tmem_ld_fence(sb);
        if (j >= it.n_tiles - 2) {  // the two tiles that hold keys q0 .. q0 + 127
#pragma unroll
          for (int i = 0; i < FA_BN; ++i)
            if (key0 + i > t) sb[i] = 0xff800000u;
        }
        float m_tile;
        {
          float mx[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) mx[u] = __uint_as_float(sb[u]);
#pragma unroll
          for (int i = 8; i < FA_BN; ++i) mx[i & 7] = fmaxf(mx[i & 7], __uint_as_float(sb[i]));
          m_tile = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
        }
        const float m_new = m_tile * p.scale_log2;    // finite in tile 0: key 0 is visible to every row
        const bool raise = m_new > m_ref + kRaise;    // always true in tile 0
        // P·V of the tile before has read P, and O may be rescaled.  Waited for as late as may be.
        bool landed = g == 0;
        auto wait_landed = [&]() {
          if (!landed) ok = tc05::mbar_wait(&sh->o_full, (uint32_t)(g - 1) & 1u, abort_flag);
          landed = true;
          tc05::tc_fence_after_sync();
        };
        if (j == 0) {
          m_ref = m_new;
        } else if (__any_sync(0xffffffffu, raise)) {
          wait_landed();
          if (!ok) break;
          const float a = raise ? ex2_fast(m_ref - m_new) : 1.0f;
          if (raise) m_ref = m_new;
          l_run *= a;
#pragma unroll 1
          for (int c = 0; c < 64; c += 8) {
            uint32_t ob[8];
            tc05::tmem_ld_32x32b_x8(tmem_o + lane_sel + c, ob);
            tc05::tmem_ld_wait();
            tc05::tmem_ld_fence(ob);
#pragma unroll
            for (int k = 0; k < 8; ++k) ob[k] = __float_as_uint(__uint_as_float(ob[k]) * a);
            tc05::tmem_st_32x32b_x8(tmem_o + lane_sel + c, ob);
          }
          tc05::tmem_st_wait();
        }
        const float neg_m = -m_ref;
        float l_tile = 0.f;  // key after key, as ever: the results are the same bits (two chains of pairs: T4096 153 us; the sums behind
                             // the hand-over of P: 182 to 191)
        auto half = [&](auto which, uint32_t (&w)[2][8]) {  // of P, sixteen keys each
          constexpr int H = decltype(which)::value;
          if (halves <= H) {
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e / 8][e % 8] = 0u;
            return;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 x = fma2(make_float2(__uint_as_float(sb[H * 32 + 2 * e]), __uint_as_float(sb[H * 32 + 2 * e + 1])), both(p.scale_log2),
                                  both(neg_m));
            const float2 pr = make_float2(ex2_fast(x.x), ex2_fast(x.y));
            l_tile += pr.x + pr.y;
            w[e / 8][e % 8] = pack_bf16x2(pr.x, pr.y);
          }
        };
        uint32_t w[2][8];
        half(std::integral_constant<int, 0>{}, w);
        wait_landed();
        if (!ok) break;
        tc05::tmem_st_32x32b_x8(tmem_p + lane_sel, w[0]);
        tc05::tmem_st_32x32b_x8(tmem_p + lane_sel + 8, w[1]);
        half(std::integral_constant<int, 1>{}, w);
        tc05::tmem_st_32x32b_x8(tmem_p + lane_sel + 16, w[0]);
        tc05::tmem_st_32x32b_x8(tmem_p + lane_sel + 24, w[1]);
        l_run += l_tile;
        tc05::tmem_st_wait();
        tc05::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) tc05::mbar_arrive(&sh->p_full);
      }
      if (!ok) break;
      ok = tc05::mbar_wait(&sh->o_full, (uint32_t)(g - 1) & 1u, abort_flag);  // the last P·V
      if (!ok) break;
      tc05::tc_fence_after_sync();
      if (stored) {  // the last item's
        if (lane == 0) tc05::tma_store_wait_read();
        __syncwarp();
      }
      // A warp stages its 32 rows of O (128-byte rows, 128-byte swizzle) and its lane 0 sends them with one TMA store.  Rows past T are
      // clipped by the tensor map.
      const float inv = 1.0f / l_run;
#pragma unroll
      for (int hb = 0; hb < 2; ++hb) {
        uint32_t ob[32];
        tc05::tmem_ld_32x32b_x32(tmem_o + lane_sel + hb * 32, ob);
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(ob);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(ob[i]) * inv, __uint_as_float(ob[i + 1]) * inv);
          o.y = pack_bf16x2(__uint_as_float(ob[i + 2]) * inv, __uint_as_float(ob[i + 3]) * inv);
          o.z = pack_bf16x2(__uint_as_float(ob[i + 4]) * inv, __uint_as_float(ob[i + 5]) * inv);
          o.w = pack_bf16x2(__uint_as_float(ob[i + 6]) * inv, __uint_as_float(ob[i + 7]) * inv);
          *reinterpret_cast<uint4*>(line + (((hb * 4 + i / 8) ^ (r & 7)) << 4)) = o;
        }
      }
      tc05::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tc05::tma_store_3d(&map_o, so + rows * (32 * 128), it.h * 64, it.q0 + rows * 32, it.b);
        tc05::tma_store_commit();
      }
      stored = true;
      if (t < p.T) p.lse[((size_t)it.b * p.H + it.h) * p.T + t] = (m_ref + log2f(l_run)) * 0.6931471805599453f;
    }
    if (lane == 0) tc05::tma_store_wait_all();  // the results have landed before shared memory goes
  }

  tc05::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (threadIdx.x == 0) atomicExch(p.status + (layout_ok ? ST_WAIT_EXPIRED : ST_BAD_ARGUMENT), 1);
  }
  if (warp == F3_STREAMS * 4) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc(*tmem_base, 512);
  }
}

// Three streams an SM are more work at a time, two are faster each (0.86 and 0.67 us a tile of a stream that is alone), and a call
// lasts no less than its longest item.  So three where an SM's share of the tiles is a few times that item: share / longest of
// 1.75 + (rows / 128) / 16, and up to 2048 rows.  Two / three streams, us: B16 T512 H8 15.8 / 13.8, B16 T1024 H12 59.6 / 51.1, B16 T1024 H5
// 24.8 / 24.1, B8 T1024 H8 20.8 / 22.5, B4 T2048 H16 62.3 / 61.6, B4 T2048 H10 39.5 / 42.6, B5 T700 H13 14.4 / 16.9, B1 T4096 H16 55 / 75, B1 T4096
// H24 84.6 / 84.1, B2 T4096 H20 133 / 139, B1 T8192 H32 391 / 407.
bool three_streams(int items, int tiles, int sms) {
  return tiles <= 16 && 8ll * items * (tiles + 1) >= (long long)sms * tiles * (28 + tiles);
}

}  // namespace

int flash_attention_forward_impl(hl_ctx* ctx, const void* q, const void* k, const void* v, long long ld_qkv, void* out,
                                 long long ld_out, float* lse, int batch, int time, int n_heads, int head_dim) {
  HL_REQUIRE(ctx && q && k && v && out && lse, "hl_flash_attention_forward: null argument");
  HL_REQUIRE(n_heads > 0, "hl_flash_attention_forward: causal_self_attention requires n_heads > 0");
  HL_REQUIRE(batch > 0 && time > 0, "hl_flash_attention_forward: batch and time must be positive");
  HL_REQUIRE(head_dim == 64 || head_dim == 128, "hl_flash_attention_forward: head_dim must be 64 or 128");
  HL_REQUIRE(ld_qkv % 8 == 0 && ld_out % 8 == 0 && ld_qkv >= (long long)n_heads * head_dim &&
                 ld_out >= (long long)n_heads * head_dim,
             "hl_flash_attention_forward: row strides must be multiples of 8 and cover all heads");
  HL_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
               reinterpret_cast<uintptr_t>(out)) & 15) == 0,
             "hl_flash_attention_forward: pointers must be 16-byte aligned");
  const uint64_t cols = (uint64_t)n_heads * head_dim;
  CUtensorMap mq, mk, mv;
  int rc;
  // boxes of 64 channels (one 128-byte swizzle row); wider heads take several boxes per tile.  [batch][time][channels], so that
  // rows past `time` are zeros: a masked P of zero times another batch entry's infinity would be NaN.
  auto operand_map = [&](CUtensorMap* map, const void* base, uint32_t box_rows) {
    return make_tensor_map_bf16_3d(map, base, cols, (uint64_t)time, (uint64_t)batch, (uint64_t)ld_qkv, (uint64_t)ld_qkv * (uint64_t)time, 64, box_rows, 1);
  };
  if ((rc = operand_map(&mq, q, FA_BM)) != HL_OK) return rc;
  if ((rc = operand_map(&mk, k, FA_BN)) != HL_OK) return rc;
  if ((rc = operand_map(&mv, v, FA_BN)) != HL_OK) return rc;
  // the output as [batch][time][channels], so that a tile's rows past `time` are clipped; boxes of 64 channels by 32 rows
  CUtensorMap mo;
  {
    const uint64_t dims[3] = {(uint64_t)cols, (uint64_t)time, (uint64_t)batch};
    const uint64_t strides[2] = {(uint64_t)ld_out * 2, (uint64_t)time * (uint64_t)ld_out * 2};
    const uint32_t box[3] = {64, 32, 1};
    if ((rc = make_tensor_map(&mo, HL_BF16, 3, out, dims, strides, box, 128)) != HL_OK) return rc;
  }
  FaParams p{};
  p.B = batch; p.T = time; p.H = n_heads;
  p.lse = lse;
  p.by_heads = QuickDiv((uint32_t)(batch * n_heads));
  p.by_h = QuickDiv((uint32_t)n_heads);
  p.scale_log2 = (1.0f / sqrtf((float)head_dim)) * 1.4426950408889634f;
  p.status = ctx->status_dev;
  const int sms = persistent_sms(ctx), tiles = ceil_div(time, FA_BM), items = tiles * batch * n_heads;
  // causal algorithmic work: QK^T and PV over the lower triangle
  ProfileScope prof(ctx, HL_PROF_ATTENTION_FWD, 2.0 * batch * n_heads * (double)time * time * head_dim);
  if (head_dim == 64 && three_streams(items, tiles, sms)) {
    HL_ALLOW_SHARED(ctx, F3_SMEM, flash_attention_fwd64_kernel);
    pdl(flash_attention_fwd64_kernel, std::min(items, sms), F3_THREADS, F3_SMEM, ctx->stream)(mq, mk, mv, mo, p);
  } else if (head_dim == 64) {
    HL_ALLOW_SHARED(ctx, FaShape<64>::SMEM, flash_attention_fwd_kernel<64>);
    pdl(flash_attention_fwd_kernel<64>, std::min(items, 2 * sms), FA_THREADS, FaShape<64>::SMEM, ctx->stream)(mq, mk, mv, mo, p);
  } else {
    HL_ALLOW_SHARED(ctx, FaShape<128>::SMEM, flash_attention_fwd_kernel<128>);
    pdl(flash_attention_fwd_kernel<128>, std::min(items, 2 * sms), FA_THREADS, FaShape<128>::SMEM, ctx->stream)(mq, mk, mv, mo, p);
  }
  HL_LAUNCH_CHECK("flash_attention_fwd_kernel");
  count_launch(ctx);
  ctx->counters.attention_launches += 1;
  return HL_OK;
}

}  // namespace hl

extern "C" int hl_flash_attention_forward(hl_ctx* ctx, const void* q, const void* k, const void* v, long long ld_qkv,
                                          void* out, long long ld_out, float* lse, int batch, int time, int n_heads,
                                          int head_dim) {
  return hl::flash_attention_forward_impl(ctx, q, k, v, ld_qkv, out, ld_out, lse, batch, time, n_heads, head_dim);
}
