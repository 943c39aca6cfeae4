// Causal flash attention backward with the scores transposed, keys as rows, for heads of 128 channels where there is work for every
// SM (attention_bwd128.cu has the kernel for fewer heads or shorter rows, attention_bwd.cu the rule and the passes around both).  A work
// item is 128 keys of one (batch, head) and walks the query tiles of 128 at or below the diagonal, one persistent CTA per SM:
//     Sᵀ = K·Qᵀ     dPᵀ = V·dOᵀ     dV += Pᵀ·dO     dK += dSᵀ·Q     dQ_tile = dS·K
//
// With queries as rows, P and dS handed over through shared memory and the 64-key tiles that then fit, the kernel moves 448 KB of
// shared memory a 128 x 64 tile, 3584 of its 4700 cycles.  With keys as rows Pᵀ and dSᵀ are A operands as they leave the registers, so
// they go back into tensor memory over the scores they came from; dS goes to shared memory once, for dQ, and tiles of 128 x 128 halve
// what dQ costs there: 480 KB a 128 x 128 tile.  The whole backward call, before and after: B4 H12 T4096 1046 and 632 us, B16 H6 T1024
// 188 and 126.  What bounds it now: the path out of the SM, 70 % busy with dQ's 64 KB of f32 reductions a tile, and the chain of
// hand-overs dS -> dK -> dQ -> read-out -> dP -> dS (the tensor core is busy half of the time).  Sixteen softmax warps of 32 queries
// instead of eight of 64 were slower (685 us); the same kernel for 64 channels was as fast as the one there is.  Scores worked on two an
// instruction: 579 -> 573.5 us.
//
// Tensor memory (512 columns): dV and dK 128 each, S and Pᵀ over it 128, and 128 for dP, dSᵀ over it and dQ over that once dK has read
// it.  S of tile g + 1 follows dV of tile g, beside the softmax warps' work on dS; dP of tile g + 1 follows the read-out of dQ.  Only
// products into the same accumulator are sure to run in the order they are issued in, so S waits for the end of the dV whose Pᵀ it
// overwrites and dQ for that of the dK whose dSᵀ it overwrites (B4 H12 T4096 592 us without, 612 with).
//
// Warps: eight for the softmax (each 32 keys x 64 queries), four that read dQ out of tensor memory and add it to the f32
// accumulator by TMA reductions, store dK and dV, and supply the rows' statistics; one for loads, one for products.
#include "attention_bwd.cuh"
#include "tc05.cuh"

namespace hl {
namespace {

constexpr int BT_TILE = 128;                      // queries and keys of a tile
constexpr int BT_HD = 128;
constexpr int BT_CHUNK = BT_TILE * 128;           // 64 channels (or queries) of 128 rows: 16 KB
constexpr int BT_OPERAND = BT_HD / 64 * BT_CHUNK;  // 32 KB
constexpr int BT_Q_STAGES = 2;                    // S of the next tile and dK of this one
constexpr int BT_SOFTMAX_WARPS = 8, BT_DRAIN_WARPS = 4;
constexpr int BT_THREADS = (BT_SOFTMAX_WARPS + BT_DRAIN_WARPS + 2) * 32;
constexpr int BT_STAGING = 2 * 4096;              // of a drain warp: two pieces of 32 rows x 128 bytes
constexpr int BT_DATA = (2 + BT_Q_STAGES + 1) * BT_OPERAND + 2 * BT_CHUNK + BT_DRAIN_WARPS * BT_STAGING;  // 224 KB

struct BtTail {
  float lse[2][BT_TILE], delta[2][BT_TILE];       // of the tile's queries: -lse log2(e), -delta scale
  uint64_t kv_full, kv_empty, q_full[BT_Q_STAGES], q_empty[BT_Q_STAGES], do_full, do_empty;
  uint64_t s_full, dp_full, p_ready, ds_ready[2], dq_full, dq_read, dkv_full, dkv_read;
  uint64_t stat_full[2], stat_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int BT_SMEM = BT_DATA + (int)sizeof(BtTail);
static_assert(BT_SMEM <= 227 * 1024, "shared memory budget");

// A CTA's place in its sequence of query tiles; every warp role advances an identical copy.
struct BtCursor {
  int item, local, it, n_tiles;
  int kj, b, h;  // key tile, batch, head
  __device__ __forceinline__ bool valid() const { return item >= 0; }
  __device__ __forceinline__ bool last() const { return it == n_tiles - 1; }
  __device__ __forceinline__ int q0() const { return (kj + it) * BT_TILE; }
};
// Items by decreasing walk length; rounds alternate direction, which evens out the CTAs' totals.
__device__ __forceinline__ void bt_load_item(BtCursor& c, int local, const FbParams& p) {
  const int n = (p.T + BT_TILE - 1) / BT_TILE, heads = p.B * p.H;
  const int grid = (int)gridDim.x, cta = (int)blockIdx.x;
  const int item = local * grid + ((local & 1) ? grid - 1 - cta : cta);
  if (item >= n * heads) { c.item = -1; return; }
  c.item = item;
  c.local = local;
  c.it = 0;
  c.kj = item / heads;
  const int bh = item - c.kj * heads;
  c.b = bh / p.H;
  c.h = bh - c.b * p.H;
  c.n_tiles = n - c.kj;
}
__device__ __forceinline__ BtCursor bt_next(const BtCursor& c, const FbParams& p) {
  BtCursor n = c;
  if (!c.last()) { n.it = c.it + 1; return n; }
  bt_load_item(n, c.local + 1, p);
  return n;
}

__global__ void __launch_bounds__(BT_THREADS, 1)
flash_attention_bwd_t_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                              const __grid_constant__ CUtensorMap map_dq, const __grid_constant__ CUtensorMap map_dk,
                              const __grid_constant__ CUtensorMap map_dv, const FbParams p) {
  extern __shared__ __align__(1024) uint8_t bt_smem[];
  uint8_t* sk = bt_smem;
  uint8_t* sv = sk + BT_OPERAND;
  uint8_t* sq = sv + BT_OPERAND;                       // [stage]
  uint8_t* sdo = sq + BT_Q_STAGES * BT_OPERAND;
  uint8_t* sds = sdo + BT_OPERAND;                     // dS as [64 queries of two][key][query]
  uint8_t* staging = sds + 2 * BT_CHUNK;
  BtTail* tail = reinterpret_cast<BtTail*>(bt_smem + BT_DATA);
  volatile int* abort_flag = &tail->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (uint64_t* b : {&tail->kv_full, &tail->kv_empty, &tail->q_full[0], &tail->q_full[1], &tail->q_empty[0], &tail->q_empty[1],
                        &tail->do_full, &tail->do_empty, &tail->s_full, &tail->dp_full, &tail->dq_full, &tail->dkv_full})
      tc05::mbar_init(b, 1);
    for (uint64_t* b : {&tail->p_ready, &tail->ds_ready[0], &tail->ds_ready[1], &tail->stat_empty[0], &tail->stat_empty[1]})
      tc05::mbar_init(b, BT_SOFTMAX_WARPS);
    for (uint64_t* b : {&tail->dq_read, &tail->dkv_read, &tail->stat_full[0], &tail->stat_full[1]}) tc05::mbar_init(b, BT_DRAIN_WARPS);
    tail->abort_flag = (tc05::smem_u32(bt_smem) & 1023u) == 0 ? 0 : 1;
    tc05::fence_barrier_init();
  }
  if (warp == BT_SOFTMAX_WARPS + BT_DRAIN_WARPS + 1) {
    tc05::tmem_alloc(&tail->tmem_base, 512);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  tc05::tc_fence_after_sync();
  const bool layout_ok = *abort_flag == 0;
  const uint32_t tmem_dv = tail->tmem_base, tmem_dk = tmem_dv + 128;
  const uint32_t tmem_s = tmem_dv + 256, tmem_dp = tmem_dv + 384;  // S, then Pᵀ; dP, then dSᵀ, then dQ
  pdl_begin();  // everything above touches nothing a predecessor wrote

  BtCursor first;
  bt_load_item(first, 0, p);

  if (warp == BT_SOFTMAX_WARPS + BT_DRAIN_WARPS) {
    // -------------------------------------------------------------------------- loads
    if (tc05::elect_one() && !*abort_flag) {
      tc05::tma_prefetch_desc(&map_q);
      tc05::tma_prefetch_desc(&map_k);
      tc05::tma_prefetch_desc(&map_v);
      tc05::tma_prefetch_desc(&map_do);
      // rows past T are zeros, also where another batch entry follows
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row, int b) {
#pragma unroll
        for (int blk = 0; blk < BT_HD / 64; ++blk) tc05::tma_load_3d(dst + blk * BT_CHUNK, map, bar, col + blk * 64, row, b);
      };
      int g = 0;
      for (BtCursor c = first; c.valid(); c = bt_next(c, p), ++g) {
        const int col = c.h * BT_HD, s = g % BT_Q_STAGES;
#pragma unroll
        for (int blk = 0; blk < BT_HD / 64; ++blk) {
          tc05::tma_prefetch_l2_3d(&map_q, col + blk * 64, c.q0(), c.b);
          tc05::tma_prefetch_l2_3d(&map_do, col + blk * 64, c.q0(), c.b);
        }
        if (c.it == 0) {
          if (!tc05::mbar_wait(&tail->kv_empty, ((uint32_t)c.local & 1u) ^ 1u, abort_flag)) break;
          tc05::mbar_arrive_expect_tx(&tail->kv_full, 2 * BT_OPERAND);
          load(sk, &map_k, &tail->kv_full, col, c.kj * BT_TILE, c.b);
          load(sv, &map_v, &tail->kv_full, col, c.kj * BT_TILE, c.b);
        }
        if (!tc05::mbar_wait(&tail->q_empty[s], ((uint32_t)(g / BT_Q_STAGES) & 1u) ^ 1u, abort_flag)) break;
        tc05::mbar_arrive_expect_tx(&tail->q_full[s], BT_OPERAND);
        load(sq + s * BT_OPERAND, &map_q, &tail->q_full[s], col, c.q0(), c.b);
        if (!tc05::mbar_wait(&tail->do_empty, ((uint32_t)g & 1u) ^ 1u, abort_flag)) break;
        tc05::mbar_arrive_expect_tx(&tail->do_full, BT_OPERAND);
        load(sdo, &map_do, &tail->do_full, col, c.q0(), c.b);
      }
    }
  } else if (warp == BT_SOFTMAX_WARPS + BT_DRAIN_WARPS + 1) {
    // -------------------------------------------------------------------------- products
    if (tc05::elect_one() && !*abort_flag) {
      constexpr uint32_t idesc_s = tc05::instr_desc_bf16_f32(128, BT_TILE, false, false);  // keys x queries
      constexpr uint32_t idesc_dkv = tc05::instr_desc_bf16_f32(128, BT_HD, false, true);      // keys x channels, A in tensor memory
      constexpr uint32_t idesc_dq = tc05::instr_desc_bf16_f32(128, BT_HD, true, true);        // queries x channels
      // descriptors step by addition, in 16-byte units
      auto rows_of = [](const uint8_t* p) { return tc05::smem_desc_sw128(tc05::smem_u32(p), 16, 1024); };
      auto chan_of = [](const uint8_t* p) { return tc05::smem_desc_sw128(tc05::smem_u32(p), BT_CHUNK, 1024); };
      auto along = [](int ks) { return (uint64_t)((ks / 4) * (BT_CHUNK >> 4) + (ks % 4) * 2); };  // sixteen channels on
      const uint64_t k_rows = rows_of(sk), v_rows = rows_of(sv), do_rows = rows_of(sdo), k_chan = chan_of(sk), do_chan = chan_of(sdo);
      const uint64_t ds_cols = chan_of(sds);
      auto issue_s = [&](const BtCursor& c, int g) -> bool {
        const int s = g % BT_Q_STAGES;
        if (c.it == 0 && !tc05::mbar_wait(&tail->kv_full, (uint32_t)c.local & 1u, abort_flag)) return false;
        if (!tc05::mbar_wait(&tail->q_full[s], (uint32_t)(g / BT_Q_STAGES) & 1u, abort_flag)) return false;
        tc05::tc_fence_after_sync();
        const uint64_t q_rows = rows_of(sq + s * BT_OPERAND);
#pragma unroll
        for (int ks = 0; ks < BT_HD / 16; ++ks) tc05::umma_ss(tmem_s, k_rows + along(ks), q_rows + along(ks), idesc_s, ks > 0 ? 1u : 0u);
        tc05::umma_commit(&tail->s_full);
        return true;
      };
      auto issue_dp = [&](int g) -> bool {
        if (!tc05::mbar_wait(&tail->do_full, (uint32_t)g & 1u, abort_flag)) return false;
        tc05::tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < BT_HD / 16; ++ks) tc05::umma_ss(tmem_dp, v_rows + along(ks), do_rows + along(ks), idesc_s, ks > 0 ? 1u : 0u);
        tc05::umma_commit(&tail->dp_full);
        return true;
      };
      BtCursor c = first;
      bool ok = c.valid() && issue_s(c, 0) && issue_dp(0);
      for (int g = 0; ok && c.valid(); ++g) {
        const BtCursor n = bt_next(c, p);
        const uint32_t par = (uint32_t)g & 1u;
        const int s = g % BT_Q_STAGES;
        // Pᵀ and dSᵀ lie in the columns that their own warps read the scores from: 64 queries are 32 columns, 64 apart
        auto packed = [](uint32_t region, int ks) { return region + (uint32_t)((ks / 4) * 64 + (ks % 4) * 8); };
        if (!tc05::mbar_wait(&tail->p_ready, par, abort_flag)) break;
        if (c.it == 0 && c.local > 0 && !tc05::mbar_wait(&tail->dkv_read, (uint32_t)(c.local - 1) & 1u, abort_flag)) break;
        tc05::tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < BT_TILE / 16; ++ks)  // sixteen queries: 2048 bytes, 128 units
          tc05::umma_ts(tmem_dv, packed(tmem_s, ks), do_chan + (uint64_t)(ks * 128), idesc_dkv, (c.it > 0 || ks > 0) ? 1u : 0u);
        tc05::umma_commit(&tail->do_empty);
        // S of the next tile over Pᵀ once dV has read it, beside this tile's dS; the next item's waits for its K, which takes this one's place
        const bool early = n.valid() && n.it > 0;
        if (!tc05::mbar_wait(&tail->do_empty, par, abort_flag)) break;
        if (early && !issue_s(n, g + 1)) break;
        const uint64_t q_chan = chan_of(sq + s * BT_OPERAND);
        bool got = true;
#pragma unroll
        for (int part = 0; part < 2; ++part) {  // of every 64 queries, the first 32 while the others are worked on
          got = got && tc05::mbar_wait(&tail->ds_ready[part], par, abort_flag);
          tc05::tc_fence_after_sync();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int ks = (i / 2) * 4 + part * 2 + (i & 1);
            if (got) tc05::umma_ts(tmem_dk, packed(tmem_dp, ks), q_chan + (uint64_t)(ks * 128), idesc_dkv, (c.it > 0 || ks > 0) ? 1u : 0u);
          }
        }
        if (!got) break;
        tc05::umma_commit(&tail->q_empty[s]);
        if (!tc05::mbar_wait(&tail->q_empty[s], (uint32_t)(g / BT_Q_STAGES) & 1u, abort_flag)) break;  // dK has read dSᵀ
        tc05::tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < BT_TILE / 16; ++ks)  // contraction over the keys
          tc05::umma_ss(tmem_dp, ds_cols + (uint64_t)(ks * 128), k_chan + (uint64_t)(ks * 128), idesc_dq, ks > 0 ? 1u : 0u);
        tc05::umma_commit(&tail->dq_full);
        if (c.last()) {
          tc05::umma_commit(&tail->kv_empty);
          tc05::umma_commit(&tail->dkv_full);
        }
        if (n.valid()) {
          if (!early && !issue_s(n, g + 1)) break;
          if (!tc05::mbar_wait(&tail->dq_read, par, abort_flag)) break;
          tc05::tc_fence_after_sync();
          if (!issue_dp(g + 1)) break;
        }
        c = n;
      }
    }
  } else if (warp >= BT_SOFTMAX_WARPS) {
    // -------------------------------------------------------------------------- dQ, dK and dV out, statistics in
    const int lg = warp & 3;  // tensor-memory lane group
    const uint32_t lane_sel = (uint32_t)(lg * 32) << 16;
    uint8_t* my_stage = staging + lg * BT_STAGING;
    bool ok = !*abort_flag;
    auto supply = [&](const BtCursor& c, int g) -> bool {  // the statistics of tile g's queries
      if (!c.valid()) return true;
      const int t = c.q0() + lg * 32 + lane;
      const bool in = t < p.T;
      const size_t at = ((size_t)c.b * p.H + c.h) * p.T + (in ? t : 0);
      const float lse = in ? __ldg(p.lse + at) : INFINITY;  // rows past T: every P becomes 0
      const float delta = in ? __ldg(p.delta + at) : 0.f;
      if (!tc05::mbar_wait(&tail->stat_empty[g & 1], ((uint32_t)(g >> 1) & 1u) ^ 1u, abort_flag)) return false;
      tail->lse[g & 1][lg * 32 + lane] = -lse * 1.4426950408889634f;
      tail->delta[g & 1][lg * 32 + lane] = -delta * p.scale;
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&tail->stat_full[g & 1]);
      return true;
    };
    // 32 rows x 128 bytes into staging piece i (128-byte swizzle)
    auto stage = [&](int i, const uint32_t (&w)[32]) {
      uint8_t* line = my_stage + i * 4096 + lane * 128;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(line + ((j ^ (lane & 7)) << 4)) = make_uint4(w[j * 4], w[j * 4 + 1], w[j * 4 + 2], w[j * 4 + 3]);
    };
    auto staging_free = [&]() {
      if (lane == 0) tc05::tma_store_wait_read();
      __syncwarp();
    };
    BtCursor c = first;
    ok = ok && supply(c, 0);
    for (int g = 0; ok && c.valid(); ++g) {
      const BtCursor n = bt_next(c, p);
      if (!supply(n, g + 1)) break;
      if (!tc05::mbar_wait(&tail->dq_full, (uint32_t)g & 1u, abort_flag)) break;
      tc05::tc_fence_after_sync();
#pragma unroll
      for (int pair = 0; pair < BT_HD / 64; ++pair) {
        uint32_t a[32], b[32];
        tc05::tmem_ld_32x32b_x32(tmem_dp + lane_sel + pair * 64, a);
        tc05::tmem_ld_32x32b_x32(tmem_dp + lane_sel + pair * 64 + 32, b);
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(a);
        tc05::tmem_ld_fence(b);
        if (pair == BT_HD / 64 - 1) {  // dQ is in registers: its columns may be written again
          tc05::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) tc05::mbar_arrive(&tail->dq_read);
        }
        staging_free();
        stage(0, a);
        stage(1, b);
        tc05::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int col = c.h * BT_HD + pair * 64, t0 = c.q0() + lg * 32;
          tc05::tma_reduce_add_3d(&map_dq, my_stage, col, t0, c.b);
          tc05::tma_reduce_add_3d(&map_dq, my_stage + 4096, col + 32, t0, c.b);
          tc05::tma_store_commit();
        }
      }
      if (c.last()) {  // dV, then dK, as bf16: 64 channels a piece
        if (!tc05::mbar_wait(&tail->dkv_full, (uint32_t)c.local & 1u, abort_flag)) break;
        tc05::tc_fence_after_sync();
#pragma unroll
        for (int i = 0; i < 2 * BT_HD / 64; ++i) {
          const int which = i / (BT_HD / 64), col = (i % (BT_HD / 64)) * 64;
          if (i % 2 == 0) staging_free();
          uint32_t w[32];
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            uint32_t raw[32];
            tc05::tmem_ld_32x32b_x32((which == 0 ? tmem_dv : tmem_dk) + lane_sel + col + part * 32, raw);
            tc05::tmem_ld_wait();
            tc05::tmem_ld_fence(raw);
#pragma unroll
            for (int j = 0; j < 32; j += 2) w[part * 16 + j / 2] = pack_bf16x2(__uint_as_float(raw[j]), __uint_as_float(raw[j + 1]));
          }
          if (i == 2 * BT_HD / 64 - 1) {
            tc05::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc05::mbar_arrive(&tail->dkv_read);
          }
          stage(i % 2, w);
          tc05::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {  // keys past T are clipped by the tensor map
            tc05::tma_store_3d(which == 0 ? &map_dv : &map_dk, my_stage + (i % 2) * 4096, c.h * BT_HD + col, c.kj * BT_TILE + lg * 32, c.b);
            tc05::tma_store_commit();
          }
        }
      }
      c = n;
    }
    if (lane == 0) tc05::tma_store_wait_all();
  } else {
    // -------------------------------------------------------------------------- softmax
    const int lg = warp & 3, half = warp >> 2;  // lane group: 32 keys; which 64 queries
    const int r = lg * 32 + lane;
    const uint32_t at = ((uint32_t)(lg * 32) << 16) + (uint32_t)(half * 64);
    bool ok = !*abort_flag;
    int g = 0;
    auto tile = [&](const BtCursor& c, auto diag_tag) -> bool {
      constexpr bool Diag = decltype(diag_tag)::value;
      const uint32_t par = (uint32_t)g & 1u;
      const uint32_t ts = tmem_s + at, tdp = tmem_dp + at;
      if (!tc05::mbar_wait(&tail->stat_full[g & 1], (uint32_t)(g >> 1) & 1u, abort_flag)) return false;
      const float* lse = tail->lse[g & 1] + half * 64;
      const float* delta = tail->delta[g & 1] + half * 64;
      if (!tc05::mbar_wait(&tail->s_full, par, abort_flag)) return false;
      tc05::tc_fence_after_sync();
      // P = 2^(S scale log2(e) - lse log2(e)), kept in f32 for dS; sixteen queries at a time, the next ones on their way
      float pv[64];
      uint32_t raw[2][16];
      tc05::tmem_ld_32x32b_x16(ts, raw[0]);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(raw[ch & 1]);
        if (ch < 3) tc05::tmem_ld_32x32b_x16(ts + (ch + 1) * 16, raw[(ch + 1) & 1]);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 l = *reinterpret_cast<const float4*>(lse + ch * 16 + i);
          const float2 ll[2] = {make_float2(l.x, l.y), make_float2(l.z, l.w)};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 x = fma2(make_float2(__uint_as_float(raw[ch & 1][i + e]), __uint_as_float(raw[ch & 1][i + e + 1])), both(p.scale_log2), ll[e / 2]);
            float2 v = make_float2(ex2_fast(x.x), ex2_fast(x.y));
            if constexpr (Diag) {  // keys after the query
              if (r > half * 64 + ch * 16 + i + e) v.x = 0.f;
              if (r > half * 64 + ch * 16 + i + e + 1) v.y = 0.f;
            }
            pv[ch * 16 + i + e] = v.x;
            pv[ch * 16 + i + e + 1] = v.y;
          }
          w[i / 2] = pack_bf16x2(pv[ch * 16 + i], pv[ch * 16 + i + 1]);
          w[i / 2 + 1] = pack_bf16x2(pv[ch * 16 + i + 2], pv[ch * 16 + i + 3]);
        }
        tc05::tmem_st_32x32b_x8(ts + ch * 8, w);  // over scores that this thread has read
      }
      tc05::tmem_st_wait();
      tc05::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&tail->p_ready);
      // dS = P (dP - D) scale, the scale folded into both terms.  This tile's dP came after the last tile's dQ had been read out, so
      // dS may be written over what that dQ read.
      if (!tc05::mbar_wait(&tail->dp_full, par, abort_flag)) return false;
      tc05::tc_fence_after_sync();
      uint8_t* line = sds + half * BT_CHUNK + r * 128;
      tc05::tmem_ld_32x32b_x16(tdp, raw[0]);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(raw[ch & 1]);
        if (ch < 3) tc05::tmem_ld_32x32b_x16(tdp + (ch + 1) * 16, raw[(ch + 1) & 1]);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 l = *reinterpret_cast<const float4*>(delta + ch * 16 + i);
          const float2 ll[2] = {make_float2(l.x, l.y), make_float2(l.z, l.w)};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 ds = mul2(make_float2(pv[ch * 16 + i + e], pv[ch * 16 + i + e + 1]),
                                   fma2(make_float2(__uint_as_float(raw[ch & 1][i + e]), __uint_as_float(raw[ch & 1][i + e + 1])), both(p.scale), ll[e / 2]));
            w[(i + e) / 2] = pack_bf16x2(ds.x, ds.y);
          }
        }
        tc05::tmem_st_32x32b_x8(tdp + ch * 8, w);
        *reinterpret_cast<uint4*>(line + (((ch * 2) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(line + (((ch * 2 + 1) ^ (r & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
        if (ch & 1) {
          tc05::tmem_st_wait();
          tc05::fence_proxy_async_smem();
          tc05::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) tc05::mbar_arrive(&tail->ds_ready[ch >> 1]);
        }
      }
      if (lane == 0) tc05::mbar_arrive(&tail->stat_empty[g & 1]);
      return true;
    };
    for (BtCursor c = first; ok && c.valid(); c = bt_next(c, p), ++g) ok = c.it == 0 ? tile(c, std::true_type{}) : tile(c, std::false_type{});
  }

  tc05::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (threadIdx.x == 0) atomicExch(p.status + (layout_ok ? ST_WAIT_EXPIRED : ST_BAD_ARGUMENT), 1);
  }
  if (warp == BT_SOFTMAX_WARPS + BT_DRAIN_WARPS + 1) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc(tmem_dv, 512);
  }
}

}  // namespace

int launch_attention_bwd_t(hl_ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                           const CUtensorMap& mdq, const CUtensorMap& mdk, const CUtensorMap& mdv, const FbParams& p) {
  HL_ALLOW_SHARED(ctx, BT_SMEM, flash_attention_bwd_t_kernel);
  const int items = ceil_div(p.T, BT_TILE) * p.B * p.H;
  pdl(flash_attention_bwd_t_kernel, std::min(items, persistent_sms(ctx)), BT_THREADS, BT_SMEM, ctx->stream)(mq, mk, mv, mdo, mdq, mdk, mdv, p);
  return HL_OK;
}

}  // namespace hl
