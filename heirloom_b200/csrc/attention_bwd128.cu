// Causal flash attention backward for heads of 128 channels (attention_bwd.cu has the 64-channel kernel and the passes around
// both).  Same roles and hand-overs: one persistent CTA per SM, TMA warp, MMA warp, eight softmax warps.  A work item is 64
// keys of one (batch, head) and walks the query tiles of 128 at or below the diagonal.
//
// The tile is what makes the head fit: with 64 keys the operands of two query tiles are in shared memory at once (K and V
// 32 KB, two stages of Q and dO 128 KB, P and dS 32 KB, staging 32 KB), and with dV and dK accumulated transposed, channels by
// keys, every product runs on all 128 rows of the tensor core and tensor memory holds S and dP (64 columns each), dVᵀ and
// dKᵀ (64 each) and two dQ tiles (128 each), so each of the five products is formed once.  A 128-key tile had room for one
// stage and one half of the head at a time: S and dP were formed twice, and every tile waited for its own loads (B4 H12 T4096:
// 1334 us then, 931 us with 64; such sizes take keys as rows now, 632 us for the whole call, and this kernel the few or short heads
// whose longest walk bounds the pass: B2 H4 T2048 53 us against 57).  Bound by shared memory: a product 64 columns wide reads its 128 rows of A for half the work of a
// full tile, which makes the five products worth nine halves, and by the softmax warps' chain that runs beside them.
#include "attention_bwd.cuh"
#include "tc05.cuh"

namespace hl {
namespace {

constexpr int FW_BM = 128, FW_BN = 64, FW_HD = 128;
constexpr int FW_Q_BLOCK = FW_BM * 128;            // 64 channels of a query tile: 16 KB
constexpr int FW_Q_BYTES = 2 * FW_Q_BLOCK;         // 32 KB
constexpr int FW_KV_BLOCK = FW_BN * 128;           // 64 channels of a key tile: 8 KB
constexpr int FW_KV_BYTES = 2 * FW_KV_BLOCK;       // 16 KB
constexpr int FW_P_BYTES = FW_BM * FW_BN * 2;      // 16 KB: [query][64 keys]
constexpr int FW_STAGES = 2;
constexpr int FW_SOFTMAX_WARPS = 8;
constexpr int FW_THREADS = (FW_SOFTMAX_WARPS + 2) * 32;
constexpr int FW_STAGING = 4096;                   // per softmax warp: 32 rows x 32 columns f32
constexpr int FW_DATA = 2 * FW_KV_BYTES + FW_STAGES * 2 * FW_Q_BYTES + 2 * FW_P_BYTES + FW_SOFTMAX_WARPS * FW_STAGING;  // 224 KB
constexpr int FW_SMEM = FW_DATA + 1024;
static_assert(FW_SMEM <= 227 * 1024, "shared memory budget");
constexpr int FW_TMEM_COLS = 512;

struct FwBarriers {
  uint64_t kv_full, kv_empty;
  uint64_t q_full[FW_STAGES], q_empty[FW_STAGES];
  uint64_t sdp_full, sdp_free, p_full, dq_full;
  uint32_t tmem_base;
  int abort_flag;
};

// A CTA's place in its sequence of query tiles; every warp role advances an identical copy.
struct FwCursor {
  int item, local, it, n_tiles;
  int kj, b, h;  // key tile, batch, head
  __device__ __forceinline__ bool valid() const { return item >= 0; }
  __device__ __forceinline__ int q_tile() const { return (kj >> 1) + it; }
};
struct FwPlace {  // where a query tile's dQ goes: first channel of the head, first row, batch
  int col, row, b;
};
// Items by decreasing walk length; rounds alternate direction, which evens out the CTAs' totals.
__device__ __forceinline__ void fw_load_item(FwCursor& c, int local, const FbParams& p) {
  const int nq = (p.T + FW_BM - 1) / FW_BM, nk = (p.T + FW_BN - 1) / FW_BN;
  const int heads = p.B * p.H, total = nk * heads;
  const int grid = (int)gridDim.x, cta = (int)blockIdx.x;
  const int item = local * grid + ((local & 1) ? grid - 1 - cta : cta);
  if (item >= total) { c.item = -1; return; }
  c.item = item;
  c.local = local;
  c.it = 0;
  c.kj = item / heads;
  const int bh = item % heads;
  c.b = bh / p.H;
  c.h = bh % p.H;
  c.n_tiles = nq - (c.kj >> 1);
}
__device__ __forceinline__ FwCursor fw_next(const FwCursor& c, const FbParams& p) {
  FwCursor n = c;
  if (c.it + 1 < c.n_tiles) { n.it = c.it + 1; return n; }
  fw_load_item(n, c.local + 1, p);
  return n;
}

__global__ void __launch_bounds__(FW_THREADS, 1)
flash_attention_bwd128_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                              const __grid_constant__ CUtensorMap map_dq, const __grid_constant__ CUtensorMap map_dk,
                              const __grid_constant__ CUtensorMap map_dv, const FbParams p) {
  extern __shared__ uint8_t fw_smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fw_smem_raw) + sizeof(FwBarriers) + 1023) & ~uintptr_t(1023));
  FwBarriers* bars = reinterpret_cast<FwBarriers*>(fw_smem_raw);
  const bool layout_ok = tiles + FW_DATA <= fw_smem_raw + FW_SMEM;
  uint8_t* sk = tiles;
  uint8_t* sv = sk + FW_KV_BYTES;
  uint8_t* sq = sv + FW_KV_BYTES;                    // [stage]
  uint8_t* sdo = sq + FW_STAGES * FW_Q_BYTES;        // [stage]
  uint8_t* sp = sdo + FW_STAGES * FW_Q_BYTES;
  uint8_t* sds = sp + FW_P_BYTES;
  uint8_t* staging = sds + FW_P_BYTES;
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tc05::mbar_init(&bars->kv_full, 1);
    tc05::mbar_init(&bars->kv_empty, 1);
    for (int s = 0; s < FW_STAGES; ++s) {
      tc05::mbar_init(&bars->q_full[s], 1);
      tc05::mbar_init(&bars->q_empty[s], 1);
    }
    tc05::mbar_init(&bars->sdp_full, 1);
    tc05::mbar_init(&bars->sdp_free, FW_SOFTMAX_WARPS);
    tc05::mbar_init(&bars->p_full, FW_SOFTMAX_WARPS);
    tc05::mbar_init(&bars->dq_full, 1);
    bars->abort_flag = layout_ok ? 0 : 1;
    tc05::fence_barrier_init();
  }
  if (warp == FW_SOFTMAX_WARPS + 1) {
    tc05::tmem_alloc(&bars->tmem_base, FW_TMEM_COLS);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  tc05::tc_fence_after_sync();
  const uint32_t tmem_s = bars->tmem_base;
  const uint32_t tmem_dp = tmem_s + 64;
  const uint32_t tmem_dv = tmem_s + 128;  // transposed: lanes are channels, columns keys
  const uint32_t tmem_dk = tmem_s + 192;
  const uint32_t tmem_dq = tmem_s + 256;  // two tiles of 128 columns, alternating
  pdl_begin();  // everything above touches nothing a predecessor wrote

  FwCursor first;
  fw_load_item(first, 0, p);

  if (warp == FW_SOFTMAX_WARPS) {
    // -------------------------------------------------------------------------- TMA producer
    if (tc05::elect_one() && !*abort_flag) {
      tc05::tma_prefetch_desc(&map_q);
      tc05::tma_prefetch_desc(&map_k);
      tc05::tma_prefetch_desc(&map_v);
      tc05::tma_prefetch_desc(&map_do);
      int g = 0;  // query tiles loaded so far
      for (FwCursor c = first; c.valid(); c = fw_next(c, p), ++g) {
        const int col = c.h * FW_HD;
        const int s = g % FW_STAGES;
        const int qrow = c.q_tile() * FW_BM;
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          tc05::tma_prefetch_l2_3d(&map_q, col + blk * 64, qrow, c.b);
          tc05::tma_prefetch_l2_3d(&map_do, col + blk * 64, qrow, c.b);
        }
        if (c.it == 0) {
          // one K/V buffer: free once the previous item's last products have been committed
          if (!tc05::mbar_wait(&bars->kv_empty, ((uint32_t)c.local & 1u) ^ 1u, abort_flag)) break;
          tc05::mbar_arrive_expect_tx(&bars->kv_full, 2 * FW_KV_BYTES);
#pragma unroll
          for (int blk = 0; blk < 2; ++blk) {
            tc05::tma_load_3d(sk + blk * FW_KV_BLOCK, &map_k, &bars->kv_full, col + blk * 64, c.kj * FW_BN, c.b);
            tc05::tma_load_3d(sv + blk * FW_KV_BLOCK, &map_v, &bars->kv_full, col + blk * 64, c.kj * FW_BN, c.b);
          }
        }
        if (!tc05::mbar_wait(&bars->q_empty[s], ((uint32_t)(g / FW_STAGES) & 1u) ^ 1u, abort_flag)) break;
        tc05::mbar_arrive_expect_tx(&bars->q_full[s], 2 * FW_Q_BYTES);
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          tc05::tma_load_3d(sq + s * FW_Q_BYTES + blk * FW_Q_BLOCK, &map_q, &bars->q_full[s], col + blk * 64, qrow, c.b);
          tc05::tma_load_3d(sdo + s * FW_Q_BYTES + blk * FW_Q_BLOCK, &map_do, &bars->q_full[s], col + blk * 64, qrow, c.b);
        }
      }
    }
  } else if (warp == FW_SOFTMAX_WARPS + 1) {
    // -------------------------------------------------------------------------- MMA issuer
    if (tc05::elect_one() && !*abort_flag) {
      constexpr uint32_t idesc_sdp = tc05::instr_desc_bf16_f32(128, FW_BN, false, false);
      constexpr uint32_t idesc_dkv = tc05::instr_desc_bf16_f32(128, FW_BN, true, true);    // channels x keys
      constexpr uint32_t idesc_dq = tc05::instr_desc_bf16_f32(128, FW_HD, false, true);
      const uint32_t ak = tc05::smem_u32(sk), av = tc05::smem_u32(sv);
      const uint64_t k_rows = tc05::smem_desc_sw128(ak, 16, 1024), v_rows = tc05::smem_desc_sw128(av, 16, 1024);
      const uint64_t k_chan = tc05::smem_desc_sw128(ak, FW_KV_BLOCK, 1024);  // K with its channels as columns: blocks 8 KB apart
      const uint32_t ap = tc05::smem_u32(sp), ads = tc05::smem_u32(sds);
      const uint64_t p_cols = tc05::smem_desc_sw128(ap, 16, 1024);           // P and dS as [query][key], keys as columns
      const uint64_t ds_cols = tc05::smem_desc_sw128(ads, 16, 1024);
      const uint64_t ds_rows = tc05::smem_desc_sw128(ads, 16, 1024);
      // S = Q·Kᵀ and dP = dO·Vᵀ of query tile number g
      auto issue_scores = [&](const FwCursor& c, int g) -> bool {
        if (c.it == 0 && !tc05::mbar_wait(&bars->kv_full, (uint32_t)c.local & 1u, abort_flag)) return false;
        const int s = g % FW_STAGES;
        if (!tc05::mbar_wait(&bars->q_full[s], (uint32_t)(g / FW_STAGES) & 1u, abort_flag)) return false;
        tc05::tc_fence_after_sync();
        const uint64_t q0 = tc05::smem_desc_sw128(tc05::smem_u32(sq + s * FW_Q_BYTES), 16, 1024);
        const uint64_t do0 = tc05::smem_desc_sw128(tc05::smem_u32(sdo + s * FW_Q_BYTES), 16, 1024);
#pragma unroll
        for (int ks = 0; ks < FW_HD / 16; ++ks)  // descriptors step by addition, in 16-byte units
          tc05::umma_ss(tmem_s, q0 + (uint64_t)((ks / 4) * (FW_Q_BLOCK >> 4) + (ks % 4) * 2),
                        k_rows + (uint64_t)((ks / 4) * (FW_KV_BLOCK >> 4) + (ks % 4) * 2), idesc_sdp, ks > 0 ? 1u : 0u);
#pragma unroll
        for (int ks = 0; ks < FW_HD / 16; ++ks)
          tc05::umma_ss(tmem_dp, do0 + (uint64_t)((ks / 4) * (FW_Q_BLOCK >> 4) + (ks % 4) * 2),
                        v_rows + (uint64_t)((ks / 4) * (FW_KV_BLOCK >> 4) + (ks % 4) * 2), idesc_sdp, ks > 0 ? 1u : 0u);
        tc05::umma_commit(&bars->sdp_full);
        return true;
      };
      FwCursor c = first;
      bool ok = c.valid() && issue_scores(c, 0);
      for (int g = 0; ok && c.valid(); ++g) {
        const FwCursor n = fw_next(c, p);
        // The next tile's scores follow as soon as this tile's have been read out; those of a new item only after this
        // item's products, since K and V have one buffer.
        const bool early = n.valid() && n.it > 0;
        if (early) {
          if (!tc05::mbar_wait(&bars->sdp_free, (uint32_t)g & 1u, abort_flag)) break;
          tc05::tc_fence_after_sync();
          if (!issue_scores(n, g + 1)) break;
        }
        if (!tc05::mbar_wait(&bars->p_full, (uint32_t)g & 1u, abort_flag)) break;
        tc05::tc_fence_after_sync();
        const int s = g % FW_STAGES;
        const uint64_t do_chan = tc05::smem_desc_sw128(tc05::smem_u32(sdo + s * FW_Q_BYTES), FW_Q_BLOCK, 1024);
        const uint64_t q_chan = tc05::smem_desc_sw128(tc05::smem_u32(sq + s * FW_Q_BYTES), FW_Q_BLOCK, 1024);
#pragma unroll
        for (int ks = 0; ks < FW_BM / 16; ++ks) {  // contraction over the tile's queries: 16 rows = 2048 bytes = 128 units
          const uint64_t step = (uint64_t)(ks * 128);
          const uint32_t acc = (c.it > 0 || ks > 0) ? 1u : 0u;  // a new item starts from zero
          tc05::umma_ss(tmem_dv, do_chan + step, p_cols + step, idesc_dkv, acc);
          tc05::umma_ss(tmem_dk, q_chan + step, ds_cols + step, idesc_dkv, acc);
        }
#pragma unroll
        for (int ks = 0; ks < FW_BN / 16; ++ks)  // dQ = dS·K over the tile's keys
          tc05::umma_ss(tmem_dq + (uint32_t)((g & 1) * FW_HD), ds_rows + (uint64_t)(ks * 2), k_chan + (uint64_t)(ks * 128), idesc_dq,
                        ks > 0 ? 1u : 0u);
        tc05::umma_commit(&bars->q_empty[s]);
        if (c.it == c.n_tiles - 1) tc05::umma_commit(&bars->kv_empty);
        tc05::umma_commit(&bars->dq_full);
        if (!early && n.valid()) {
          if (!tc05::mbar_wait(&bars->sdp_free, (uint32_t)g & 1u, abort_flag)) break;
          tc05::tc_fence_after_sync();
          if (!issue_scores(n, g + 1)) break;
        }
        c = n;
      }
    }
  } else {
    // -------------------------------------------------------------------------- softmax warps
    const int lg = warp & 3;          // tensor-memory lane group
    const int half = warp >> 2;       // which 32 key columns / 64 dQ columns / 32 keys of dVᵀ and dKᵀ
    const int r = lg * 32 + lane;     // row within the tile
    const uint32_t lane_sel = (uint32_t)(lg * 32) << 16;
    bool ok = !*abort_flag;
    uint8_t* my_stage = staging + warp * FW_STAGING;
    // Half of this warp's share of a dQ tile, 32 rows x 32 columns: out of tensor memory, into the staging rows (128 bytes,
    // 128-byte swizzle) and added by a TMA reduction.  The two halves of a tile are a softmax apart, so that the staging
    // rows have been read when the second one wants them.
    auto add_dq = [&](const FwPlace& at, int g, int part) {
      uint32_t qb[32];
      tc05::tmem_ld_32x32b_x32(tmem_dq + (uint32_t)((g & 1) * FW_HD) + lane_sel + half * 64 + part * 32, qb);
      if (lane == 0) tc05::tma_store_wait_read();
      tc05::tmem_ld_wait();
      tc05::tmem_ld_fence(qb);
      __syncwarp();
      uint8_t* line = my_stage + lane * 128;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<uint4*>(line + ((i ^ (lane & 7)) << 4)) = make_uint4(qb[i * 4], qb[i * 4 + 1], qb[i * 4 + 2], qb[i * 4 + 3]);
      tc05::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tc05::tma_reduce_add_3d(&map_dq, my_stage, at.col + half * 64 + part * 32, at.row + lg * 32, at.b);
        tc05::tma_store_commit();
      }
    };
    // dVᵀ and dKᵀ of an item: this thread's channel lg*32 + lane, 32 keys, as bf16 pairs (words 0-15 dV, 16-31 dK)
    auto load_dkv = [&](uint32_t (&w)[32]) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t raw[8];
        tc05::tmem_ld_32x32b_x8((q < 4 ? tmem_dv : tmem_dk) + lane_sel + half * 32 + (q & 3) * 8, raw);
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(raw);
#pragma unroll
        for (int i = 0; i < 8; i += 2) w[q * 4 + i / 2] = pack_bf16x2(__uint_as_float(raw[i]), __uint_as_float(raw[i + 1]));
      }
    };
    // Turned back through the staging rows: two tiles of 32 keys x 32 channels (64-byte rows, 64-byte swizzle), a warp's 32
    // channels side by side, and out with one TMA store each.  Keys past T are clipped by the tensor map.
    auto store_dkv = [&](const uint32_t (&w)[32], const FwCursor& c) {
      if (lane == 0) tc05::tma_store_wait_read();
      __syncwarp();
#pragma unroll
      for (int which = 0; which < 2; ++which)
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          const uint32_t word = w[which * 16 + k / 2];
          const uint16_t bits = (uint16_t)((k & 1) ? word >> 16 : word & 0xffffu);
          const int off = which * 2048 + k * 64 + ((((lane >> 3) ^ ((k >> 1) & 3)) << 4) | ((lane & 7) << 1));
          *reinterpret_cast<uint16_t*>(my_stage + off) = bits;
        }
      tc05::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        const int col = c.h * FW_HD + lg * 32, key0 = c.kj * FW_BN + half * 32;
        tc05::tma_store_3d(&map_dv, my_stage, col, key0, c.b);
        tc05::tma_store_3d(&map_dk, my_stage + 2048, col, key0, c.b);
        tc05::tma_store_commit();
      }
    };
    auto row_stats = [&](const FwCursor& c, float* lse_raw, float* dlt_raw) {
      const int tt = c.valid() ? c.q_tile() * FW_BM + r : 0;
      const bool in = c.valid() && tt < p.T;
      const size_t stat = in ? ((size_t)c.b * p.H + c.h) * p.T + tt : 0;
      *lse_raw = in ? __ldg(p.lse + stat) : INFINITY;  // rows past T: every P becomes 0
      *dlt_raw = in ? __ldg(p.delta + stat) : 0.f;
    };
    auto scale_stats = [&](float lse_raw, float dlt_raw, float* neg_lse2, float* neg_dlt_scaled) {
      *neg_lse2 = -lse_raw * 1.4426950408889634f;
      *neg_dlt_scaled = -dlt_raw * p.scale;
    };
    FwCursor c = first;
    FwPlace prev{}, prev2{};  // of the last two tiles
    float neg_lse2, neg_dlt_scaled;
    {
      float l0, d0;
      row_stats(c, &l0, &d0);
      scale_stats(l0, d0, &neg_lse2, &neg_dlt_scaled);
    }
    int g = 0, last_local = 0;
    auto tile = [&](auto boundary_tag, auto diag_tag) -> bool {
      constexpr bool Boundary = decltype(boundary_tag)::value;
      constexpr bool Diag = decltype(diag_tag)::value;
      const FwCursor n = fw_next(c, p);
      const int t = c.q_tile() * FW_BM + r;  // query position
      const int key0 = c.kj * FW_BN + half * 32;
      float next_lse_raw, next_dlt_raw;
      row_stats(n, &next_lse_raw, &next_dlt_raw);
      // the second half of the dQ tile before last: its buffer is written again only after this warp's next arrival on p_full
      if (g > 1) add_dq(prev2, g - 2, 1);
      if (!tc05::mbar_wait(&bars->sdp_full, (uint32_t)g & 1u, abort_flag)) return false;
      tc05::tc_fence_after_sync();
      uint32_t pp[4][4], dd[4][4];  // P and dS of this thread's 32 key columns, bf16 pairs
      uint32_t sb[2][8], db[2][8];  // eight columns at a time, the next eight on their way
      tc05::tmem_ld_32x32b_x8(tmem_s + lane_sel + half * 32, sb[0]);
      tc05::tmem_ld_32x32b_x8(tmem_dp + lane_sel + half * 32, db[0]);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(sb[ch & 1]);
        tc05::tmem_ld_fence(db[ch & 1]);
        if (ch < 3) {
          tc05::tmem_ld_32x32b_x8(tmem_s + lane_sel + half * 32 + ch * 8 + 8, sb[(ch + 1) & 1]);
          tc05::tmem_ld_32x32b_x8(tmem_dp + lane_sel + half * 32 + ch * 8 + 8, db[(ch + 1) & 1]);
        } else {  // all of S and dP is in registers: the next tile's may overwrite them
          tc05::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) tc05::mbar_arrive(&bars->sdp_free);
        }
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          float pr[2], dsv[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float pv = ex2_fast(fmaf(__uint_as_float(sb[ch & 1][i + e]), p.scale_log2, neg_lse2));
            if constexpr (Diag) pv = (key0 + ch * 8 + i + e > t) ? 0.f : pv;
            pr[e] = pv;
            dsv[e] = pv * fmaf(__uint_as_float(db[ch & 1][i + e]), p.scale, neg_dlt_scaled);
          }
          pp[ch][i / 2] = pack_bf16x2(pr[0], pr[1]);
          dd[ch][i / 2] = pack_bf16x2(dsv[0], dsv[1]);
        }
      }
      asm volatile("" : "+f"(next_lse_raw), "+f"(next_dlt_raw));  // first use of the loaded values: not before here
      scale_stats(next_lse_raw, next_dlt_raw, &neg_lse2, &neg_dlt_scaled);
      // the previous tile's products have finished: its dQ is ready and P/dS may be overwritten
      if (g > 0) {
        if (!tc05::mbar_wait(&bars->dq_full, (uint32_t)(g - 1) & 1u, abort_flag)) return false;
        tc05::tc_fence_after_sync();
      }
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        const int off = r * 128 + (((half * 4 + ch) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(sp + off) = make_uint4(pp[ch][0], pp[ch][1], pp[ch][2], pp[ch][3]);
        *reinterpret_cast<uint4*>(sds + off) = make_uint4(dd[ch][0], dd[ch][1], dd[ch][2], dd[ch][3]);
      }
      uint32_t dkv[Boundary ? 32 : 1];
      if constexpr (Boundary) load_dkv(dkv);  // before the new item's first products may overwrite them
      tc05::fence_proxy_async_smem();
      tc05::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&bars->p_full);
      if constexpr (Boundary) {
        FwCursor done;
        fw_load_item(done, c.local - 1, p);
        store_dkv(dkv, done);
      }
      if (g > 0) add_dq(prev, g - 1, 0);
      prev2 = prev;
      prev = FwPlace{c.h * FW_HD, c.q_tile() * FW_BM, c.b};
      last_local = c.local;
      c = n;
      ++g;
      return true;
    };
    while (ok && c.valid()) {
      if (c.it == 0) ok = g > 0 ? tile(std::true_type{}, std::true_type{}) : tile(std::false_type{}, std::true_type{});
      else ok = tile(std::false_type{}, std::false_type{});
    }
    if (ok && g > 0) {  // what is left of the last two dQ tiles, and dK, dV of the last item
      if (g > 1) add_dq(prev2, g - 2, 1);
      if (tc05::mbar_wait(&bars->dq_full, (uint32_t)(g - 1) & 1u, abort_flag)) {
        tc05::tc_fence_after_sync();
        add_dq(prev, g - 1, 0);
        add_dq(prev, g - 1, 1);
        uint32_t dkv[32];
        load_dkv(dkv);
        FwCursor done;
        fw_load_item(done, last_local, p);
        store_dkv(dkv, done);
        if (lane == 0) tc05::tma_store_wait_all();
      }
    }
  }

  tc05::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (threadIdx.x == 0) atomicExch(p.status + (layout_ok ? ST_WAIT_EXPIRED : ST_BAD_ARGUMENT), 1);
  }
  if (warp == FW_SOFTMAX_WARPS + 1) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc(tmem_s, FW_TMEM_COLS);
  }
}

}  // namespace

int launch_attention_bwd128(hl_ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                            const CUtensorMap& mdq, const CUtensorMap& mdk, const CUtensorMap& mdv, const FbParams& p) {
  HL_ALLOW_SHARED(ctx, FW_SMEM, flash_attention_bwd128_kernel);
  const int items = ceil_div(p.T, FW_BN) * p.B * p.H;
  pdl(flash_attention_bwd128_kernel, std::min(items, persistent_sms(ctx)), FW_THREADS, FW_SMEM, ctx->stream)(mq, mk, mv, mdo, mdq, mdk,
                                                                                                          mdv, p);
  return HL_OK;
}

}  // namespace hl
