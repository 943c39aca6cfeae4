// The weight gradients of several layers in one launch: dW_i[n_out, n_in] = dY_iᵀ · X_i over the same tokens, and the bias
// gradients beside them (column sums of dY_i).
//
// One product of this kind has a few dozen 256 x 256 tiles and a long contraction.  By itself it had to share the contraction
// between CTAs to fill the chip, with partial sums through memory and a second kernel, and paid the start and the end of a launch
// for every product; a pass over dY for the column sums came on top.  The tiles of several layers together fill whole waves with
// undivided contractions (16384 tokens, d 768, d_ff 3072: 208 us a layer and 38 us of column sums before).
//
// CTA pairs as in gemm_tcgen05.cu: a 256 x 256 tile, six stages of 64 tokens, operands read down their rows (both MN-major).  One
// accumulator of 256 tensor-memory columns; the other 256 take column sums of dY, as a product with a block of ones, 32 columns
// wide.  The tiles of a row of tiles share that work, each for every n_tiles-th block of tokens, and spread it over eight blocks of
// columns, so that no f32 sum runs over more than a fraction of the tokens; the fractions are added in f64.  A second
// accumulator would hide the two or three microseconds of a tile's epilogue behind 25 to 100 us of contraction; the sums save more.
#include "kernels.h"
#include "tc05.cuh"

namespace hl {
namespace {

constexpr int GG_BM = 128, GG_BN = 256, GG_BK = 64;   // rows of a CTA (the pair has 256), columns of the tile, tokens a stage
constexpr int GG_STAGES = 6;
constexpr int GG_A_BYTES = GG_BM * GG_BK * 2;
constexpr int GG_STAGE_BYTES = 2 * GG_A_BYTES;        // and half of B's columns
constexpr int GG_EPI_WARPS = 8;
constexpr int GG_TILE_BYTES = 4096;                   // an epilogue warp's staging tile: 32 rows x 32 f32
constexpr int GG_THREADS = (2 + GG_EPI_WARPS) * 32;
constexpr int GG_ONES = 2048;                         // 16 columns x 64 tokens of 1.0 (a pair has 32)
constexpr int GG_SUM_BLOCKS = 8, GG_SUM_COLS = 32;
constexpr int GG_DATA = GG_STAGES * GG_STAGE_BYTES + GG_EPI_WARPS * GG_TILE_BYTES + GG_ONES;
constexpr int GG_SMEM = GG_DATA + 256;
static_assert(GG_SMEM <= 227 * 1024, "shared memory budget");

struct GroupJob {
  CUtensorMap a, b, c;
  float* sums;            // [n_tiles][m] or null
  int m, n_tiles, tile0;  // tile0: tiles of the jobs before
};
struct GroupParams {
  GroupJob job[kMaxGroupJobs];
  int jobs, tiles, k_blocks;
  unsigned long long wait_limit_ns;
  int* status;
};
static_assert(sizeof(GroupParams) <= 32 * 1024 - 4, "kernel parameters");

struct GroupShared {
  uint64_t full[GG_STAGES], empty[GG_STAGES];
  uint64_t tmem_full, tmem_empty;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(GroupShared) <= 256, "barriers outgrow their place");

// The `local`-th tile of this pair: job, row and column of tiles; every warp role walks the same sequence.
struct GroupItem {
  int job, m_tile, n_tile;
};
__device__ __forceinline__ bool group_item(const GroupParams& p, int local, GroupItem& it) {
  const int tile = (int)(blockIdx.x >> 1) + local * (int)(gridDim.x >> 1);
  if (tile >= p.tiles) return false;
  int j = it.job;  // items ascend
  while (j + 1 < p.jobs && p.job[j + 1].tile0 <= tile) ++j;
  const int t = tile - p.job[j].tile0;
  it.job = j;
  it.m_tile = t / p.job[j].n_tiles;
  it.n_tile = t - it.m_tile * p.job[j].n_tiles;
  return true;
}

__global__ void __launch_bounds__(GG_THREADS, 1)
gemm_group_kernel(const __grid_constant__ GroupParams p) {
  extern __shared__ __align__(1024) uint8_t gg_smem[];  // swizzled tiles want 1024 bytes; checked below
  uint8_t* staging_base = gg_smem + GG_STAGES * GG_STAGE_BYTES;
  uint8_t* ones = staging_base + GG_EPI_WARPS * GG_TILE_BYTES;
  GroupShared* sh = reinterpret_cast<GroupShared*>(gg_smem + GG_DATA);
  volatile int* abort_flag = &sh->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = tc05::cluster_cta_rank();  // the even CTA leads
  if (threadIdx.x == 0) {
    for (int s = 0; s < GG_STAGES; ++s) {
      tc05::mbar_init(&sh->full[s], 1);
      tc05::mbar_init(&sh->empty[s], 1);
    }
    tc05::mbar_init(&sh->tmem_full, 1);
    tc05::mbar_init(&sh->tmem_empty, 2 * GG_EPI_WARPS);
    sh->abort_flag = (tc05::smem_u32(gg_smem) & 1023u) == 0 ? 0 : 1;
    tc05::fence_barrier_init();
  }
  for (int i = threadIdx.x; i < GG_ONES / 4; i += GG_THREADS) reinterpret_cast<uint32_t*>(ones)[i] = 0x3f803f80u;
  tc05::fence_proxy_async_smem();
  if (warp == 1) {
    tc05::tmem_alloc_pair(&sh->tmem_base, 512);
    tc05::tmem_relinquish_pair();
  }
  tc05::tc_fence_before_sync();
  tc05::cluster_sync_all();
  tc05::tc_fence_after_sync();
  const uint32_t tmem = sh->tmem_base;
  const uint32_t tmem_sums = tmem + GG_BN;
  pdl_begin();  // everything above touches nothing a predecessor wrote

  GroupItem it{0, 0, 0};
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (tc05::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int local = 0; ok && group_item(p, local, it); ++local) {
        const GroupJob& job = p.job[it.job];
        tc05::tma_prefetch_desc(&job.a);
        tc05::tma_prefetch_desc(&job.b);
        const int m_row = it.m_tile * 2 * GG_BM + (int)rank * GG_BM;          // this CTA's 128 columns of dY
        const int n_row = it.n_tile * GG_BN + (int)rank * (GG_BN / 2);        // this CTA's 128 columns of X
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!tc05::mbar_wait(&sh->empty[stage], phase ^ 1u, abort_flag, p.wait_limit_ns)) { ok = false; break; }
          uint8_t* sa = gg_smem + stage * GG_STAGE_BYTES;
          uint8_t* sb = sa + GG_A_BYTES;
          // both CTAs' bytes are counted on the leader's barrier; only the leader announces them
          const uint32_t bar = tc05::cluster_map_shared(&sh->full[stage], 0);
          if (rank == 0) tc05::mbar_arrive_expect_tx(&sh->full[stage], 2 * GG_STAGE_BYTES);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            tc05::tma_load_2d_pair(sa + j * (GG_BK * 128), &job.a, bar, m_row + j * 64, kb * GG_BK);
            tc05::tma_load_2d_pair(sb + j * (GG_BK * 128), &job.b, bar, n_row + j * 64, kb * GG_BK);
          }
          if (++stage == GG_STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (rank == 0 && tc05::elect_one()) {
      constexpr uint32_t idesc = tc05::instr_desc_bf16_f32(2 * GG_BM, GG_BN, true, true);
      constexpr uint32_t idesc_sums = tc05::instr_desc_bf16_f32(2 * GG_BM, GG_SUM_COLS, true, false);
      const uint64_t ones_desc = tc05::smem_desc_sw128(tc05::smem_u32(ones), 16, 1024);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int local = 0; ok && group_item(p, local, it); ++local) {
        const GroupJob& job = p.job[it.job];
        const int n_tiles = job.n_tiles;
        const bool sums = job.sums != nullptr;
        const int share = sums ? (p.k_blocks - it.n_tile + n_tiles - 1) / n_tiles : 0;  // token blocks this tile sums up
        const int per_block = max(1, (share + GG_SUM_BLOCKS - 1) / GG_SUM_BLOCKS);
        if (!tc05::mbar_wait(&sh->tmem_empty, ((uint32_t)local & 1u) ^ 1u, abort_flag, p.wait_limit_ns)) break;
        tc05::tc_fence_after_sync();
        int next_sum = it.n_tile, summed = 0;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!tc05::mbar_wait(&sh->full[stage], phase, abort_flag, p.wait_limit_ns)) { ok = false; break; }
          tc05::tc_fence_after_sync();
          const uint32_t sa = tc05::smem_u32(gg_smem + stage * GG_STAGE_BYTES);
          const uint32_t sb = sa + GG_A_BYTES;
          const bool sum_now = sums && kb == next_sum;
          const uint32_t sum_col = tmem_sums + (uint32_t)(summed / per_block * GG_SUM_COLS);
          const bool sum_first = summed % per_block == 0;
#pragma unroll
          for (int ks = 0; ks < GG_BK / 16; ++ks) {
            const uint64_t da = tc05::smem_desc_sw128(sa + ks * (16 * 128), GG_BK * 128, 1024);
            const uint64_t db = tc05::smem_desc_sw128(sb + ks * (16 * 128), GG_BK * 128, 1024);
            tc05::umma_ss_pair(tmem, da, db, idesc, (kb > 0 || ks > 0) ? 1u : 0u);
            if (sum_now) tc05::umma_ss_pair(sum_col, da, ones_desc, idesc_sums, (!sum_first || ks > 0) ? 1u : 0u);
          }
          if (sum_now) { next_sum += n_tiles; ++summed; }
          tc05::umma_commit_pair(tc05::cluster_map_shared(&sh->empty[stage], 0));
          tc05::umma_commit_pair(tc05::cluster_map_shared(&sh->empty[stage], 1));
          if (++stage == GG_STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) {
          tc05::umma_commit_pair(tc05::cluster_map_shared(&sh->tmem_full, 0));
          tc05::umma_commit_pair(tc05::cluster_map_shared(&sh->tmem_full, 1));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int ew = warp - 2;
    const int lane_group = warp & 3;  // tensor-memory lanes this warp may read
    const int half = ew >> 2;         // which 128 of the tile's 256 columns
    const uint32_t lane_sel = (uint32_t)(lane_group * 32) << 16;
    uint8_t* staging = staging_base + ew * GG_TILE_BYTES;
    for (int local = 0; group_item(p, local, it); ++local) {
      const GroupJob& job = p.job[it.job];
      const int row0 = it.m_tile * 2 * GG_BM + (int)rank * GG_BM + lane_group * 32, row = row0 + lane;
      if (!tc05::mbar_wait(&sh->tmem_full, (uint32_t)local & 1u, abort_flag, p.wait_limit_ns)) break;
      tc05::tc_fence_after_sync();
      double sum = 0.0;
      if (half == 0 && job.sums != nullptr) {
        const int share = (p.k_blocks - it.n_tile + job.n_tiles - 1) / job.n_tiles;
        const int per_block = max(1, (share + GG_SUM_BLOCKS - 1) / GG_SUM_BLOCKS);
        for (int b = 0; b * per_block < share; ++b) {
          uint32_t s[8];  // the block's columns are all the same
          tc05::tmem_ld_32x32b_x8(tmem_sums + lane_sel + b * GG_SUM_COLS, s);
          tc05::tmem_ld_wait();
          tc05::tmem_ld_fence(s);
          sum += (double)__uint_as_float(s[0]);
        }
      }
      uint32_t acc[2][32];
      tc05::tmem_ld_32x32b_x32(tmem + lane_sel + half * 128, acc[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(acc[c & 1]);
        if (c < 3) {
          tc05::tmem_ld_32x32b_x32(tmem + lane_sel + half * 128 + (c + 1) * 32, acc[(c + 1) & 1]);
        } else {  // all of it is in registers: the next tile may overwrite it
          tc05::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) tc05::mbar_arrive_cluster(tc05::cluster_map_shared(&sh->tmem_empty, 0));
        }
        if (lane == 0) tc05::tma_store_wait_read();
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(staging + lane * 128 + ((q ^ (lane & 7)) << 4)) =
              make_uint4(acc[c & 1][q * 4], acc[c & 1][q * 4 + 1], acc[c & 1][q * 4 + 2], acc[c & 1][q * 4 + 3]);
        tc05::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {  // columns and rows past the edge are clipped
          tc05::tma_store_2d(&job.c, staging, it.n_tile * GG_BN + half * 128 + c * 32, row0);
          tc05::tma_store_commit();
        }
      }
      if (half == 0 && job.sums != nullptr && row < job.m) job.sums[(size_t)it.n_tile * job.m + row] = (float)sum;
    }
    if (lane == 0) tc05::tma_store_wait_all();
  }

  tc05::tc_fence_before_sync();
  // neither CTA leaves while the other still reads its shared memory or arrives on its barriers; every loop above is bounded
  tc05::cluster_sync_all();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);  // copies in flight land first
    if (threadIdx.x == 0) atomicExch(p.status + ST_WAIT_EXPIRED, 1);
  }
  if (warp == 1) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc_pair(tmem, 512);
  }
}

}  // namespace

int gemm_group_tiles(int n_out, int n_in) { return ceil_div(n_out, 2 * GG_BM) * ceil_div(n_in, GG_BN); }
size_t gemm_group_sums(int n_out, int n_in) { return ((size_t)ceil_div(n_in, GG_BN) * n_out + 63) & ~size_t(63); }

int gemm_group_run(hl_ctx* ctx, const WeightGradJob* jobs, int count, int tokens, float* sums, FoldBatch* fold) {
  if (count == 0) return HL_OK;
  HL_REQUIRE(count <= kMaxGroupJobs && tokens > 0, "gemm_group: too many products");
  GroupParams p{};
  double flops = 0.0;
  for (int i = 0; i < count; ++i) {
    const WeightGradJob& j = jobs[i];
    HL_REQUIRE(j.n_out % 8 == 0 && j.n_in % 8 == 0, "gemm_group: sizes must be multiples of 8");
    GroupJob& g = p.job[i];
    int rc = make_tensor_map_bf16_2d(&g.a, j.dy, (uint64_t)j.n_out, (uint64_t)tokens, (uint64_t)j.n_out, 64, GG_BK);
    if (rc != HL_OK) return rc;
    rc = make_tensor_map_bf16_2d(&g.b, j.x, (uint64_t)j.n_in, (uint64_t)tokens, (uint64_t)j.n_in, 64, GG_BK);
    if (rc != HL_OK) return rc;
    const uint64_t dims[2] = {(uint64_t)j.n_in, (uint64_t)j.n_out};
    const uint64_t strides[1] = {(uint64_t)j.n_in * 4};
    const uint32_t box[2] = {32, 32};
    rc = make_tensor_map(&g.c, HL_F32, 2, j.dw, dims, strides, box, 128);
    if (rc != HL_OK) return rc;
    g.m = j.n_out;
    g.n_tiles = ceil_div(j.n_in, GG_BN);
    g.tile0 = p.tiles;
    p.tiles += gemm_group_tiles(j.n_out, j.n_in);
    if (j.db) {
      g.sums = sums;
      sums += gemm_group_sums(j.n_out, j.n_in);
    }
    flops += 2.0 * j.n_out * j.n_in * (double)tokens;
  }
  p.jobs = count;
  p.k_blocks = ceil_div(tokens, GG_BK);
  p.wait_limit_ns = ctx->wait_limit_ns ? ctx->wait_limit_ns : tc05::kWaitLimitNs;
  p.status = ctx->status_dev;
  static int resident_pairs = 0;  // a GPC with an odd number of SMs leaves one out
  if (resident_pairs == 0) {
    HL_CUDA(cudaFuncSetAttribute(gemm_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GG_SMEM));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(ctx->sm_count & ~1));
    cfg.blockDim = dim3(GG_THREADS);
    cfg.dynamicSmemBytes = GG_SMEM;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    HL_CUDA(cudaOccupancyMaxActiveClusters(&n, gemm_group_kernel, &cfg));
    HL_REQUIRE(n > 0, "gemm_group: no CTA pair fits on this device");
    resident_pairs = n;
  }
  {
    ProfileScope prof(ctx, HL_PROF_GEMM, flops);
    HL_CUDA(launch_pdl(gemm_group_kernel, (unsigned)(2 * std::min({p.tiles, resident_pairs, std::max(1, persistent_sms(ctx) / 2)})), GG_THREADS, GG_SMEM, ctx->stream, 2, p));
  }
  count_launch(ctx);
  ctx->counters.gemm_tcgen05_launches += 1;
  ctx->counters.gemm_pair_launches += 1;
  // the shares of every bias gradient, one launch for up to sixteen
  bool any = false;
  for (int i = 0; i < count; ++i) {
    if (!jobs[i].db) continue;
    if (fold->n == FoldBatch::kMaxJobs) {
      int rc = fold_batch_flush(ctx, fold);
      if (rc != HL_OK) return rc;
    }
    fold_batch_add(fold, p.job[i].sums, p.job[i].n_tiles, jobs[i].n_out, jobs[i].n_out, jobs[i].db, nullptr, nullptr);
    any = true;
  }
  return any ? fold_batch_flush(ctx, fold) : HL_OK;  // the next group writes its shares to the same place
}

}  // namespace hl
