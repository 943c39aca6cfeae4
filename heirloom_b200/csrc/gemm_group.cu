// The weight gradients of several layers in one launch: dW_i[n_out, n_in] = dY_iᵀ · X_i over the same tokens, and the bias
// gradients beside them (column sums of dY_i).
//
// One product of this kind has a few dozen 256 x 256 tiles and a long contraction.  By itself it had to share the contraction
// between CTAs to fill the chip, with partial sums through memory and a second kernel, and paid the start and the end of a launch
// for every product; a pass over dY for the column sums came on top.  The tiles of several layers together fill whole waves with
// undivided contractions (16384 tokens, d 768, d_ff 3072: 208 us a layer and 38 us of column sums before).
//
// CTA pairs as in gemm_tcgen05.cu: a 256 x 256 tile, six stages of 64 tokens, operands read down their rows (both MN-major).  One
// accumulator of 256 tensor-memory columns.  A second one would hide the two or three microseconds of a tile's epilogue behind 25 to
// 100 us of contraction.
//
// Column sums of dY: the epilogue warps, idle until the tile is done, add up the CTA's stages of dY as they pass, up to eight blocks
// of four tokens in f32 and the rest in f64 (additions of f64 alone cost 3 % of a step).  The tiles of a row of tiles share that
// work, each for every n_tiles-th block of 64 tokens; the quarters of a block are parts of their own.  A summed stage goes back to
// the producer when the warps have read it, which happens beside its products; they learn of it by a commit, since an arrival by
// the issuing thread held the products up.  As products with a block of ones the sums were up to forty times further off than column
// sums by themselves, because the tensor core cuts its f32 sums off at every step (16384 tokens: 1.7e-5 of the terms' magnitudes,
// those 4.2e-7, these 9e-8), and took longer (124M step 17.10 ms with them, 16.78 with these, 16.65 without any).
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
constexpr int GG_SUM_FLUSH = 8;                       // f32 additions of four values each before they go to f64
constexpr int GG_SUM_PARTS = GG_EPI_WARPS / 2;        // the epilogue warps: two blocks of 64 columns, four quarters of a stage's tokens
constexpr int GG_DATA = GG_STAGES * GG_STAGE_BYTES + GG_EPI_WARPS * GG_TILE_BYTES;
constexpr int GG_SMEM = GG_DATA + 256;
static_assert(GG_SMEM <= 227 * 1024, "shared memory budget");

struct GroupJob {
  CUtensorMap a, b, c;
  float* sums;            // [n_tiles * GG_SUM_PARTS][m] or null
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
  uint64_t sum_ready[GG_STAGES], sum_done[GG_STAGES];  // a stage whose dY is summed has been filled, has been read
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
  GroupShared* sh = reinterpret_cast<GroupShared*>(gg_smem + GG_DATA);
  volatile int* abort_flag = &sh->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = tc05::cluster_cta_rank();  // the even CTA leads
  if (threadIdx.x == 0) {
    for (int s = 0; s < GG_STAGES; ++s) {
      tc05::mbar_init(&sh->full[s], 1);
      tc05::mbar_init(&sh->empty[s], 1);
      tc05::mbar_init(&sh->sum_ready[s], 1);
      tc05::mbar_init(&sh->sum_done[s], GG_EPI_WARPS);
    }
    tc05::mbar_init(&sh->tmem_full, 1);
    tc05::mbar_init(&sh->tmem_empty, 2 * GG_EPI_WARPS);
    sh->abort_flag = (tc05::smem_u32(gg_smem) & 1023u) == 0 ? 0 : 1;
    tc05::fence_barrier_init();
  }
  if (warp == 1) {
    tc05::tmem_alloc_pair(&sh->tmem_base, GG_BN);
    tc05::tmem_relinquish_pair();
  }
  tc05::tc_fence_before_sync();
  tc05::cluster_sync_all();
  tc05::tc_fence_after_sync();
  const uint32_t tmem = sh->tmem_base;
  pdl_begin();  // everything above touches nothing a predecessor wrote

  GroupItem it{0, 0, 0};
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (tc05::elect_one()) {
      int stage = 0;
      uint32_t phase = 0, held = 0, done_phase = 0;  // a bit per stage: its sum warps have to be waited for; and with which parity
      bool ok = true;
      for (int local = 0; ok && group_item(p, local, it); ++local) {
        const GroupJob& job = p.job[it.job];
        int next_sum = job.sums != nullptr ? it.n_tile : p.k_blocks;
        tc05::tma_prefetch_desc(&job.a);
        tc05::tma_prefetch_desc(&job.b);
        const int m_row = it.m_tile * 2 * GG_BM + (int)rank * GG_BM;          // this CTA's 128 columns of dY
        const int n_row = it.n_tile * GG_BN + (int)rank * (GG_BN / 2);        // this CTA's 128 columns of X
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!tc05::mbar_wait(&sh->empty[stage], phase ^ 1u, abort_flag, p.wait_limit_ns)) { ok = false; break; }
          if (held >> stage & 1u) {
            if (!tc05::mbar_wait(&sh->sum_done[stage], done_phase >> stage & 1u, abort_flag, p.wait_limit_ns)) { ok = false; break; }
            done_phase ^= 1u << stage;
            held ^= 1u << stage;
          }
          if (kb == next_sum) {
            held |= 1u << stage;
            next_sum += job.n_tiles;
          }
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
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int local = 0; ok && group_item(p, local, it); ++local) {
        const GroupJob& job = p.job[it.job];
        if (!tc05::mbar_wait(&sh->tmem_empty, ((uint32_t)local & 1u) ^ 1u, abort_flag, p.wait_limit_ns)) break;
        tc05::tc_fence_after_sync();
        int next_sum = job.sums != nullptr ? it.n_tile : p.k_blocks;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!tc05::mbar_wait(&sh->full[stage], phase, abort_flag, p.wait_limit_ns)) { ok = false; break; }
          tc05::tc_fence_after_sync();
          const uint32_t sa = tc05::smem_u32(gg_smem + stage * GG_STAGE_BYTES);
          const uint32_t sb = sa + GG_A_BYTES;
          if (kb == next_sum) {
            tc05::umma_commit_pair_both(&sh->sum_ready[stage]);  // when the blocks before this one are done: soon enough, and no wait here
            next_sum += job.n_tiles;
          }
#pragma unroll
          for (int ks = 0; ks < GG_BK / 16; ++ks) {
            const uint64_t da = tc05::smem_desc_sw128(sa + ks * (16 * 128), GG_BK * 128, 1024);
            const uint64_t db = tc05::smem_desc_sw128(sb + ks * (16 * 128), GG_BK * 128, 1024);
            tc05::umma_ss_pair(tmem, da, db, idesc, (kb > 0 || ks > 0) ? 1u : 0u);
          }
          tc05::umma_commit_pair_both(&sh->empty[stage]);
          if (++stage == GG_STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) {
          tc05::umma_commit_pair_both(&sh->tmem_full);
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
    // Column sums: eight columns of a block of 64 (128-byte rows, a token each, 128-byte swizzle) a lane, every fourth of the 16
    // tokens that are the warp's share of a stage; tokens past the end are zeros.
    const int sum_block = ew & 1, sum_part = ew >> 1, sum_t0 = sum_part * 16 + (lane >> 3), sum_unit = lane & 7;
    uint32_t ready_phase = 0;  // a bit per stage
    bool ok = true;
    for (int local = 0; group_item(p, local, it); ++local) {
      const GroupJob& job = p.job[it.job];
      const int row0 = it.m_tile * 2 * GG_BM + (int)rank * GG_BM + lane_group * 32;
      if (job.sums != nullptr) {
        double sum[8];
        float2 few[4];  // of up to GG_SUM_FLUSH blocks
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          sum[2 * e] = sum[2 * e + 1] = 0.0;
          few[e] = both(0.f);
        }
        auto flush = [&]() {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            sum[2 * e] += (double)few[e].x;
            sum[2 * e + 1] += (double)few[e].y;
            few[e] = both(0.f);
          }
        };
        int blocks = 0;
        for (int kb = it.n_tile; kb < p.k_blocks; kb += job.n_tiles) {
          const int stage = (int)(((long long)local * p.k_blocks + kb) % GG_STAGES);
          ok = tc05::mbar_wait(&sh->sum_ready[stage], ready_phase >> stage & 1u, abort_flag, p.wait_limit_ns);
          if (!ok) break;
          ready_phase ^= 1u << stage;
          const uint8_t* block = gg_smem + stage * GG_STAGE_BYTES + sum_block * (GG_BK * 128);
          uint4 v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int t = sum_t0 + u * 4;
            v[u] = *reinterpret_cast<const uint4*>(block + t * 128 + ((sum_unit ^ (t & 7)) << 4));
          }
          auto four = [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
            return add2(add2(unpack_bf16x2(a), unpack_bf16x2(b)), add2(unpack_bf16x2(c), unpack_bf16x2(d)));
          };
          few[0] = add2(few[0], four(v[0].x, v[1].x, v[2].x, v[3].x));
          few[1] = add2(few[1], four(v[0].y, v[1].y, v[2].y, v[3].y));
          few[2] = add2(few[2], four(v[0].z, v[1].z, v[2].z, v[3].z));
          few[3] = add2(few[3], four(v[0].w, v[1].w, v[2].w, v[3].w));
          if (++blocks % GG_SUM_FLUSH == 0) flush();
          __syncwarp();
          if (lane == 0) tc05::mbar_arrive(&sh->sum_done[stage]);
        }
        if (!ok) break;
        flush();
        float out[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 8);
          sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 16);
          out[e] = (float)sum[e];
        }
        const int c = it.m_tile * 2 * GG_BM + (int)rank * GG_BM + sum_block * 64 + sum_unit * 8;  // m is a multiple of 8
        if (lane < 8 && c < job.m) {
          float* at = job.sums + (size_t)(it.n_tile * GG_SUM_PARTS + sum_part) * job.m + c;
          *reinterpret_cast<float4*>(at) = make_float4(out[0], out[1], out[2], out[3]);
          *reinterpret_cast<float4*>(at + 4) = make_float4(out[4], out[5], out[6], out[7]);
        }
      }
      if (!tc05::mbar_wait(&sh->tmem_full, (uint32_t)local & 1u, abort_flag, p.wait_limit_ns)) break;
      tc05::tc_fence_after_sync();
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
          if (lane == 0) tc05::mbar_arrive_cluster_read(tc05::cluster_map_shared(&sh->tmem_empty, 0));
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
    tc05::tmem_dealloc_pair(tmem, GG_BN);
  }
}

}  // namespace

int gemm_group_tiles(int n_out, int n_in) { return ceil_div(n_out, 2 * GG_BM) * ceil_div(n_in, GG_BN); }
size_t gemm_group_sums(int n_out, int n_in) { return ((size_t)ceil_div(n_in, GG_BN) * GG_SUM_PARTS * n_out + 63) & ~size_t(63); }

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
  HL_ALLOW_SHARED(ctx, GG_SMEM, gemm_group_kernel);
  static PerDevice pairs;  // a GPC with an odd number of SMs leaves one out
  const int resident_pairs = pairs.value(ctx->device, [&] { return resident_clusters(gemm_group_kernel, 2, GG_THREADS, GG_SMEM); });
  HL_REQUIRE(resident_pairs > 0, "gemm_group: no CTA pair fits on this device");
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
    fold_batch_add(fold, p.job[i].sums, p.job[i].n_tiles * GG_SUM_PARTS, jobs[i].n_out, jobs[i].n_out, jobs[i].db, nullptr, nullptr);
    any = true;
  }
  return any ? fold_batch_flush(ctx, fold) : HL_OK;  // the next group writes its shares to the same place
}

}  // namespace hl
