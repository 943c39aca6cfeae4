// The bf16 GEMM for products that leave most of the chip idle when they are cut into the persistent kernel's 128 x 256
// tiles (gemm_tcgen05.cu): few tokens, narrow layers, weight gradients of small models.  Same operands, rounding points and
// epilogues.
//
// What bounds these products is latency: the few k blocks of a tile, the epilogue after them, and the launch.  So one CTA
// per 128 x 64 or 128 x 128 tile, not persistent; its barriers, tensor memory and descriptors are set up while
// the previous kernel of the stream still runs (programmatic dependent launch); and a contraction is shared by the CTAs of
// a cluster, whose partial sums are added in rank order out of each other's shared memory, each CTA finishing a part of
// the tile's rows.  There is no second kernel for the sums and every epilogue works on shared contractions too.
// The accumulator goes through shared memory once, so that the epilogue reads the residual and writes the result in whole
// row segments.
#include <cooperative_groups.h>

#include "kernels.h"
#include "tc05.cuh"

namespace hl {
namespace {

namespace cg = cooperative_groups;

constexpr int GS_BM = 128, GS_BK = 64;
constexpr int GS_THREADS = 256;
constexpr int GS_A_BYTES = GS_BM * GS_BK * 2;
constexpr int GS_MAX_STAGES = 8;

template <int BN, int STAGES>
struct GsSizes {
  static constexpr int STAGE_BYTES = GS_A_BYTES + BN * GS_BK * 2;   // 24 / 32 KB
  static constexpr int DATA = STAGES * STAGE_BYTES;
  static constexpr int LD = BN + 4;                                 // accumulator rows in shared memory: conflict-free writes
  static constexpr int SUMS = GS_BM * LD * 4;                       // behind it the row sums of the two halves of every k block
  static constexpr int ACC_BYTES = SUMS + 2 * GS_BM * 8;
  static_assert(ACC_BYTES <= DATA && ACC_BYTES % 16 == 0, "the accumulator reuses the stages");
  static constexpr int TAIL = DATA;                                 // barriers
  // The residual or pre-activation rows of the tile: a place of their own where one CTA has the SM, else in the stages, behind the
  // accumulator.
  static constexpr int CTAS_PER_SM = DATA <= 104 * 1024 ? 2 : 1;
  static constexpr int AUX = CTAS_PER_SM == 1 ? TAIL + 256 : ACC_BYTES;
  static constexpr int AUX_BYTES = GS_BM * BN * 2;
  static constexpr int SMEM = CTAS_PER_SM == 1 ? AUX + AUX_BYTES : TAIL + 256;  // base aligned to 1024 bytes, as the kernel checks
  static_assert(CTAS_PER_SM == 1 || AUX + AUX_BYTES <= DATA, "the rows fit behind the accumulator");
  static_assert(CTAS_PER_SM * (SMEM + 1024) <= 228 * 1024, "shared memory budget");
};

struct GsParams {
  int m, n, k_blocks, k_blocks_per_rank;
  int m_tiles, splits;
  int epilogue;
  bool out_bf16;
  int a_kb_wrap, b_kb_wrap;  // > 0: the operand holds this many k blocks and is read again from its start after them
  unsigned long long wait_limit_ns;
  const float* bias;
  const __nv_bfloat16* aux_in;
  long long ld_aux_in;
  void* c;
  long long ldc;
  __nv_bfloat16* aux_out;
  long long ld_aux_out;
  float* row_sum;  // [m] or null: sum over the contraction of A's rows (A MN-major)
  int* status;
};

struct GsTail {
  uint64_t full[GS_MAX_STAGES], empty[GS_MAX_STAGES], done;
  uint32_t tmem_base;
  int abort_flag;
};

template <bool A_MN, bool B_MN, int BN, int STAGES>
__global__ void __launch_bounds__(GS_THREADS, (GsSizes<BN, STAGES>::CTAS_PER_SM))
gemm_small_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GsParams p) {
  using Z = GsSizes<BN, STAGES>;
  extern __shared__ __align__(1024) uint8_t smem[];
  GsTail* tail = reinterpret_cast<GsTail*>(smem + Z::TAIL);
  volatile int* abort_flag = &tail->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)blockIdx.x % p.splits, tile = (int)blockIdx.x / p.splits;
  const int m0 = (tile % p.m_tiles) * GS_BM, n0 = (tile / p.m_tiles) * BN;
  const int kb0 = rank * p.k_blocks_per_rank, kb1 = min(p.k_blocks, kb0 + p.k_blocks_per_rank);

  // Row sums (a bias gradient beside its weight gradient): in the tiles of the first column four warps that have nothing to do
  // until the epilogue add up A's stages as they pass, four values in f32, the rest in f64, which is no further off than column sums by
  // themselves: 16384 tokens 5.8e-8 of the terms' magnitudes at most, those 4.2e-7, and 1.7e-5 when they were a product with a block
  // of ones, whose f32 sums the tensor core cuts off at every step.  (256-token model's step 186 -> 179 us without those products.)
  const bool sums = A_MN && p.row_sum != nullptr && n0 == 0;
  constexpr int SUM_WARP0 = 4, SUM_WARPS = 4;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc05::mbar_init(&tail->full[s], 1);
      tc05::mbar_init(&tail->empty[s], sums ? 1 + SUM_WARPS : 1);
    }
    tc05::mbar_init(&tail->done, 1);
    tail->abort_flag = (tc05::smem_u32(smem) & 1023u) == 0 ? 0 : 1;
    tc05::fence_barrier_init();
    tc05::tma_prefetch_desc(&map_a);
    tc05::tma_prefetch_desc(&map_b);
  }
  if (warp == 1) {
    tc05::tmem_alloc(&tail->tmem_base, BN);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  tc05::tc_fence_after_sync();
  const uint32_t tmem = tail->tmem_base;
  pdl_trigger();
  pdl_wait();

  // This thread's four columns, and the rows it finishes of this CTA's share of the tile.
  constexpr int QUADS = BN / 4, ROWS_PER_PASS = GS_THREADS / QUADS;
  const int rows_mine = GS_BM / p.splits, row_first = rank * rows_mine;
  const int quad = threadIdx.x % QUADS, sub = threadIdx.x / QUADS;
  const int col = n0 + quad * 4;
  const bool col_ok = col < p.n;  // n is a multiple of 8
  const bool need_aux = p.epilogue == HL_EPI_BIAS_RESIDUAL || p.epilogue == HL_EPI_DGELU;
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.bias && col_ok) bias = __ldg(reinterpret_cast<const float4*>(p.bias + col));
  // All of them are requested at once, beside the contraction or right behind it: row by row in the loop below, a load's latency
  // per eight rows, they took 8 of 23 us (4096 x 512 x 2048 with residual).
  auto fetch_aux = [&]() {
    for (int i = threadIdx.x; i < rows_mine * (BN / 8); i += GS_THREADS) {
      const int r = i / (BN / 8), u = i % (BN / 8), row = m0 + row_first + r, c = n0 + u * 8;
      if (row < p.m && c < p.n)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc05::smem_u32(smem + Z::AUX + i * 16)),
                     "l"(p.aux_in + (size_t)row * p.ld_aux_in + c) : "memory");
    }
  };
  if (need_aux && Z::CTAS_PER_SM == 1) fetch_aux();

  if (warp == 0) {
    if (tc05::elect_one()) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, stage = i % STAGES;
        if (!tc05::mbar_wait(&tail->empty[stage], ((uint32_t)(i / STAGES) & 1u) ^ 1u, abort_flag, p.wait_limit_ns)) break;
        uint8_t* sa = smem + stage * Z::STAGE_BYTES;
        uint8_t* sb = sa + GS_A_BYTES;
        const int ka = p.a_kb_wrap > 0 ? kb % p.a_kb_wrap : kb, kbb = p.b_kb_wrap > 0 ? kb % p.b_kb_wrap : kb;
        tc05::mbar_arrive_expect_tx(&tail->full[stage], Z::STAGE_BYTES);
        if (A_MN) {
#pragma unroll
          for (int j = 0; j < GS_BM / 64; ++j)
            tc05::tma_load_2d(sa + j * (GS_BK * 128), &map_a, &tail->full[stage], m0 + j * 64, ka * GS_BK);
        } else {
          tc05::tma_load_2d(sa, &map_a, &tail->full[stage], ka * GS_BK, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            tc05::tma_load_2d(sb + j * (GS_BK * 128), &map_b, &tail->full[stage], n0 + j * 64, kbb * GS_BK);
        } else {
          tc05::tma_load_2d(sb, &map_b, &tail->full[stage], kbb * GS_BK, n0);
        }
      }
    }
  } else if (warp == 1) {
    if (tc05::elect_one()) {
      constexpr uint32_t idesc = tc05::instr_desc_bf16_f32(GS_BM, BN, A_MN, B_MN);
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, stage = i % STAGES;
        if (!tc05::mbar_wait(&tail->full[stage], (uint32_t)(i / STAGES) & 1u, abort_flag, p.wait_limit_ns)) { ok = false; break; }
        tc05::tc_fence_after_sync();
        const uint32_t sa = tc05::smem_u32(smem + stage * Z::STAGE_BYTES), sb = sa + GS_A_BYTES;
#pragma unroll
        for (int ks = 0; ks < GS_BK / 16; ++ks) {
          const uint64_t da = A_MN ? tc05::smem_desc_sw128(sa + ks * (16 * 128), GS_BK * 128, 1024)
                                   : tc05::smem_desc_sw128(sa + ks * 32, 16, 1024);
          const uint64_t db = B_MN ? tc05::smem_desc_sw128(sb + ks * (16 * 128), GS_BK * 128, 1024)
                                   : tc05::smem_desc_sw128(sb + ks * 32, 16, 1024);
          tc05::umma_ss(tmem, da, db, idesc, (i > 0 || ks > 0) ? 1u : 0u);
        }
        tc05::umma_commit(&tail->empty[stage]);
      }
      if (ok) tc05::umma_commit(&tail->done);
    }
  }
  // This lane's two rows of A (columns in memory: a stage holds two blocks of 64, token by token, 128-byte swizzle), over 32 of a
  // stage's 64 tokens; tokens past the end are zeros.
  double row_sum[2] = {0.0, 0.0};
  const int sum_block = warp & 1, sum_half = (warp >> 1) & 1;
  if (sums && warp >= SUM_WARP0) {
    for (int kb = kb0; kb < kb1; ++kb) {
      const int i = kb - kb0, stage = i % STAGES;
      if (!tc05::mbar_wait(&tail->full[stage], (uint32_t)(i / STAGES) & 1u, abort_flag, p.wait_limit_ns)) break;
      const uint8_t* block = smem + stage * Z::STAGE_BYTES + sum_block * (GS_BK * 128);
#pragma unroll 4
      for (int t = sum_half * 32; t < sum_half * 32 + 32; t += 4) {
        float2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          v[u] = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(block + (t + u) * 128 + (((lane >> 2) ^ ((t + u) & 7)) << 4) + (lane & 3) * 4));
        const float2 four = add2(add2(v[0], v[1]), add2(v[2], v[3]));
        row_sum[0] += (double)four.x;
        row_sum[1] += (double)four.y;
      }
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(&tail->empty[stage]);
    }
  }

  // ---- epilogue: all eight warps
  const bool have = kb0 < kb1;
  bool ok = true;
  if (have) ok = tc05::mbar_wait(&tail->done, 0, abort_flag, p.wait_limit_ns);
  __syncthreads();  // every role has left its loop: nothing reads or writes the stages any more
  tc05::tc_fence_after_sync();
  if (need_aux && Z::CTAS_PER_SM == 2) fetch_aux();
  float* acc = reinterpret_cast<float*>(smem);
  {
    const int lg = warp & 3, half = warp >> 2, r = lg * 32 + lane;
#pragma unroll
    for (int c = 0; c < BN / 2; c += 32) {
      uint32_t bits[32];
      const int c0 = half * (BN / 2) + c;
      if (have) {
        tc05::tmem_ld_32x32b_x32(tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)c0, bits);
        tc05::tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) bits[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 32; i += 4)
        *reinterpret_cast<uint4*>(acc + r * Z::LD + c0 + i) = make_uint4(bits[i], bits[i + 1], bits[i + 2], bits[i + 3]);
    }
  }
  double* acc_sums = reinterpret_cast<double*>(smem + Z::SUMS);  // [half][row]
  if (sums && warp >= SUM_WARP0)
    *reinterpret_cast<double2*>(acc_sums + sum_half * GS_BM + sum_block * 64 + lane * 2) = make_double2(row_sum[0], row_sum[1]);
  if (need_aux) asm volatile("cp.async.wait_all;" ::: "memory");
  tc05::tc_fence_before_sync();
  cg::cluster_group cluster = cg::this_cluster();
  if (p.splits > 1) cluster.sync(); else __syncthreads();
  if (warp == 1) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc(tmem, BN);
  }
  // a rolled loop, because a CTA that lands on an SM which has not run this kernel yet pays for every cache line of its code
#pragma unroll 1
  for (int i = 0; i * ROWS_PER_PASS < rows_mine; ++i) {
    const int r = sub + i * ROWS_PER_PASS;
    const int row = m0 + row_first + r;
    if (r >= rows_mine || row >= p.m || !col_ok) continue;
    float* at = acc + (row_first + r) * Z::LD + quad * 4;
    float v[4];
    if (p.splits > 1) {
      // All of them on their way before the first is added: one after the other they took a load from a peer each (256 tokens of 128 channels
      // 187 -> 180 us a step, 700 ragged tokens of 192 channels 340 -> 331, 1024 of 384 channels 815 -> 799).
      float4 t[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) t[s] = s < p.splits ? *reinterpret_cast<const float4*>(cluster.map_shared_rank(at, s)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[0] = v[1] = v[2] = v[3] = 0.f;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        if (s >= p.splits) break;
        v[0] += t[s].x; v[1] += t[s].y; v[2] += t[s].z; v[3] += t[s].w;
      }
    } else {
      const float4 t = *reinterpret_cast<const float4*>(at);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    v[0] += bias.x; v[1] += bias.y; v[2] += bias.z; v[3] += bias.w;
    if (p.epilogue == HL_EPI_BIAS_GELU) {
      // h = bf16(acc + bias) is the main output; g = bf16(gelu(h)) the second one
      uint2 g;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = bf16_round(v[e]);
      g.x = pack_bf16x2(gelu_fwd_fast(v[0]), gelu_fwd_fast(v[1]));
      g.y = pack_bf16x2(gelu_fwd_fast(v[2]), gelu_fwd_fast(v[3]));
      *reinterpret_cast<uint2*>(p.aux_out + (size_t)row * p.ld_aux_out + col) = g;
    } else if (need_aux) {
      const uint2 aux_now = *reinterpret_cast<const uint2*>(smem + Z::AUX + (r * BN + quad * 4) * 2);
      const float2 a0 = unpack_bf16x2(aux_now.x), a1 = unpack_bf16x2(aux_now.y);
      const float a[4] = {a0.x, a0.y, a1.x, a1.y};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        v[e] = p.epilogue == HL_EPI_BIAS_RESIDUAL ? a[e] + bf16_round(v[e]) : v[e] * gelu_grad_fast(a[e]);
    }
    if (p.out_bf16)
      *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.c) + (size_t)row * p.ldc + col) =
          make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    else
      *reinterpret_cast<float4*>(static_cast<float*>(p.c) + (size_t)row * p.ldc + col) = make_float4(v[0], v[1], v[2], v[3]);
  }
  if (sums && threadIdx.x < rows_mine && m0 + row_first + (int)threadIdx.x < p.m) {
    double v = 0.0;
    double* at = acc_sums + row_first + threadIdx.x;
    for (int s = 0; s < p.splits; ++s)
      for (int half = 0; half < 2; ++half) v += p.splits > 1 ? *cluster.map_shared_rank(at + half * GS_BM, s) : at[half * GS_BM];
    p.row_sum[m0 + row_first + threadIdx.x] = (float)v;
  }
  if (p.splits > 1) tc05::cluster_meet();  // no CTA leaves while another still reads its sums
  if (!ok || *abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);  // copies in flight land before shared memory is released
    if (threadIdx.x == 0) atomicExch(p.status + ST_WAIT_EXPIRED, 1);
  }
}

template <bool A_MN, bool B_MN, int BN, int STAGES>
int launch_small(hl_ctx* ctx, const CUtensorMap& ma, const CUtensorMap& mb, const GsParams& p, int grid) {
  using Z = GsSizes<BN, STAGES>;
  auto kern = gemm_small_kernel<A_MN, B_MN, BN, STAGES>;
  HL_ALLOW_SHARED(ctx, Z::SMEM, kern);
  HL_CUDA(launch_pdl(kern, (unsigned)grid, GS_THREADS, Z::SMEM, ctx->stream, p.splits, ma, mb, p));
  count_launch(ctx);
  ctx->counters.gemm_tcgen05_launches += 1;
  return HL_OK;
}

template <int BN, int STAGES>
int launch_majors(hl_ctx* ctx, bool a_mn, bool b_mn, const CUtensorMap& ma, const CUtensorMap& mb, const GsParams& p, int grid) {
  if (a_mn) return b_mn ? launch_small<true, true, BN, STAGES>(ctx, ma, mb, p, grid) : launch_small<true, false, BN, STAGES>(ctx, ma, mb, p, grid);
  return b_mn ? launch_small<false, true, BN, STAGES>(ctx, ma, mb, p, grid) : launch_small<false, false, BN, STAGES>(ctx, ma, mb, p, grid);
}

}  // namespace

// Which products run here, in which of three forms, and how many CTAs share a contraction: the smallest estimate, in
// microseconds, of
//   deep    128 x 64 tiles, eight stages, one CTA per SM     3.0 + 0.17 a k block (+ 1.6 when shared)
//   narrow  128 x 64 tiles, four stages, two CTAs per SM     3.0 + 0.34 a k block (+ 1.6)
//   wide    128 x 128 tiles, six stages, one CTA per SM      4.4 + 0.21 a k block (+ 2.5)
//   persistent kernel, 128 x 256 tiles                       6.0 + 0.33 a k block and wave (+ 4.5 when split or dealt out)
// where the first three have to fit into one wave.  The constants are fitted to products replayed back to back (4 to 65 k
// blocks, 1 to 288 CTAs; they are met within 10 to 15 %).  A k block costs a deep CTA less than the persistent kernel
// because it moves half the bytes, and the fixed part is what the set-up costs that the predecessor does not hide.
// Examples, persistent kernel against this one: 256 x 384 x 128 6.4 -> 3.7 us, 128 x 128 x 256 (transposed operands) 8.9 -> 4.0,
// 500 x 768 x 3072 22.4 -> 9.9, 2048 x 512 x 2048 15.2 -> 8.8, 4096 x 512 x 2048 19.1 -> 11.3, 3072 x 768 x 4099 (transposed)
// 23.8 -> 17.6.
namespace {
// CTAs of one wave of clusters of `splits`: a cluster sits in one GPC, so clusters of four and eight leave SMs over.  Asked of
// the driver once per form; form 0 deep, 1 narrow, 2 wide.
int wave_ctas(int form, int splits, int device, int sm_count) {
  static PerDevice clusters[3][4];
  const int at = splits == 1 ? 0 : splits == 2 ? 1 : splits == 4 ? 2 : 3;
  if (at == 0) return sm_count * (form == 1 ? 2 : 1);
  const int n = clusters[form][at].value(device, [&] {
    const size_t smem = form == 0 ? GsSizes<64, 8>::SMEM : form == 1 ? GsSizes<64, 4>::SMEM : GsSizes<128, 6>::SMEM;
    auto ask = [&](auto kern) {
      const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
      if (!ok) cudaGetLastError();
      return ok ? std::max(1, resident_clusters(kern, splits, GS_THREADS, smem)) : 1;
    };
    return form == 0 ? ask(gemm_small_kernel<true, true, 64, 8>)
                     : form == 1 ? ask(gemm_small_kernel<true, true, 64, 4>) : ask(gemm_small_kernel<true, true, 128, 6>);
  });
  return std::min(n * splits, sm_count * (form == 1 ? 2 : 1));
}
}  // namespace

GemmSmallPlan gemm_small_plan(const hl_gemm_desc* d, const GemmPlan& big, int device, int sm_count) {
  const int kb = ceil_div(d->k, GS_BK), m_tiles = ceil_div(d->m, GS_BM);
  const long long narrow = (long long)m_tiles * ceil_div(d->n, 64), wide = (long long)m_tiles * ceil_div(d->n, 128);
  const long long tiles = (long long)m_tiles * ceil_div(d->n, 256);
  float best = 6.0f;
  if (big.sk_tiles > 0) best += 0.33f * (float)tiles * (float)kb / (float)sm_count + 4.5f;
  else best += 0.33f * (float)ceil_div(kb, big.splits) * (float)ceil_div_ll(tiles * big.splits, sm_count) + (big.splits > 1 ? 4.5f : 0.f);
  // Products of bf16 pieces that stand for f32 operands keep at least the number of partial sums that they had: their error
  // is that of the accumulation.
  const int least = d->a_k_period > 0 || d->b_k_period > 0 ? std::min(big.splits, 8) : 1;
  GemmSmallPlan plan{0, 64, false};
  for (int s = 1; s <= 8 && (s == 1 || 2 * s <= kb); s *= 2) {
    if (s < least) continue;
    const float steps = (float)ceil_div(kb, s), shared = s > 1 ? 1.6f : 0.f;
    auto take = [&](float t, int bn, bool deep) {
      if (t < best) { best = t; plan = GemmSmallPlan{s, bn, deep}; }
    };
    if (narrow * s <= wave_ctas(0, s, device, sm_count)) take(3.0f + 0.17f * steps + shared, 64, true);
    else if (narrow * s <= wave_ctas(1, s, device, sm_count)) take(3.0f + 0.34f * steps + shared, 64, false);
    if (wide * s <= wave_ctas(2, s, device, sm_count)) take(4.4f + 0.21f * steps + (s > 1 ? 2.5f : 0.f), 128, false);
  }
  // A weight gradient (both operands down their rows) runs beside the next layer's kernels, and four stages leave these half of the SM:
  // with up to eight k blocks a CTA a step of 1024 tokens and 256 channels takes 466 us for 494, 384 tokens of 512 channels 1075 for 1088.
  // With 32 k blocks (2048 tokens of 512 channels) it is 2432 for 2408, and products that the next kernel waits for lose as well (700 tokens
  // of 192 channels 360 for 345 us).
  if (plan.deep && d->a_layout == HL_MN_MAJOR && d->b_layout == HL_MN_MAJOR && ceil_div(kb, plan.splits) <= 8) plan.deep = false;
  return plan;
}

// Arguments have been checked by the caller (gemm_bf16_run).
int gemm_small_run(hl_ctx* ctx, const hl_gemm_desc* d, const GemmSmallPlan& plan, const void* a, const void* b, void* c,
                   const float* bias, const void* aux_in, void* aux_out, float* row_sum) {
  const bool a_mn = d->a_layout == HL_MN_MAJOR, b_mn = d->b_layout == HL_MN_MAJOR;
  const int a_k = d->a_k_period > 0 ? d->a_k_period : d->k, b_k = d->b_k_period > 0 ? d->b_k_period : d->k;
  GsParams p{};
  p.m = d->m; p.n = d->n;
  p.k_blocks = ceil_div(d->k, GS_BK);
  p.splits = plan.splits;
  p.k_blocks_per_rank = ceil_div(p.k_blocks, p.splits);
  p.m_tiles = ceil_div(d->m, GS_BM);
  p.epilogue = d->epilogue;
  p.out_bf16 = d->out_dtype == HL_BF16;
  p.a_kb_wrap = d->a_k_period > 0 ? d->a_k_period / GS_BK : 0;
  p.b_kb_wrap = d->b_k_period > 0 ? d->b_k_period / GS_BK : 0;
  p.wait_limit_ns = ctx->wait_limit_ns ? ctx->wait_limit_ns : tc05::kWaitLimitNs;
  p.bias = bias;
  p.aux_in = static_cast<const __nv_bfloat16*>(aux_in);
  p.ld_aux_in = d->ld_aux_in > 0 ? d->ld_aux_in : d->ldc;
  p.c = c; p.ldc = d->ldc;
  p.aux_out = static_cast<__nv_bfloat16*>(aux_out);
  p.ld_aux_out = d->ld_aux_out > 0 ? d->ld_aux_out : d->ldc;
  p.row_sum = row_sum;
  p.status = ctx->status_dev;
  CUtensorMap ma, mb;
  int rc = a_mn ? make_tensor_map_bf16_2d(&ma, a, (uint64_t)d->m, (uint64_t)a_k, (uint64_t)d->lda, 64, GS_BK)
                : make_tensor_map_bf16_2d(&ma, a, (uint64_t)a_k, (uint64_t)d->m, (uint64_t)d->lda, GS_BK, GS_BM);
  if (rc != HL_OK) return rc;
  rc = b_mn ? make_tensor_map_bf16_2d(&mb, b, (uint64_t)d->n, (uint64_t)b_k, (uint64_t)d->ldb, 64, GS_BK)
            : make_tensor_map_bf16_2d(&mb, b, (uint64_t)b_k, (uint64_t)d->n, (uint64_t)d->ldb, GS_BK, (uint32_t)plan.bn);
  if (rc != HL_OK) return rc;
  const int grid = p.m_tiles * ceil_div(d->n, plan.bn) * p.splits;
  ProfileScope prof(ctx, HL_PROF_GEMM, 2.0 * (double)d->m * (double)d->n * (double)d->k);
  if (plan.bn == 128) return launch_majors<128, 6>(ctx, a_mn, b_mn, ma, mb, p, grid);
  return plan.deep ? launch_majors<64, 8>(ctx, a_mn, b_mn, ma, mb, p, grid) : launch_majors<64, 4>(ctx, a_mn, b_mn, ma, mb, p, grid);
}

}  // namespace hl
