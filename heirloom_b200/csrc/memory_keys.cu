// Half-key gradients of the product-key lookup on the tensor cores: dK = Wᵀ·Q of one table, W[t, row] being the sum of the score
// gradients of token t whose slots map to the row.
//
// W has top_k entries in a row of `side`, but with a few hundred rows a table every row collects about tokens * top_k / side terms:
// sums over scattered rows pile onto few addresses, and the dense f32 product of product_key_dkeys_kernel is bound by f32 issue
// (16384 tokens, 32 of 2 x 512 rows of 256: 301 us).  Here both operands are three bf16 pieces each (hi + mid + lo is the f32 value
// exactly; the queries are cut up beforehand, W's entries on their way into shared memory), and the six products above 2^-24 of the
// largest run as bf16 products, which are exact in f32.  The tensor core's additions truncate, so the large products (hi * hi) have an
// accumulator of their own that is emptied into registers every 32 tokens, two additions deep, and the sums between are rounded
// f32 additions; the five small products, 2^-8 of them and less, share another that is emptied every 1024 tokens.  Error against f64
// (norms; f32 product's): 16384 tokens 1.2e-7 (1.9e-7), 4096 1.2e-7 (1.6e-7), 2048 0.95e-7 (1.05e-7).  With all six in one accumulator
// 64 tokens deep it was 2.2e-7, 2.4e-7 and 2.1e-7.
//
// A CTA takes 128 rows of one table, all columns and a share of the tokens.  A stage of 32 tokens: the queries' pieces by TMA; of
// W, sixteen warps put the entries of two tokens each into a tile that is zero otherwise, and take them out again before the tile
// is used next (slots that share a row are added first, in a fixed order).  The same warps
// empty the accumulators, beside the small products of the next stage.  A stage's twelve instructions of 128 x 256 x 16 take 1536
// cycles; bound by those warps' chain of loads, exchanges and stores, some 5400 cycles a stage (tensor pipe 33 % active, instructions
// issued in 31 % of the cycles): 83 us for the size above, 16 more for the queries' pieces.  Eighteen warps leave a thread 96
// registers, of which the kernel for 256 columns spills 484 bytes.
#include "kernels.h"
#include "tc05.cuh"

namespace hl {
namespace {

constexpr int KG_TOKENS = 32;   // a stage
constexpr int KG_STAGES = 3;
constexpr int KG_SMALL = 32;    // stages until the small products' accumulator is emptied
constexpr int KG_ROWS = 128;
constexpr int KG_WARPS = 16;
constexpr int KG_THREADS = (KG_WARPS + 2) * 32;
constexpr int KG_CHUNK = KG_TOKENS * 128;            // 64 rows or columns of a stage: 4 KB
constexpr int KG_W_PIECE = 2 * KG_CHUNK;
constexpr int KG_TW = KG_TOKENS / KG_WARPS;          // tokens of a warp in a stage
// Pieces rebuild a value only where all three are finite, and an infinity times a piece of either sign is NaN.  So where any score
// gradient or query is this large, infinite or NaN, the sums are f32 products of the values themselves, zeros of W included, on the
// same CTAs (some ten times as slow); below it no product or sum of up to 2^27 terms overflows.
constexpr float kWide = 0x1p47f;

template <int NC>
struct KgLayout {  // NC: 64-column chunks
  static constexpr int Q_PIECE = NC * KG_CHUNK;
  static constexpr int STAGE = 3 * (KG_W_PIECE + Q_PIECE);
  static constexpr int SMEM = KG_STAGES * STAGE + 256;
};
static_assert(KgLayout<4>::SMEM <= 227 * 1024, "shared memory budget");

struct KgBarriers {
  uint64_t full[KG_STAGES], empty[KG_STAGES];  // full: the queries' bytes and the warps that build W
  uint64_t large_full, large_empty, small_full, small_empty;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(KgBarriers) <= 256, "barriers outgrow their place");

template <int NC>
__global__ void __launch_bounds__(KG_THREADS, 1)
key_gradient_kernel(const __grid_constant__ CUtensorMap map_q, const int64_t* __restrict__ idx, const float* __restrict__ query,
                    long long ld_query, const float* __restrict__ grad_scores, const int* __restrict__ wide_seen,
                    float* __restrict__ partial, int tokens, int top_k, int side, int half, int slots, int tokens_per_block,
                    int* __restrict__ status, unsigned long long wait_limit_ns, int skip_stage) {
  extern __shared__ __align__(1024) uint8_t kg_smem[];
  using L = KgLayout<NC>;
  constexpr int N = NC * 64;
  KgBarriers* bars = reinterpret_cast<KgBarriers*>(kg_smem + KG_STAGES * L::STAGE);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int table = blockIdx.z, r0 = blockIdx.y * KG_ROWS;
  const int t_begin = min(tokens, (int)blockIdx.x * tokens_per_block), t_end = min(tokens, t_begin + tokens_per_block);

  if (threadIdx.x == 0) {
    for (int i = 0; i < KG_STAGES; ++i) {
      tc05::mbar_init(&bars->full[i], KG_WARPS + 1);
      tc05::mbar_init(&bars->empty[i], 1);
    }
    tc05::mbar_init(&bars->large_full, 1);
    tc05::mbar_init(&bars->large_empty, KG_WARPS);
    tc05::mbar_init(&bars->small_full, 1);
    tc05::mbar_init(&bars->small_empty, KG_WARPS);
    bars->abort_flag = (tc05::smem_u32(kg_smem) & 1023u) == 0 ? 0 : 1;
    tc05::fence_barrier_init();
  }
  for (int s = 0; s < KG_STAGES; ++s)
    for (int i = threadIdx.x; i < 3 * KG_W_PIECE / 16; i += KG_THREADS)
      *reinterpret_cast<uint4*>(kg_smem + s * L::STAGE + i * 16) = make_uint4(0, 0, 0, 0);
  tc05::fence_proxy_async_smem();
  if (warp == KG_WARPS) {
    tc05::tmem_alloc(&bars->tmem_base, 512);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  tc05::tc_fence_after_sync();
  const uint32_t tmem_large = bars->tmem_base, tmem_small = tmem_large + 256;
  pdl_begin();
  const bool wide = __ldcg(wide_seen) != 0;
  const int stages = wide ? 0 : (t_end - t_begin + KG_TOKENS - 1) / KG_TOKENS;
  // at the end of which stages the small products' accumulator is emptied; the large ones' is at the end of each
  auto ends_small = [&](int s) { return s % KG_SMALL == KG_SMALL - 1 || s == stages - 1; };

  if (warp == KG_WARPS + 1) {
    // ------------------------------------------------------------------ queries
    if (tc05::elect_one() && !*abort_flag) {
      tc05::tma_prefetch_desc(&map_q);
      int st = 0;
      uint32_t phase = 0;
      for (int s = 0; s < stages; ++s) {
        if (!tc05::mbar_wait(&bars->empty[st], phase ^ 1u, abort_flag, wait_limit_ns)) break;
        if (s == skip_stage) break;  // test hook: this stage never fills
        tc05::mbar_arrive_expect_tx(&bars->full[st], 3 * L::Q_PIECE);
        uint8_t* q = kg_smem + st * L::STAGE + 3 * KG_W_PIECE;
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int c = 0; c < NC; ++c)
            tc05::tma_load_3d(q + p * L::Q_PIECE + c * KG_CHUNK, &map_q, &bars->full[st], table * half + c * 64, t_begin + s * KG_TOKENS, p);
        if (++st == KG_STAGES) { st = 0; phase ^= 1u; }
      }
    }
  } else if (warp == KG_WARPS) {
    // ------------------------------------------------------------------ products
    if (tc05::elect_one() && !*abort_flag) {
      constexpr uint32_t idesc = tc05::instr_desc_bf16_f32(KG_ROWS, N, true, true);
      int st = 0;
      uint32_t phase = 0, large = 0, small = 0;  // how often each accumulator has been handed over, modulo 2
      for (int s = 0; s < stages; ++s) {
        if (!tc05::mbar_wait(&bars->full[st], phase, abort_flag, wait_limit_ns)) break;
        if (s % KG_SMALL == 0 && !tc05::mbar_wait(&bars->small_empty, small ^ 1u, abort_flag, wait_limit_ns)) break;
        tc05::tc_fence_after_sync();
        const uint32_t w = tc05::smem_u32(kg_smem + st * L::STAGE), q = w + 3 * KG_W_PIECE;
        auto product = [&](uint32_t d, int pw, int pq, int ks, uint32_t acc) {
          tc05::umma_ss(d, tc05::smem_desc_sw128(w + pw * KG_W_PIECE + ks * 2048, KG_CHUNK, 1024),
                        tc05::smem_desc_sw128(q + pq * L::Q_PIECE + ks * 2048, KG_CHUNK, 1024), idesc, acc);
        };
#pragma unroll
        for (int pair = 0; pair < 5; ++pair) {
          constexpr int kW[5] = {2, 0, 1, 1, 0}, kQ[5] = {0, 2, 1, 0, 1};
#pragma unroll
          for (int ks = 0; ks < KG_TOKENS / 16; ++ks) product(tmem_small, kW[pair], kQ[pair], ks, s % KG_SMALL == 0 && pair == 0 && ks == 0 ? 0u : 1u);
        }
        if (!tc05::mbar_wait(&bars->large_empty, large ^ 1u, abort_flag, wait_limit_ns)) break;
        tc05::tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < KG_TOKENS / 16; ++ks) product(tmem_large, 0, 0, ks, ks == 0 ? 0u : 1u);
        tc05::umma_commit(&bars->empty[st]);
        tc05::umma_commit(&bars->large_full);
        large ^= 1u;
        if (ends_small(s)) { tc05::umma_commit(&bars->small_full); small ^= 1u; }
        if (++st == KG_STAGES) { st = 0; phase ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------------ W and the sums
    const unsigned side32 = (unsigned)side;
    auto row_of = [&](int slot) -> int {  // within this CTA's rows, -1 outside
      const int row = (int)(table ? (unsigned)slot % side32 : (unsigned)slot / side32) - r0;
      return slot < 0 || row < 0 || row >= KG_ROWS ? -1 : row;
    };
    auto slot_of = [&](int t, int& slot, float& g) {  // this lane's of token t; -1: none, or none of the table
      const bool in = t < t_end && lane < top_k;
      const long long at = in ? __ldg(idx + (size_t)t * top_k + lane) : -1;
      slot = at >= 0 && at < slots ? (int)at : -1;
      g = in ? __ldg(grad_scores + (size_t)t * top_k + lane) : 0.f;
    };
    int next_slot[KG_TW];
    float next_g[KG_TW];
    auto fetch = [&](int t0) {  // of the stage whose first token is t0
#pragma unroll
      for (int i = 0; i < KG_TW; ++i) slot_of(t0 + warp + i * KG_WARPS, next_slot[i], next_g[i]);
    };
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const int col0 = (warp >> 2) * (N / 4);  // this thread's columns of its row
    float sum[N / 4];
#pragma unroll
    for (int i = 0; i < N / 4; ++i) sum[i] = 0.f;
    auto drain = [&](uint64_t* full, uint64_t* empty, uint32_t from, uint32_t& phase) -> bool {
      if (!tc05::mbar_wait(full, phase, abort_flag, wait_limit_ns)) return false;
      phase ^= 1u;
      tc05::tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < N / 4; c += 16) {
        uint32_t v[16];
        tc05::tmem_ld_32x32b_x16(from + (uint32_t)(col0 + c) + lane_sel, v);
        tc05::tmem_ld_wait();
        tc05::tmem_ld_fence(v);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(v[i]);
      }
      tc05::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc05::mbar_arrive(empty);
      return true;
    };
    uint32_t large = 0, small = 0;
    auto drain_after = [&](int s) -> bool {  // what stage s was the last one of
      if (!drain(&bars->large_full, &bars->large_empty, tmem_large, large)) return false;
      return !ends_small(s) || drain(&bars->small_full, &bars->small_empty, tmem_small, small);
    };
    // where this lane's entries of each stage's tile stand (-1: nowhere), so that they can be taken out again
    int placed[KG_STAGES][KG_TW];
#pragma unroll
    for (int i = 0; i < KG_STAGES; ++i)
#pragma unroll
      for (int j = 0; j < KG_TW; ++j) placed[i][j] = -1;
    auto put = [&](uint8_t* at, float x) {
      const __nv_bfloat16 hi = __float2bfloat16_rn(x);
      const float rest = x - __bfloat162float(hi);
      const __nv_bfloat16 mid = __float2bfloat16_rn(rest);
      *reinterpret_cast<__nv_bfloat16*>(at) = hi;
      *reinterpret_cast<__nv_bfloat16*>(at + KG_W_PIECE) = mid;
      *reinterpret_cast<__nv_bfloat16*>(at + 2 * KG_W_PIECE) = __float2bfloat16_rn(rest - __bfloat162float(mid));
    };
    bool ok = !*abort_flag;
    if (wide) {
      for (int t = t_begin; t < t_end; ++t) {
        int slot;
        float g, w = 0.f;  // w: this thread's row of W, the token's slots in order
        slot_of(t, slot, g);
        const int of = row_of(slot);
        for (int j = 0; j < top_k; ++j) {
          const int at = __shfl_sync(0xffffffffu, of, j);
          const float more = __shfl_sync(0xffffffffu, g, j);
          if (at == (warp & 3) * 32 + lane) w += more;
        }
        const float* q = query + (size_t)t * ld_query + table * half + col0;
#pragma unroll
        for (int i = 0; i < N / 4; i += 4)
          if (col0 + i < half) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(q + i));
            sum[i] = fmaf(w, v.x, sum[i]);
            sum[i + 1] = fmaf(w, v.y, sum[i + 1]);
            sum[i + 2] = fmaf(w, v.z, sum[i + 2]);
            sum[i + 3] = fmaf(w, v.w, sum[i + 3]);
          }
      }
    }
    if (ok && stages > 0) fetch(t_begin);
    for (int s0 = 0; ok && s0 < stages; s0 += KG_STAGES) {
#pragma unroll
      for (int st = 0; st < KG_STAGES; ++st) {
        const int s = s0 + st;
        if (!ok || s >= stages) break;
        int row[KG_TW];
        float g[KG_TW];
#pragma unroll
        for (int i = 0; i < KG_TW; ++i) {
          row[i] = row_of(next_slot[i]);
          g[i] = next_g[i];
        }
        if (s + 1 < stages) fetch(t_begin + (s + 1) * KG_TOKENS);
        // The first lane of those whose slots share a row gets the sum of all: every lane holds the sum from itself up to the one
        // that its pointer names, adds that one's and takes over its pointer.  A token's slots share few rows (a handful for 32 slots):
        // five rounds at most where adding one after the other took up to thirty.
        int next[KG_TW];
        bool any = false;
#pragma unroll
        for (int i = 0; i < KG_TW; ++i) {
          const unsigned same = __match_any_sync(0xffffffffu, row[i]), above = same & ~((2u << lane) - 1u);
          next[i] = row[i] >= 0 && above != 0 ? __ffs(above) - 1 : -1;
          if ((same & ((1u << lane) - 1u)) != 0) row[i] = -1;
          any |= next[i] >= 0;
        }
        while (__any_sync(0xffffffffu, any)) {
          any = false;
#pragma unroll
          for (int i = 0; i < KG_TW; ++i) {
            const int from = next[i] >= 0 ? next[i] : lane;
            const float v = __shfl_sync(0xffffffffu, g[i], from);
            const int further = __shfl_sync(0xffffffffu, next[i], from);
            if (next[i] >= 0) {
              g[i] += v;
              next[i] = further;
            }
            any |= next[i] >= 0;
          }
        }
        if (!tc05::mbar_wait(&bars->empty[st], ((uint32_t)(s / KG_STAGES) & 1u) ^ 1u, abort_flag, wait_limit_ns)) { ok = false; break; }
        uint8_t* w = kg_smem + st * L::STAGE;
#pragma unroll
        for (int i = 0; i < KG_TW; ++i)
          if (placed[st][i] >= 0) {
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint16_t*>(w + p * KG_W_PIECE + placed[st][i]) = 0;
          }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < KG_TW; ++i) {
          const int t = warp + i * KG_WARPS, r = row[i];
          placed[st][i] = r < 0 ? -1 : (r >> 6) * KG_CHUNK + t * 128 + ((((r >> 3) & 7) ^ (t & 7)) << 4) + (r & 7) * 2;
          if (r >= 0) put(w + placed[st][i], g[i]);
        }
        tc05::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc05::mbar_arrive(&bars->full[st]);
        if (s > 0) ok = drain_after(s - 1);
      }
    }
    if (ok && stages > 0) ok = drain_after(stages - 1);
    // partial[share of the tokens][table][side][half]
    const int row = r0 + (warp & 3) * 32 + lane;
    if (ok && row < side) {
      float* dst = partial + (((size_t)blockIdx.x * 2 + table) * side + row) * half;
#pragma unroll
      for (int i = 0; i < N / 4; i += 4)
        if (col0 + i < half) *reinterpret_cast<float4*>(dst + col0 + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
    }
  }
  tc05::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (threadIdx.x == 0) atomicExch(status + ST_WAIT_EXPIRED, 1);
  }
  if (warp == KG_WARPS) {
    tc05::tc_fence_after_sync();
    tc05::tmem_dealloc(tmem_large, 512);
  }
}

// The queries' three pieces, one below the other: eight values a thread; and whether any value is too wide for pieces.
__global__ void split_queries_kernel(const float* __restrict__ query, long long ld, uint4* __restrict__ out, int tokens, int dim,
                                     const float* __restrict__ grad_scores, size_t scores, int* __restrict__ wide_seen) {
  pdl_begin();
  bool wide = false;
  auto look = [&](float x) { wide |= !(fabsf(x) < kWide); };  // NaN too
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < scores; i += (size_t)gridDim.x * blockDim.x) look(__ldg(grad_scores + i));
  const size_t per_piece = (size_t)tokens * dim / 8;
  const int groups = dim / 8;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < per_piece; i += (size_t)gridDim.x * blockDim.x) {
    const unsigned t = (unsigned)i / (unsigned)groups, c = (unsigned)i - t * (unsigned)groups;  // fewer than 2^31 groups: checked at launch
    const float4* src = reinterpret_cast<const float4*>(query + (size_t)t * ld + c * 8);
    const float4 a = __ldg(src), b = __ldg(src + 1);
    const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) look(x[j]);
    uint4 piece[3];
    split8_bf16(x, piece);
#pragma unroll
    for (int p = 0; p < 3; ++p) out[p * per_piece + i] = piece[p];
  }
  if (wide) *wide_seen = 1;
}

template <int NC>
int launch_key_gradient(hl_ctx* ctx, const KeyGradient& k, const CUtensorMap& map_q, const int* wide_seen, int shares, float* partial) {
  HL_ALLOW_SHARED(ctx, KgLayout<NC>::SMEM, key_gradient_kernel<NC>);
  const int tokens_per_block = ceil_div(ceil_div(k.tokens, shares), KG_TOKENS) * KG_TOKENS;
  pdl(key_gradient_kernel<NC>, dim3(shares, ceil_div(k.side, KG_ROWS), 2), KG_THREADS, KgLayout<NC>::SMEM, ctx->stream)(
      map_q, k.idx, k.query, k.ld_query, k.grad_scores, wide_seen, partial, k.tokens, k.top_k, k.side, k.half, k.slots, tokens_per_block,
      ctx->status_dev, ctx->wait_limit_ns ? ctx->wait_limit_ns : tc05::kWaitLimitNs, ctx->gemm_skip_kblock);
  HL_LAUNCH_CHECK("key_gradient_kernel");
  count_launch(ctx);
  return HL_OK;
}

constexpr size_t kWideWordBytes = 256;  // in front of the pieces: the word that says whether a value is too wide for them
size_t query_bytes(const KeyGradient& k) { return ((size_t)k.tokens * k.half * 2 * 3 * sizeof(__nv_bfloat16) + 255) & ~size_t(255); }

}  // namespace

// From 2048 tokens on: the f32 product is the more accurate one below (1024 tokens: 0.95e-7 against 1.13e-7), where its sums are
// short.  Whole backward call before / after, us: 16384 tokens 2 x 512 x 256 374 / 212, 2 x 32 x 32 100 / 81; 4096, 2 x 200 x 96 53 / 39;
// 2048, 2 x 512 x 256 87 / 63.  A row's slots are a warp's lanes, hence at most 32.
constexpr int kMinTokens = 2048;
int key_gradient_shares(const hl_ctx* ctx, const KeyGradient& k) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(k.query);
  if (k.tokens < kMinTokens || k.top_k > 32 || k.half > 256 || k.half % 8 != 0 || k.ld_query % 4 != 0 || (at & 15) != 0 ||
      (size_t)k.tokens * k.half * 2 >= (size_t(1) << 31))
    return 0;
  const int tiles = 2 * ceil_div(k.side, KG_ROWS);
  return std::max(1, std::min(ceil_div(k.tokens, 2 * KG_TOKENS), ctx->sm_count / tiles));
}

size_t key_gradient_bytes(const KeyGradient& k, int shares) {
  return kWideWordBytes + query_bytes(k) + sizeof(float) * (size_t)shares * 2 * k.side * k.half;
}

int key_gradient_run(hl_ctx* ctx, const KeyGradient& k, int shares, void* scratch, float** partial) {
  int* wide_seen = static_cast<int*>(scratch);
  uint8_t* pieces = static_cast<uint8_t*>(scratch) + kWideWordBytes;
  *partial = reinterpret_cast<float*>(pieces + query_bytes(k));
  const int dim = 2 * k.half;
  const size_t groups = (size_t)k.tokens * dim / 8;
  pdl(split_queries_kernel, (unsigned)std::min<size_t>((groups + 255) / 256, (size_t)ctx->sm_count * 8), 256, 0, ctx->stream)(
      k.query, k.ld_query, reinterpret_cast<uint4*>(pieces), k.tokens, dim, k.grad_scores, (size_t)k.tokens * k.top_k, wide_seen);
  HL_LAUNCH_CHECK("split_queries_kernel");
  count_launch(ctx);
  CUtensorMap map_q;
  const int rc = make_tensor_map_bf16_3d(&map_q, pieces, (uint64_t)dim, (uint64_t)k.tokens, 3, (uint64_t)dim, (uint64_t)dim * k.tokens, 64, KG_TOKENS, 1);
  if (rc != HL_OK) return rc;
  switch (ceil_div(k.half, 64)) {
    case 1: return launch_key_gradient<1>(ctx, k, map_q, wide_seen, shares, *partial);
    case 2: return launch_key_gradient<2>(ctx, k, map_q, wide_seen, shares, *partial);
    case 3: return launch_key_gradient<3>(ctx, k, map_q, wide_seen, shares, *partial);
    default: return launch_key_gradient<4>(ctx, k, map_q, wide_seen, shares, *partial);
  }
}

}  // namespace hl
