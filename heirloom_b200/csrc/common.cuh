// Shared declarations for the sm_100a backend: context, error channel, dtype tags,
// vector helpers.  Everything here is internal; the public surface is include/heirloom_b200.h.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda.h>
#include <stdint.h>
#include <stddef.h>
#include <string>
#include <utility>
#include <algorithm>
#include "../../include/heirloom_b200.h"
#include "per_device.h"

namespace hl {

// Thread-local UTF-8 message behind hl_last_error(); mirrors the reference's
// CudaError{message} channel (heirloom-kernels/src/cuda.rs:259-280).
void set_error(const std::string& msg);
int fail(const std::string& msg);                      // sets the message, returns HL_ERR_*
int fail_cuda(cudaError_t e, const char* what);

#define HL_CUDA(expr)                                                     \
  do {                                                                    \
    cudaError_t _e = (expr);                                              \
    if (_e != cudaSuccess) return ::hl::fail_cuda(_e, #expr);             \
  } while (0)

#define HL_REQUIRE(cond, msg)                                             \
  do {                                                                    \
    if (!(cond)) return ::hl::fail(std::string(msg));                     \
  } while (0)

// Lets a kernel have that much dynamic shared memory on the context's device.
#define HL_ALLOW_SHARED(ctx, bytes, ...)                                                                            \
  do {                                                                                                              \
    static ::hl::PerDevice _allowed;                                                                                \
    HL_CUDA(_allowed.once((ctx)->device, [&] {                                                                      \
      return cudaFuncSetAttribute(__VA_ARGS__, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes));          \
    }));                                                                                                            \
  } while (0)

#define HL_LAUNCH_CHECK(name)                                             \
  do {                                                                    \
    cudaError_t _e = cudaGetLastError();                                  \
    if (_e != cudaSuccess) return ::hl::fail_cuda(_e, name);              \
  } while (0)

// Device status words.  Kernels never trap: a bad index or an expired wait writes a code
// here and the host folds it into the error channel at the next hl_ctx_sync/hl_status_check
// (the reference reads a status word after each launch, cuda.rs:7184-7193).
enum StatusSlot : int {
  ST_BAD_INDEX = 0,      // out-of-range gather/scatter/target index
  ST_WAIT_EXPIRED = 1,   // a bounded mbarrier wait ran out
  ST_BAD_ARGUMENT = 2,
  ST_SLOTS = 8
};

struct Counters {
  unsigned long long launches, gemm_tcgen05_launches, attention_launches, h2d_bytes, d2h_bytes,
      allocations, allocated_bytes, nccl_calls, nccl_bytes, gemm_pair_launches;
};

}  // namespace hl

struct hl_ctx {
  int device = 0;
  int sm_count = 0;
  unsigned long long wait_limit_ns = 0;  // bound of the kernels' waits where they take one (0 = the two-second default)
  bool forward_only = false;           // no backward pass follows: what only it would read need not be written
  int gemm_skip_kblock = -1;           // test hook of hl_ctx_set_test_hooks
  int reserve_sms = 0;                 // SMs the persistent kernels leave free while gradient collectives are in flight
  int comm_sms = 0;                    // how many they leave when asked to (0 = none); set when the communicator is made
  cudaStream_t stream = nullptr;       // compute stream
  cudaStream_t comm_stream = nullptr;  // collective stream
  int* status_dev = nullptr;           // hl::ST_SLOTS ints: status_host as the device sees it
  int* status_host = nullptr;          // pinned mirror
  void* workspace = nullptr;           // grow-only scratch (split-K partials, reductions)
  size_t workspace_bytes = 0;
  unsigned* gemm_sched = nullptr;      // counter of the GEMM's dynamic tile order: every processed tile adds one
  unsigned gemm_sched_base = 0;        // its value once every launch queued so far has finished
  unsigned faults = 0;                 // how often a bounded wait has run out so far
  void* gemm_flags = nullptr;          // per-CTA hand-over flags of the GEMM's work split, zeroed once
  hl::Counters counters{};
  void* nccl = nullptr;                // hl::NcclState*
  void* profiler = nullptr;            // hl::Profiler*, present while per-kernel timing is on
};

namespace hl {
// Programmatic dependent launch: the kernel may be resident before its predecessor on the stream has finished, so that its
// launch and its set-up cost no time of their own.  Such a kernel calls pdl_wait() before it touches anything a predecessor
// wrote (or still reads), and pdl_trigger() to let its own successor come in early; a wait covers all earlier kernels,
// because each of them waited too before it finished.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// For a kernel without set-up worth overlapping.  An early trigger does not take SMs from the kernel itself: its dependents
// come in only when all of its own blocks have started.
__device__ __forceinline__ void pdl_begin() {
  pdl_trigger();
  pdl_wait();
}
// The same for a kernel whose blocks stream through memory for a while (`streams`): it calls pdl_trigger() itself when its
// loop is over, so that no dependent sits on its SMs all that time.
__device__ __forceinline__ void pdl_begin(bool streams) {
  if (!streams) pdl_trigger();
  pdl_wait();
}
// `shared_percent` >= 0: the split of the SM's memory into shared memory and L1 that the kernel asks for (see `streaming`).
template <typename... P, typename... A>
cudaError_t launch_pdl_split(int shared_percent, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             int cluster, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[3] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  int n = 1;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)cluster; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (shared_percent >= 0) {
    attr[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[n].val.sharedMemCarveout = (unsigned)shared_percent;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
  return launch_pdl_split(-1, kernel, grid, block, smem, stream, cluster, std::forward<A>(args)...);
}

// How many clusters of a kernel the current device holds at once; 0 when it cannot be told.
template <typename... P>
int resident_clusters(void (*kernel)(P...), int cluster, int threads, size_t smem) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(cluster * 1024));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)cluster; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess) return n;
  cudaGetLastError();
  return 0;
}

constexpr double kStreamingBytes = 16e6;

// pdl(kernel, grid, block, shared memory, stream)(arguments): the launch above in place of <<< >>>, errors through
// cudaGetLastError like there.
template <typename... P>
struct PdlLauncher {
  void (*kernel)(P...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
  int shared_percent = -1;
  // A kernel that waits for memory keeps its loads in flight in L1.  Launched as a dependent it starts on SMs that never run
  // empty, and without a wish of its own it keeps the split that a GEMM left behind: 227 KB of shared memory, hardly any L1
  // (loss kernel, 16384 x 50304: 1216 us instead of 927; column sums of 16384 x 3072: 49 instead of 30).  Asking for L1 lets
  // the SM drain first, which a kernel of a few microseconds would feel, so only launches of 16 MB and up (3 us at full rate) ask.
  // `bytes`: what the launch reads and writes; `percent`: the shared memory of its resident blocks.
  PdlLauncher streaming(double bytes, int percent = 8) const {
    PdlLauncher l = *this;
    l.shared_percent = bytes >= kStreamingBytes ? percent : -1;
    return l;
  }
  void operator()(P... args) const { launch_pdl_split(shared_percent, kernel, grid, block, smem, stream, 1, args...); }
};
template <typename... P>
PdlLauncher<P...> pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  return PdlLauncher<P...>{kernel, grid, block, smem, stream};
}

int ensure_workspace(hl_ctx* ctx, size_t bytes);
// For a form that can be done without: false, with the arena as it was, where the device has no room for the larger one beside it.
bool try_workspace(hl_ctx* ctx, size_t bytes);
inline void count_launch(hl_ctx* ctx, unsigned long long n = 1) { ctx->counters.launches += n; }
// SMs a persistent one-CTA-per-SM kernel should fill: all of them, minus those left to the collective kernels.  A CTA of
// those kernels takes a whole SM's registers or shared memory, so it cannot start on an SM a collective kernel sits
// on, and a grid of one CTA per SM would wait for that SM with its share of the tiles.
inline int persistent_sms(const hl_ctx* ctx) { return std::max(1, ctx->sm_count - ctx->reserve_sms); }

// Opt-in per-kernel timing: a scope brackets the launches of one op with two events on the
// compute stream; hl_profile_read folds them by category after a stream sync (the reference's
// opt-in launch-family timing, heirloom-kernels/src/cuda.rs:8574-8611, forces a sync per
// launch instead).  `work` is the algorithmic flops (GEMM, attention) or bytes (the rest).
void profile_begin(hl_ctx* ctx, int category, double work);
void profile_end(hl_ctx* ctx);
struct ProfileScope {
  hl_ctx* ctx;
  ProfileScope(hl_ctx* c, int category, double work) : ctx(c) { if (c->profiler) profile_begin(c, category, work); }
  ~ProfileScope() { if (ctx->profiler) profile_end(ctx); }
};

inline size_t dtype_size(int dtype) {
  switch (dtype) {
    case HL_F32: return 4;
    case HL_BF16: return 2;
    case HL_F64: return 8;
    case HL_I64: return 8;
    case HL_U8: return 1;
    default: return 0;
  }
}

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }

// n / d for 0 <= n < 2^31 by a multiplication (Granlund and Montgomery 1994, "Division by invariant integers using multiplication"), for divisors known at launch: a division
// takes some 200 cycles.
struct QuickDiv {
  uint32_t mul, shift;
  QuickDiv(uint32_t d = 1) : shift(0) {
    while ((1ull << shift) < d) ++shift;
    mul = (uint32_t)(((1ull << 32) * ((1ull << shift) - d)) / d + 1);
  }
  __device__ __forceinline__ int operator()(int n) const { return (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shift); }
};

// f32 -> bf16 round-to-nearest-even (same rounding as the reference's storage.rs:440-445).
__device__ __forceinline__ __nv_bfloat16 to_bf16(float x) { return __float2bfloat16_rn(x); }
__device__ __forceinline__ float from_bf16(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

// tanh-approximate GELU and its derivative (reference: src/tensor.rs:5152-5154,
// src/tensor/autograd.rs:2891-2897).
template <typename T>
__device__ __forceinline__ T gelu_fwd(T x) {
  const T c = T(0.7978845608028654);
  T inner = c * (x + T(0.044715) * x * x * x);
  return T(0.5) * x * (T(1) + tanh(inner));
}
template <typename T>
__device__ __forceinline__ T gelu_grad(T x) {
  const T c = T(0.7978845608028654);
  T inner = c * (x + T(0.044715) * x * x * x);
  T t = tanh(inner);
  T sech2 = T(1) - t * t;
  T dinner = c * (T(1) + T(3.0 * 0.044715) * x * x);
  return T(0.5) * (T(1) + t) + T(0.5) * x * sech2 * dinner;
}
__device__ __forceinline__ float gelu_fwd_f(float x) {
  float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(inner));
}
__device__ __forceinline__ float gelu_grad_f(float x) {
  float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  float t = tanhf(inner);
  float sech2 = 1.0f - t * t;
  float dinner = 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x * x);
  return 0.5f * (1.0f + t) + 0.5f * x * sech2 * dinner;
}

// Round-to-nearest-even to bf16 precision with integer ops (same result as the conversion
// instruction for every finite input and infinities).  The GEMM epilogues use it because the
// conversion instructions share the 16-lane special-function pipe with tanh.
__device__ __forceinline__ uint32_t bf16_rne_bits(float x) {
  uint32_t u = __float_as_uint(x);
  u += 0x7FFFu + ((u >> 16) & 1u);
  return u & 0xFFFF0000u;
}
__device__ __forceinline__ float bf16_round_alu(float x) { return __uint_as_float(bf16_rne_bits(x)); }
// Packs two floats that are already bf16-representable (low 16 bits zero).
__device__ __forceinline__ uint32_t pack_rounded_bf16x2(float lo, float hi) {
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}

// 2^x in one MUFU op (relative error about 2^-22; results below the normal range flush to zero,
// 2^-inf = 0).  exp2f() adds a range check and two scalings around the same instruction.
__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Hardware tanh (one MUFU op, relative error about 2^-11): enough for values that are rounded
// to bf16 right after, as in the GEMM epilogues.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The tanh form of GELU and its derivative, written as the shortest chains of fused multiply-adds (the epilogues that use
// them are bound by their instruction count): gelu(x) = hx + hx*t with hx = x/2, t = tanh(x*(k0 + k1*x^2)).
__device__ __forceinline__ float gelu_fwd_fast(float x) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.7978845608028654f * 0.044715f;
  const float x2 = x * x;
  const float t = tanh_fast(x * fmaf(x2, k1, k0));
  const float hx = 0.5f * x;
  return fmaf(hx, t, hx);
}
// Two f32 operations an instruction (the same roundings as two single ones).
__device__ __forceinline__ unsigned long long as_u64(float2 v) { return (unsigned long long)__float_as_uint(v.y) << 32 | __float_as_uint(v.x); }
__device__ __forceinline__ float2 as_float2(unsigned long long u) { return make_float2(__uint_as_float((unsigned)u), __uint_as_float((unsigned)(u >> 32))); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(as_u64(a)), "l"(as_u64(b)), "l"(as_u64(c)));
  return as_float2(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(as_u64(a)), "l"(as_u64(b)));
  return as_float2(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(as_u64(a)), "l"(as_u64(b)));
  return as_float2(r);
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 gelu_fwd_fast2(float2 x) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.7978845608028654f * 0.044715f;
  const float2 a = mul2(x, fma2(mul2(x, x), both(k1), both(k0)));
  const float2 t = make_float2(tanh_fast(a.x), tanh_fast(a.y));
  const float2 hx = mul2(x, both(0.5f));
  return fma2(hx, t, hx);
}
// gelu'(x) = (1 + t)/2 + hx*(1 - t^2)*(k0 + 3*k1*x^2)
__device__ __forceinline__ float gelu_grad_fast(float x) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.7978845608028654f * 0.044715f;
  const float x2 = x * x;
  const float t = tanh_fast(x * fmaf(x2, k1, k0));
  const float dinner = fmaf(x2, 3.0f * k1, k0);
  const float sech2 = fmaf(-t, t, 1.0f);
  return fmaf(0.5f * x * sech2, dinner, fmaf(0.5f, t, 0.5f));
}
__device__ __forceinline__ float2 gelu_grad_fast2(float2 x) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.7978845608028654f * 0.044715f;
  const float2 x2 = mul2(x, x);
  const float2 a = mul2(x, fma2(x2, both(k1), both(k0)));
  const float2 t = make_float2(tanh_fast(a.x), tanh_fast(a.y));
  const float2 dinner = fma2(x2, both(3.0f * k1), both(k0));
  const float2 sech2 = fma2(make_float2(-t.x, -t.y), t, both(1.0f));
  return fma2(mul2(mul2(x, both(0.5f)), sech2), dinner, fma2(t, both(0.5f), both(0.5f)));
}

// Eight f32 values as three bf16 pieces each, sixteen bytes a piece: hi = bf16(x), mid = bf16(x - hi), lo = bf16(x - hi - mid).  The
// differences are exact, so that hi + mid + lo == x whenever the three 8-bit mantissas reach the last bit of x.
__device__ __forceinline__ void split8_bf16(const float (&x)[8], uint4 (&piece)[3]) {
  uint32_t w[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = x[2 * i], b = x[2 * i + 1];
    w[0][i] = pack_bf16x2(a, b);
    a -= __uint_as_float(w[0][i] << 16);
    b -= __uint_as_float(w[0][i] & 0xFFFF0000u);
    w[1][i] = pack_bf16x2(a, b);
    w[2][i] = pack_bf16x2(a - __uint_as_float(w[1][i] << 16), b - __uint_as_float(w[1][i] & 0xFFFF0000u));
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) piece[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    T other = __shfl_xor_sync(0xffffffffu, v, o);
    v = other > v ? other : v;
  }
  return v;
}

// Block-wide sum for blockDim.x <= 1024 (multiple of 32); result valid in every thread.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* smem /* >= 32 entries */) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  T r = (lane < nw) ? smem[lane] : T(0);
  r = warp_sum(r);
  return r;
}
template <typename T>
__device__ __forceinline__ T block_max(T v, T* smem, T lowest) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  T r = (lane < nw) ? smem[lane] : lowest;
  r = warp_max(r);
  return r;
}

}  // namespace hl
