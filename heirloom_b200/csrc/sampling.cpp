// Next-token sampling on the host, over one row of logits: the reference's controls (repetition, frequency and presence
// penalties, temperature, top-k, top-p, greedy at temperature 0; src/nn.rs:1595-1751) in one native call.  Host code: the
// logits are in host memory by then, and 50 k doubles take tens of microseconds here where a walk over them in Python
// takes milliseconds (8 tokens of a 50304-word vocabulary: 62 ms of host time before, 0.6 ms with this).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <exception>
#include <limits>
#include <string>
#include <vector>

#include "../../include/heirloom_b200.h"

namespace hl {
int fail(const std::string& msg);
namespace {
#define HL_REQUIRE(cond, msg) \
  do { \
    if (!(cond)) return ::hl::fail(std::string(msg)); \
  } while (0)

// Eight lanes as one GCC vector: one AVX-512 register, two AVX2 ones or four of SSE2, by the function it is inlined into.
constexpr int LANES = 8;
typedef double Lanes __attribute__((vector_size(8 * LANES)));
typedef int64_t Words __attribute__((vector_size(8 * LANES)));
#define HL_INLINE inline __attribute__((always_inline))
HL_INLINE void load_lanes(Lanes* v, const double* p) { __builtin_memcpy(v, p, sizeof(Lanes)); }

// *y = e^*x for *x <= 0: x = n ln2 + r, |r| <= ln2/2, the Taylor polynomial of degree 13 (its remainder is 4e-18 of e^r) and
// n added to the exponent.  Below -708 the result is 0; those terms are 1e-308 of the largest one.
HL_INLINE void exp_lanes(const Lanes* x, Lanes* y) {
  // ln2 in two parts (Cody and Waite): rounded to f32, so that its product with a whole number below 2^29 is exact, and the rest
  constexpr double kLog2e = 1.4426950408889634074, kLn2Hi = 0.693147182464599609375, kLn2Lo = -1.904654299957768e-09;
  constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer in the low bits
  const Words tiny = *x < -708.0;
  const Lanes zero = *x * 0.0;
  const Lanes c = (Lanes)(((Words)*x & ~tiny) | ((Words)(zero - 708.0) & tiny));
  const Lanes shifted = c * kLog2e + kShift;
  const Lanes n = shifted - kShift;
  const Lanes r = (c - n * kLn2Hi) - n * kLn2Lo;
  Lanes s = r * (1.0 / 6227020800.0) + 1.0 / 479001600.0;
  s = s * r + 1.0 / 39916800.0;
  s = s * r + 1.0 / 3628800.0;
  s = s * r + 1.0 / 362880.0;
  s = s * r + 1.0 / 40320.0;
  s = s * r + 1.0 / 5040.0;
  s = s * r + 1.0 / 720.0;
  s = s * r + 1.0 / 120.0;
  s = s * r + 1.0 / 24.0;
  s = s * r + 1.0 / 6.0;
  s = s * r + 0.5;
  s = s * r + 1.0;
  s = s * r + 1.0;
  const Lanes scale = (Lanes)(((Words)shifted + 1023) << 52);
  *y = (Lanes)((Words)(s * scale) & ~tiny);
}

// p[i] = e^(x[i] - mx) over n (a multiple of LANES) entries, -inf giving 0; returns their sum
HL_INLINE double exp_sum_body(const double* x, double mx, double* p, size_t n) {
  Lanes sums = {0};
  for (size_t i = 0; i < n; i += LANES) {
    Lanes v, e;
    load_lanes(&v, x + i);
    v -= mx;
    exp_lanes(&v, &e);
    __builtin_memcpy(p + i, &e, sizeof e);
    sums += e;
  }
  double s = 0.0;
  for (int j = 0; j < LANES; ++j) s += sums[j];
  return s;
}
// the largest of n entries (the rest of the last lanes padded with -inf), and whether all n are finite (v - v is 0 then)
HL_INLINE double max_body(const double* x, size_t n, bool* all_finite) {
  const size_t whole = n / LANES * LANES;
  double mx = -INFINITY, zero = 0.0;
  if (whole > 0) {
    Lanes m, z = {0};
    load_lanes(&m, x);
    for (size_t i = 0; i < whole; i += LANES) {
      Lanes v;
      load_lanes(&v, x + i);
      const Words more = v > m;
      m = (Lanes)(((Words)v & more) | ((Words)m & ~more));
      z += v - v;
    }
    for (int j = 0; j < LANES; ++j) { mx = m[j] > mx ? m[j] : mx; zero += z[j]; }
  }
  for (size_t i = whole; i < n; ++i) { mx = x[i] > mx ? x[i] : mx; zero += x[i] - x[i]; }
  *all_finite = zero == 0.0;
  return mx;
}
#define HL_AVX2 __attribute__((target("avx2,fma")))
#define HL_AVX512 __attribute__((target("avx512f,avx512dq,fma")))
double exp_sum_plain(const double* x, double mx, double* p, size_t n) { return exp_sum_body(x, mx, p, n); }
HL_AVX2 double exp_sum_avx2(const double* x, double mx, double* p, size_t n) { return exp_sum_body(x, mx, p, n); }
HL_AVX512 double exp_sum_avx512(const double* x, double mx, double* p, size_t n) { return exp_sum_body(x, mx, p, n); }
double max_plain(const double* x, size_t n, bool* all) { return max_body(x, n, all); }
HL_AVX2 double max_avx2(const double* x, size_t n, bool* all) { return max_body(x, n, all); }
HL_INLINE void divide_body(double* x, double by, size_t n) {
  for (size_t i = 0; i < n; i += LANES) {
    Lanes v;
    load_lanes(&v, x + i);
    v /= by;
    __builtin_memcpy(x + i, &v, sizeof v);
  }
}
void divide_plain(double* x, double by, size_t n) { divide_body(x, by, n); }
HL_AVX512 void divide_avx512(double* x, double by, size_t n) { divide_body(x, by, n); }
HL_AVX512 double max_avx512(const double* x, size_t n, bool* all) { return max_body(x, n, all); }
int vector_level() {
  static const int level = !__builtin_cpu_supports("avx2") || !__builtin_cpu_supports("fma") ? 0
                           : __builtin_cpu_supports("avx512f") && __builtin_cpu_supports("avx512dq") ? 2 : 1;
  return level;
}
double exp_sum(const double* x, double mx, double* p, size_t n) {
  const int level = vector_level();
  return level == 2 ? exp_sum_avx512(x, mx, p, n) : level == 1 ? exp_sum_avx2(x, mx, p, n) : exp_sum_plain(x, mx, p, n);
}
double max_of(const double* x, size_t n, bool* all) {
  const int level = vector_level();
  return level == 2 ? max_avx512(x, n, all) : level == 1 ? max_avx2(x, n, all) : max_plain(x, n, all);
}

// x[i] = src[i] / by; by 1.0 leaves the value as it is
HL_INLINE void widen_body(const float* src, double by, double* x, size_t n) {
  typedef float Narrow __attribute__((vector_size(4 * LANES)));
  const size_t whole = n / LANES * LANES;
  for (size_t i = 0; i < whole; i += LANES) {
    Narrow f;
    __builtin_memcpy(&f, src + i, sizeof f);
    Lanes v = __builtin_convertvector(f, Lanes);
    v /= by;
    __builtin_memcpy(x + i, &v, sizeof v);
  }
  for (size_t i = whole; i < n; ++i) x[i] = (double)src[i] / by;
}
void widen_plain(const float* src, double by, double* x, size_t n) { widen_body(src, by, x, n); }
HL_AVX512 void widen_avx512(const float* src, double by, double* x, size_t n) { widen_body(src, by, x, n); }
// the first index at or after i whose value is larger than `least`; n when there is none (no NaN compares as larger)
HL_INLINE size_t next_above_body(const double* x, size_t i, size_t n, double least) {
  for (; i + 4 * LANES <= n; i += 4 * LANES) {
    Words any = {0};
    for (int u = 0; u < 4; ++u) {
      Lanes v;
      load_lanes(&v, x + i + u * LANES);
      any |= v > least;
    }
    int64_t bits = 0;
    for (int j = 0; j < LANES; ++j) bits |= any[j];
    if (bits) break;
  }
  for (; i < n; ++i)
    if (x[i] > least) break;
  return i;
}
size_t next_above_plain(const double* x, size_t i, size_t n, double least) { return next_above_body(x, i, n, least); }
HL_AVX512 size_t next_above_avx512(const double* x, size_t i, size_t n, double least) { return next_above_body(x, i, n, least); }
HL_INLINE bool finite_body(const float* x, size_t n) {
  typedef int32_t Bits __attribute__((vector_size(64)));
  const size_t whole = n / 16 * 16;
  Bits bad = {0};
  for (size_t i = 0; i < whole; i += 16) {
    Bits b;
    __builtin_memcpy(&b, x + i, sizeof b);
    bad |= (b & 0x7f800000) == 0x7f800000;
  }
  int32_t any = 0;
  for (int j = 0; j < 16; ++j) any |= bad[j];
  for (size_t i = whole; i < n; ++i) any |= !std::isfinite(x[i]);
  return any == 0;
}
bool finite_plain(const float* x, size_t n) { return finite_body(x, n); }
HL_AVX512 bool finite_avx512(const float* x, size_t n) { return finite_body(x, n); }

struct Candidate {
  double value;
  long long token;
};
// the order of a stable sort by descending value: larger first, ties to the lower index, NaN last
bool ranks_before(const Candidate& a, const Candidate& b) {
  if (a.value > b.value) return true;
  if (a.value < b.value) return false;
  const bool an = std::isnan(a.value), bn = std::isnan(b.value);
  if (an != bn) return bn;
  return a.token < b.token;
}

// p[i] = e^(x[i] - max) over the finite entries of x (padded with -inf), 0 elsewhere, and their sum; false when none is
// finite
bool softmax(const double* x, size_t n, size_t padded, double* p, double* sum) {
  bool all;
  double mx = max_of(x, n, &all);
  if (!all) {
    mx = -INFINITY;
    for (size_t i = 0; i < n; ++i)
      if (std::isfinite(x[i]) && x[i] > mx) mx = x[i];
  }
  if (mx == -INFINITY) {
    for (size_t i = 0; i < n; ++i) p[i] = 0.0;
    *sum = 1.0;
    return false;
  }
  *sum = exp_sum(x, mx, p, padded);
  if (!all) {  // infinities and NaNs carry no probability
    *sum = 0.0;
    for (size_t i = 0; i < n; ++i) {
      if (!std::isfinite(x[i])) p[i] = 0.0;
      *sum += p[i];
    }
  }
  if (*sum == 0.0) *sum = 1.0;
  return true;
}

// the last maximal index, comparing as the reference's max_by does (a NaN wins over what stands before it)
size_t last_argmax(const double* x, size_t n) {
  bool all;
  const double mx = max_of(x, n, &all);
  if (all) {
    size_t i = n - 1;
    while (x[i] != mx) --i;
    return i;
  }
  size_t best = 0;
  for (size_t i = 1; i < n; ++i)
    if (!(x[i] < x[best])) best = i;
  return best;
}

// The smallest prefix of the ranked candidates whose values add up to `mass`, zeros left out, moved to the front; returns
// its length.  Partitions by rank and keeps the half in which the mass is reached, so no full sort.
size_t ranked_prefix(std::vector<Candidate>& c, double mass) {
  size_t lo = 0, hi = c.size();
  double before = 0.0;  // mass of [0, lo), all of which stays
  while (hi - lo > 64) {
    Candidate a = c[lo], b = c[lo + (hi - lo) / 2], d = c[hi - 1];
    if (ranks_before(b, a)) std::swap(a, b);
    if (ranks_before(d, b)) b = ranks_before(d, a) ? a : d;
    const auto mid = std::partition(c.begin() + lo, c.begin() + hi, [&](const Candidate& x) { return ranks_before(x, b); });
    const size_t m = (size_t)(mid - c.begin());
    double part = 0.0;
    for (size_t i = lo; i < m; ++i) part += c[i].value;
    if (before + part >= mass) {
      hi = m;
    } else {
      before += part;
      // the pivot itself ranks first of the rest: put it there, so that every round shrinks the range
      const auto pivot = std::find_if(c.begin() + m, c.begin() + hi, [&](const Candidate& x) { return x.token == b.token; });
      std::iter_swap(c.begin() + m, pivot);
      if (c[m].value == 0.0) return m;
      before += c[m].value;
      lo = m + 1;
      if (before >= mass) return lo;
    }
  }
  std::sort(c.begin() + lo, c.begin() + hi, ranks_before);
  for (size_t i = lo; i < hi; ++i) {
    if (c[i].value == 0.0) return i;
    before += c[i].value;
    if (before >= mass) return i + 1;
  }
  return hi;
}

}  // namespace
bool all_finite_f32(const float* x, size_t n) { return vector_level() == 2 ? finite_avx512(x, n) : finite_plain(x, n); }

namespace {
int sample_token(const void* logits, int dtype, long long vocab, const int64_t* context, long long n_context, const hl_sampling_options* o,
                 double draw, int64_t* token, double* probability, double* log_probability) {
  HL_REQUIRE(logits && o && token && probability && log_probability && (context || n_context == 0), "hl_sample_token: null argument");
  HL_REQUIRE(vocab > 0 && n_context >= 0, "hl_sample_token: requires at least one logit");
  HL_REQUIRE(dtype == HL_F32 || dtype == HL_F64, "hl_sample_token: logits must be f32 or f64");
  const size_t n = (size_t)vocab, padded = (n + LANES - 1) / LANES * LANES;
  static thread_local std::vector<double> x, p;  // grown to the largest vocabulary seen
  if (p.size() < padded) { x.resize(padded); p.resize(padded); }
  const bool penalties = o->repetition_penalty > 1.0 || o->frequency_penalty != 0.0 || o->presence_penalty != 0.0;
  if (dtype == HL_F32) {  // divided by the temperature on the way when nothing comes between
    const float* src = static_cast<const float*>(logits);
    const double by = !penalties && o->temperature > 0.0 ? o->temperature : 1.0;
    if (vector_level() == 2) widen_avx512(src, by, x.data(), n);
    else widen_plain(src, by, x.data(), n);
  } else {
    const double* src = static_cast<const double*>(logits);
    for (size_t i = 0; i < n; ++i) x[i] = src[i];
  }
  for (size_t i = n; i < padded; ++i) x[i] = -INFINITY;
  if (penalties) {
    std::vector<int64_t> seen(context, context + n_context);  // sorted, so that a token's occurrences stand together
    std::sort(seen.begin(), seen.end());
    HL_REQUIRE(seen.empty() || seen[0] >= 0, "hl_sample_token: negative token id in the context");
    for (size_t i = 0, j; i < seen.size() && seen[i] < vocab; i = j) {
      for (j = i; j < seen.size() && seen[j] == seen[i];) ++j;
      double& v = x[(size_t)seen[i]];
      if (o->repetition_penalty > 1.0) v = v > 0.0 ? v / o->repetition_penalty : v * o->repetition_penalty;
      v -= o->frequency_penalty * (double)(j - i);
      v -= o->presence_penalty;
    }
  }
  if (o->temperature > 0.0 && (penalties || dtype != HL_F32)) {
    if (vector_level() == 2) divide_avx512(x.data(), o->temperature, padded);
    else divide_plain(x.data(), o->temperature, padded);
  }

  // the tokens that stay, in rank order, when a filter is set
  const bool by_k = o->top_k > 0, by_p = o->top_p > 0.0 && o->top_p < 1.0;
  if (by_k || by_p) {
    std::vector<Candidate> kept;
    if (by_k && o->top_k < vocab) {
      const size_t k = (size_t)o->top_k;
      kept.reserve(k + 1);  // a heap whose front is the candidate that ranks last
      for (size_t i = 0; i < k; ++i) kept.push_back(Candidate{x[i], (long long)i});
      std::make_heap(kept.begin(), kept.end(), ranks_before);
      double least = kept.front().value;
      for (size_t i = k; i < n; ++i) {  // a later index loses a tie, so only a larger value (or the first after a NaN) gets in
        if (!std::isnan(least)) {
          i = vector_level() == 2 ? next_above_avx512(x.data(), i, n, least) : next_above_plain(x.data(), i, n, least);
          if (i == n) break;
        } else if (std::isnan(x[i])) {
          continue;
        }
        std::pop_heap(kept.begin(), kept.end(), ranks_before);
        kept.back() = Candidate{x[i], (long long)i};
        std::push_heap(kept.begin(), kept.end(), ranks_before);
        least = kept.front().value;
      }
    } else {
      kept.resize(n);
      for (size_t i = 0; i < n; ++i) kept[i] = Candidate{x[i], (long long)i};
    }
    double sum = 1.0;
    auto by_token = [](const Candidate& a, const Candidate& b) { return a.token < b.token; };
    if (by_p) {
      // probabilities of the kept tokens; the smallest prefix of the ranked ones that reaches the mass stays
      std::vector<double> y((kept.size() + LANES - 1) / LANES * LANES, -INFINITY), q(y.size());
      if (kept.size() < n) std::sort(kept.begin(), kept.end(), by_token);
      for (size_t i = 0; i < kept.size(); ++i) y[i] = kept[i].value;
      const bool any = softmax(y.data(), kept.size(), y.size(), q.data(), &sum);
      for (size_t i = 0; i < kept.size(); ++i)  // no finite logit: all of the mass on index 0
        kept[i].value = any ? q[i] / sum : (kept[i].token == 0 ? 1.0 : 0.0);
      kept.resize(ranked_prefix(kept, o->top_p));
    }
    if (kept.empty()) kept.push_back(Candidate{0.0, (long long)last_argmax(x.data(), n)});
    // everything else is filtered out; what stays is few, so it is worked on by itself, in index order
    if (kept.size() < n / 32) {
      std::sort(kept.begin(), kept.end(), by_token);
    } else {  // a mark per token and one walk instead of a sort
      std::vector<unsigned char> stays(n, 0);
      for (const Candidate& c : kept) stays[(size_t)c.token] = 1;
      size_t at = 0;
      for (size_t i = 0; i < n; ++i)
        if (stays[i]) kept[at++].token = (long long)i;
    }
    const size_t m = kept.size(), mp = (m + LANES - 1) / LANES * LANES;
    std::vector<double> y(mp, -INFINITY), q(mp);
    for (size_t i = 0; i < m; ++i) y[i] = x[(size_t)kept[i].token];
    const bool any = softmax(y.data(), m, mp, q.data(), &sum);
    for (size_t i = 0; i < m; ++i) q[i] /= sum;
    auto answer = [&](long long t, double prob) {
      *token = t;
      *probability = prob;
      *log_probability = std::log(std::max(prob, std::numeric_limits<double>::min()));
      return HL_OK;
    };
    auto greedy = [&]() {
      const size_t best = last_argmax(y.data(), m);
      if (m < n && y[best] == -INFINITY) {  // every token ties at -inf: the last one wins, index 0 holds the mass
        return answer(vocab - 1, vocab == 1 ? 1.0 : 0.0);
      }
      return answer(kept[best].token, any ? q[best] : (kept[best].token == 0 ? 1.0 : 0.0));
    };
    if (o->temperature == 0.0) return greedy();
    if (!any || (draw <= 0.0)) {  // index 0 comes first in the walk, with whatever probability it has
      const double p0 = !any ? 1.0 : kept[0].token == 0 ? q[0] : 0.0;
      if (draw <= p0) return answer(0, p0);
    }
    double cumulative = 0.0;
    for (size_t i = 0; i < m; ++i) {
      cumulative += any ? q[i] : 0.0;
      if (draw <= cumulative) return answer(kept[i].token, q[i]);
    }
    return greedy();
  }

  double sum;
  if (!softmax(x.data(), n, padded, p.data(), &sum)) p[0] = 1.0;
  size_t t = n;
  if (o->temperature != 0.0) {
    double cumulative = 0.0;
    for (size_t i = 0; i < n; ++i) {
      cumulative += p[i] / sum;
      if (draw <= cumulative) { t = i; break; }
    }
  }
  if (t == n) t = last_argmax(x.data(), n);
  const double prob = p[t] / sum;
  *token = (int64_t)t;
  *probability = prob;
  *log_probability = std::log(std::max(prob, std::numeric_limits<double>::min()));
  return HL_OK;
}
}  // namespace
}  // namespace hl

extern "C" int hl_sample_token(const void* logits, int dtype, long long vocab, const int64_t* context, long long n_context,
                               const hl_sampling_options* o, double draw, int64_t* token, double* probability,
                               double* log_probability) {
  try {
    return hl::sample_token(logits, dtype, vocab, context, n_context, o, draw, token, probability, log_probability);
  } catch (const std::exception& e) {  // memory for the row's working copies; callers in C cannot catch it
    return hl::fail(std::string("hl_sample_token: ") + e.what());
  }
}
