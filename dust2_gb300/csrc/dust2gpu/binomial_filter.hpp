// Binomial draws decided in FP32, with a bound on every decision.
//
// The samplers of distributions.hpp turn uniforms into an integer through
// comparisons only: BINV compares the uniform with cumulative
// probabilities, BTRS takes a floor and compares with a squeeze and an
// acceptance bound.  Their FP64 arithmetic is needed for the rare
// comparison whose two sides nearly agree; everywhere else a few digits
// decide it.  This header evaluates both sides in FP32 (and
// integers for the position n p + 1/2), with a bound on the distance from
// the FP64 evaluation, and takes a decision only when the two sides differ
// by more than the bound.  Otherwise the draw is undecided: the generator
// is left at the attempt's first uniform and the caller runs the FP64
// sampler from there.  A decided draw consumes the same uniforms and
// returns the same integer as the FP64 sampler, always; nothing is
// approximate in the result.
//
// Why: on this GPU one FP64 warp instruction holds an SM partition for 76
// cycles and one FP32 instruction for about 1.2 (measured, 4 warps per
// partition; 64-bit integer multiply-add 6, reciprocal or logarithm unit
// 8), so the FP64 samplers (about 130 FP64 instructions per SIR
// particle-step) were the whole cost of a filter.  Against FP64 draws
// alone, on one GB300: the 64-group batched SIR filter (200 observations)
// 159.0 -> 61.2 ms, 32 x 8192 SEIR particles x 60 observations 297 -> 146
// ms, one SIR filter of 1000 particles 5.98 -> 3.36 ms.  (With the steps on
// counts, count_draws.hpp, and the rest of the step and tail kernels as they
// are now: 33, 67 and 2.4 ms.)
//
// Error bounds, in units of e = 2^-24 (half an FP32 ulp, relative): every
// FP32 operation adds 1 e; rcp and sqrt of the special function unit add
// 2 e, ex2 4 e, and lg2 4 e absolute for arguments in (1/2, 2) and 4 e
// relative elsewhere (the PTX manual's bounds).  The FP64 side's own
// rounding (at most 5e-7 in the acceptance test, where log k! reaches
// 2.7e8) is inside the constant terms.  tests/binomial_filter_check.cu
// compares the draws, with every special-function result moved by its bound.
#pragma once

#include <cmath>
#include <cstdint>

#include "common.hpp"
#include "math.hpp"
#include "random.hpp"

namespace dust2gpu {
namespace random {
namespace filter {

// The special function unit on the device, libm on the host (tests).
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ float rcp32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt32(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float lg2_32(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex2_32(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#else
// DUST2_FILTER_NUDGE(err) lets a test move each result by its bound.
#if !defined(DUST2_FILTER_NUDGE)
#define DUST2_FILTER_NUDGE(units) 0.0f
#endif
inline float rcp32(float x) {
  const float r = 1.0f / x;
  return r + r * DUST2_FILTER_NUDGE(2);
}
inline float sqrt32(float x) {
  const float r = std::sqrt(x);
  return r + r * DUST2_FILTER_NUDGE(2);
}
inline float lg2_32(float x) {
  const float r = std::log2(x);
  return r + (x > 0.5f && x < 2.0f ? 1.0f : r) * DUST2_FILTER_NUDGE(4);
}
inline float ex2_32(float x) {
  const float r = std::exp2(x);
  return r + r * DUST2_FILTER_NUDGE(4);
}
#endif

constexpr float E = 0x1p-24f;
constexpr float LOG2E = 0x1.715476p+0f;
constexpr float LN2 = 0x1.62e430p-1f;

// A count as the filter takes it: an integer in [0, 2^24), exact in FP32.
// (The FP32 bits of a double in [1, 2^24) are bits 29-60 less the three
// top exponent bits' bias.)
DUST2_HD bool count_of(double n, float* out) {
  const std::uint64_t u = math::bits_of(n);
  const std::uint32_t hi = static_cast<std::uint32_t>(u >> 32);
  const std::uint32_t lo = static_cast<std::uint32_t>(u);
  const float f = u == 0 ? 0.0f :
    math::float_from_bits(((hi << 3) | (lo >> 29)) + 0x40000000u);
  *out = f;
  return u == 0 || (hi - 0x3ff00000u < 0x01800000u &&
                    (lo & 0x1fffffffu) == 0 && std::trunc(f) == f);
}

// A count as a double.
DUST2_HD double count_to_double(float k) {
  const std::uint32_t f = math::float_bits_of(k);
  const std::uint32_t hi = f == 0 ? 0u : (f >> 3) + 0x38000000u;
  return math::from_bits((static_cast<std::uint64_t>(hi) << 32) |
                         static_cast<std::uint32_t>(f << 29));
}

// A probability in [2^-60, 1/2] as the filter takes it.  `rel` bounds the
// relative distance of all of these from the FP64 probability, 0 when they
// were made from it.
struct prob {
  float p;           // 2 e
  float l;           // -log(1 - p), 9 e
  std::uint32_t hi;  // p 2^62 = hi 2^31 + lo, lo < 2^31, rounded down
  std::uint32_t lo;
  float rel;
};

// -log(1 - p) = 2 atanh(z), z = p / (2 - p) <= 1/3, by its series through
// z^15 (the next term is below 2e-9 relative): 9 e.
DUST2_HD float neg_log1m(float p) {
  const float z = p * rcp32(2.0f - p);
  const float z2 = z * z;
  float s = 1.0f / 15;
  s = std::fmaf(s, z2, 1.0f / 13);
  s = std::fmaf(s, z2, 1.0f / 11);
  s = std::fmaf(s, z2, 1.0f / 9);
  s = std::fmaf(s, z2, 1.0f / 7);
  s = std::fmaf(s, z2, 1.0f / 5);
  s = std::fmaf(s, z2, 1.0f / 3);
  s = std::fmaf(s, z2, 1.0f);
  return 2.0f * z * s;
}

// The largest `rel` that the bounds below have room for; with a larger one
// (or NaN) every draw is undecided.
constexpr float REL_MAX = 4 * E;

constexpr std::uint64_t BITS_MIN_P = 0x3c30000000000000ull;  // 2^-60

// For 2^-60 <= p <= 1/2 (on the bits).
DUST2_HD prob make_prob(double p) {
  const std::uint64_t u = math::bits_of(p);
  const std::uint64_t r = u + 0x10000000u;  // to nearest, ties up
  const int e = static_cast<int>(u >> 52);  // 963 .. 1022
  const std::uint64_t mant = (u & 0x000fffffffffffffull) |
    0x0010000000000000ull;
  const std::uint64_t p62 = e >= 1013 ? mant << (e - 1013) :
    mant >> (1013 - e);
  prob q;
  q.p = math::float_from_bits(static_cast<std::uint32_t>(r >> 29) +
                              0x40000000u);
  q.l = neg_log1m(q.p);
  q.hi = static_cast<std::uint32_t>(p62 >> 31);
  q.lo = static_cast<std::uint32_t>(p62) & 0x7fffffffu;
  q.rel = 0;
  return q;
}

// BINV: the least x with U <= F(x) = f(0) + ... + f(x), f(0) = exp(-t),
// t = n l, f(x) = f(x-1) s (n + 1 - x) / x, s = p / (1 - p).
//   f(0): t has 10 e relative, the exponent's rounding 2 e more, ex2 4 e:
//         12 t e + 4 e.  A factor adds at most 12 e (s 7 e, the
//         reciprocal 2 e, three products).
//   F(x): the sum over j <= x of f(j) (12 t + 4 + 12 j) e is at most
//         (12 t + 4 + 12 n p) e, with n p <= t; each of at most 40
//         additions rounds by at most e / 2 (F < 1), and U by 2 e.
// So |F - FP64| <= (24 t + 26) e + 2 t rel, and the walk stops for
// certain when U is farther than that from F(x) on both sides.  (With
// n p < 10, x > 40 has probability below 1e-12.)  Returns x, or -1.
DUST2_HD float inversion(rng_state& rng, float n, const prob& q, float t) {
  const float u =
    static_cast<float>(static_cast<std::uint32_t>(next(rng) >> 32)) *
    0x1p-32f;
  const float s = q.p * rcp32(1.0f - q.p);
  float f = ex2_32(-LOG2E * t);
  const float band = std::fmaf(26 * E + 2 * q.rel, t, 28 * E);
  float lower = f - band;  // F(x) - band
  const float width = 2 * band;
  float x = 0;
  float left = n;  // n + 1 - x of the next factor, exact
  while (u > lower + width && x < 40.0f) {
    x += 1.0f;
    f *= s * left * rcp32(x);
    left -= 1.0f;
    lower += f;
  }
  if (u < lower) {
    return x;
  }
  previous(rng.state);
  return -1.0f;
}

// h(x) = (x! e^x / x^x)^2 / (2 pi), so that log x! = x log x - x +
// log(2 pi h(x)) / 2 for every x >= 0: the values for x < 10, then
// Stirling's series x + 1/6 + 1/(72 x) - 31/(6480 x^2) - 139/(155520 x^3)
// (the next term is below 3e-8 relative).  5 e.
#define DUST2_STIRLING_H                                                   \
  0x1.45f306p-3f, 0x1.2d0ea6p+0f, 0x1.1610ecp+1f, 0x1.95db22p+1f,          \
  0x1.0ade86p+2f, 0x1.4ad4f8p+2f, 0x1.8ace5ep+2f, 0x1.cac98ap+2f,          \
  0x1.0562eep+3f, 0x1.25617cp+3f
#if defined(__CUDACC__)
__device__ const float stirling_h_dev[10] = {DUST2_STIRLING_H};
#endif
inline const float stirling_h_host[10] = {DUST2_STIRLING_H};

// x >= 10
DUST2_HD float stirling_h10(float x) {
  const float r = rcp32(x);
  float s = std::fmaf(-139.0f / 155520, r, -31.0f / 6480);
  s = std::fmaf(s, r, 1.0f / 72);
  return x + std::fmaf(s, r, 1.0f / 6);
}

DUST2_HD float stirling_h(float x) {
  if (x < 10.0f) {
#if defined(__CUDA_ARCH__)
    return stirling_h_dev[static_cast<int>(x)];
#else
    return stirling_h_host[static_cast<int>(x)];
#endif
  }
  return stirling_h10(x);
}

// x log(x / m) - d for x = m + d >= 0, m > 0: with v = d / (x + m) it is
// d v + 2 x (v^3/3 + v^5/5 + ...), without cancellation for |v| < 1/4
// (through v^13; 20 e relative), and directly otherwise (112 e relative:
// the value is then at least a tenth of x).  d is given, not formed from
// x and m, so its own error enters relatively.
DUST2_HD float deviance(float x, float m, float d) {
  const float v = d * rcp32(x + m);
  const float v2 = v * v;
  if (v2 < 0.0625f) {
    float s = 1.0f / 13;
    s = std::fmaf(s, v2, 1.0f / 11);
    s = std::fmaf(s, v2, 1.0f / 9);
    s = std::fmaf(s, v2, 1.0f / 7);
    s = std::fmaf(s, v2, 1.0f / 5);
    s = std::fmaf(s, v2, 1.0f / 3);
    return v * std::fmaf(2.0f * x * v2, s, d);
  }
  return x > 0.0f ? std::fmaf(x * LN2, lg2_32(x * rcp32(m)), -d) : -d;
}

// The same for |d| <= 1 and m >= 10, by its series in z = d / m through
// z^6 (the next term is below 3e-8).
DUST2_HD float deviance_near(float m, float d) {
  const float z = d * rcp32(m);
  float s = std::fmaf(1.0f / 30, z, -1.0f / 20);
  s = std::fmaf(s, z, 1.0f / 12);
  s = std::fmaf(s, z, -1.0f / 6);
  s = std::fmaf(s, z, 1.0f / 2);
  return d * z * s;
}

// BTRS for n p >= 10.  With c = n p + 1/2 = ci + cf (in integers, cf to
// 2^-31, n p rel from rel):
//   g = (2 a / us + b) u and y = cf + g, k = ci + floor(y).  spq, the root
//   of n p (1 - p), has half of p's own 2 e and of rel (at most 4 e) and of
//   three roundings, and sqrt's 2 e: 6.5 e; b 8.5 e, and
//   a = 0.01 p + 0.0248 b - 0.0873 > 0.08 loses at most a factor 2.1 and
//   has 23 e.  The uniforms are cut to 32 bits, so us is also known to
//   2^-32 only and t = 2 a / us has 27 e + 2^-32 / us; u's 2^-32 adds less
//   than e b.  So y has |u| ((34 e + 2^-32 / us) t + 14 e b), and from cf
//   2 e: the floor is certain when y is farther than that from an integer.
//   us >= 0.07: certain except for two values of its 32 bits.  v <= v_r,
//   v_r = 0.92 - 4.2 / b with 4.2 / b < 0.62: 12 e.
//   The acceptance test's left side log(v alpha / (a / us^2 + b)): 55 e,
//   from the cut uniforms 2^-32 (2 / us + 1 / v), and lg2's
//   4 e max(1, |lg2|).  Its right side is log f(k) - log f(m),
//   m = floor((n + 1) p) the mode, f the binomial probabilities: the
//   FP64 sampler forms it from table entries of log k!, here it is
//     -[D(k) - D(m)] + 1/2 log(h(m) h(n - m) / (h(k) h(n - k))),
//     D(x) = deviance(x, n p) + deviance(n - x, n q)
//   (log x! by h; the linear terms of the two deviances cancel), which
//   has no large terms: 112 e D(k) + 20 e D(m) + 30 e, and for the two
//   logarithms of the h (at most 48 in base 2) 4 e of the first and 120 e.
//   From rel, f(k) has 2 |k - n p| rel and f(m) 2 rel; where (n + 1) p
//   rounds to the other side of an integer, f(m) has 2.1 rel more: 17 e.
// Returns k, or -1 when undecided (the generator is then at the undecided
// attempt's first uniform).
DUST2_HD float btrs(rng_state& rng, float n, const prob& q, float np) {
  const std::uint32_t ni = static_cast<std::uint32_t>(n);
  const std::uint64_t c31 = static_cast<std::uint64_t>(ni) * q.hi +
    ((static_cast<std::uint64_t>(ni) * q.lo) >> 31) + (1u << 30);
  const float ci = static_cast<float>(static_cast<std::uint32_t>(c31 >> 31));
  const float cf =
    static_cast<float>(static_cast<std::uint32_t>(c31) & 0x7fffffffu) *
    0x1p-31f;
  const float spq = sqrt32(np * (1.0f - q.p));
  const float b = std::fmaf(2.53f, spq, 1.15f);
  const float a = std::fmaf(0.01f, q.p, std::fmaf(0.0248f, b, -0.0873f));
  const float inv_b = rcp32(b);
  // v's bounds, in units of 2^-32 as v is
  const float v_r = std::fmaf(-4.2f * 0x1p32f, inv_b, 0.92f * 0x1p32f);
  const float v_low = v_r - 12 * E * 0x1p32f;
  const float v_high = v_r + 12 * E * 0x1p32f;
  const float y_band = std::fmaf(np, q.rel, std::fmaf(b, E, 4 * E));
  const float a2 = 2.0f * 0x1p32f * a;
  const float b_band = 14 * E * b;
  // the acceptance test's terms that do not depend on the candidate: alpha
  // 2^-32, and -D(m) - 1/2 log(h(m) h(n - m))
  const float alpha = std::fmaf(5.1f, inv_b, 2.83f) * spq * 0x1p-32f;
  const float nq = n - np;
  const float off = 0.5f - cf;
  float mode;
  {
    const float fm = std::floor(q.p - off);
    const float m = ci + fm;
    const float dm = fm + off;
    mode = std::fmaf(
      -0.5f * LN2, lg2_32(stirling_h10(m) * stirling_h10(n - m)),
      -(deviance_near(np, dm) + deviance_near(nq, -dm)));
  }
  for (int attempt = 0; attempt < 1000; ++attempt) {
    const std::uint32_t hu = static_cast<std::uint32_t>(next(rng) >> 32);
    const std::uint32_t hv = static_cast<std::uint32_t>(next(rng) >> 32);
    // u = U - 1/2 in units of 2^-32 (cut), us = 1/2 - |u|
    const bool neg = hu < 0x80000000u;
    const std::uint32_t ad = neg ? 0x80000000u - hu : hu - 0x80000000u;
    const std::uint32_t us = 0x80000000u - ad;
    const float au = static_cast<float>(ad) * 0x1p-32f;
    const float inv_us = rcp32(static_cast<float>(us));  // 2^-32 / us
    const float v = static_cast<float>(hv);
    const float t = a2 * inv_us;
    const float y = std::fmaf(t + b, neg ? -au : au, cf);
    const float band_y = std::fmaf(
      au, std::fmaf(t, inv_us + 34 * E, b_band), y_band);
    const float fl = std::floor(y);
    if (std::fabs(y - fl - 0.5f) < 0.5f - band_y) {
      const float k = ci + fl;
      // 0.07 2^32 = 300647710.72
      const bool squeeze = us >= 300647712u;
      if (squeeze && v < v_low) {
        return k;
      }
      if (us <= 300647709u || (squeeze && v > v_high)) {
        if (k < 0.0f || k > n) {
          continue;
        }
        // a / us^2 = (a2 / 2) (2^32 / us) / us
        const float lhs =
          lg2_32(v * alpha *
                 rcp32(std::fmaf(0.5f * 0x1p32f * t, inv_us, b)));
        const float dk = fl + off;
        const float d_k = deviance(k, np, dk) + deviance(n - k, nq, -dk);
        const float lg_h = lg2_32(stirling_h(k) * stirling_h(n - k));
        // left side minus right side
        const float diff = std::fmaf(LN2, std::fmaf(0.5f, lg_h, lhs),
                                     d_k + mode);
        const float cut = std::fmaf(2.0f, inv_us, rcp32(v));
        const float band = std::fmaf(
          112 * E, d_k, std::fmaf(4 * E, std::fabs(lhs) + std::fabs(lg_h),
                                  240 * E + cut)) +
          2.0f * q.rel * std::fabs(dk);
        if (diff < -band) {
          return k;
        }
        if (diff > band) {
          continue;
        }
      }
    }
    previous(rng.state);
    previous(rng.state);
    return -1.0f;
  }
  return -1.0f;
}

// Binomial(n, p) for a count n >= 1 and a probability p <= 1/2; -1 when
// undecided.  Where n p (3 e) is too close to 10 to choose the sampler,
// small() says whether the FP64 product is below 10 (1 or 0; -1 leaves the
// draw undecided).
template <typename F>
DUST2_HD float binomial(rng_state& rng, float n, const prob& q,
                        const F& small) {
  if (!(q.rel <= REL_MAX)) {
    return -1.0f;
  }
  const float np = n * q.p;
  int inv = np < 10.0f ? 1 : 0;
  if (std::fabs(np - 10.0f) <= 10.0f * (8 * E + q.rel)) {
    inv = small();
    if (inv < 0) {
      return -1.0f;
    }
  }
  return inv ? inversion(rng, n, q, n * q.l) : btrs(rng, n, q, np);
}

}  // namespace filter
}  // namespace random
}  // namespace dust2gpu
