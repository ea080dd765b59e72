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
// ms, one SIR filter of 1000 particles 5.98 -> 3.36 ms.
//
// Error bounds, in units of e = 2^-24 (half an FP32 ulp, relative): every
// FP32 operation adds 1 e; rcp and sqrt of the special function unit add
// 2 e, ex2 4 e, and lg2 4 e absolute for arguments in (1/2, 2) and 4 e
// relative elsewhere (the PTX manual's bounds).  The FP64 side's own
// rounding (at most 5e-7 in the acceptance test, where log k! reaches
// 2.7e8) is inside the constant terms.  tests/binomial_filter_check.cu
// measures both sides.
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

// A count as the filter takes it: an integer in [1, 2^24), exact in FP32.
DUST2_HD bool count_of(double n, float* out) {
  const std::uint64_t u = math::bits_of(n);
  const std::uint32_t hi = static_cast<std::uint32_t>(u >> 32);
  const std::uint32_t lo = static_cast<std::uint32_t>(u);
  // exponent rebias: the FP32 bits are (u >> 29) without the three top
  // exponent bits that a value in range has as 100 or 011
  const float f = math::float_from_bits(((hi << 3) | (lo >> 29)) +
                                        0x40000000u);
  *out = f;
  return hi - 0x3ff00000u < 0x01800000u && (lo & 0x1fffffffu) == 0 &&
    std::trunc(f) == f;
}

// An integer in [0, 2^24) as a double.
DUST2_HD double count_to_double(int k) {
  const std::uint32_t f = math::float_bits_of(static_cast<float>(k));
  const std::uint32_t hi = k == 0 ? 0u : (f >> 3) + 0x38000000u;
  return math::from_bits((static_cast<std::uint64_t>(hi) << 32) |
                         static_cast<std::uint32_t>(f << 29));
}

// A probability in [2^-60, 1/2] as the filter takes it.
struct prob {
  float p;           // 1 e
  float l;           // -log(1 - p), 9 e
  std::uint32_t hi;  // floor(p 2^62) = hi 2^31 + lo, lo < 2^31
  std::uint32_t lo;
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
  return q;
}

// m 2^-53 in FP32 for m < 2^53: 2 e.
DUST2_HD float unit32(std::uint64_t m) {
  const float hi = static_cast<float>(static_cast<std::uint32_t>(m >> 21));
  const float lo =
    static_cast<float>(static_cast<std::uint32_t>(m) & 0x1fffffu);
  return std::fmaf(hi, 0x1p-32f, lo * 0x1p-53f);
}

// BINV: the least x with U <= F(x) = f(0) + ... + f(x), f(0) = exp(-t),
// t = n l, f(x) = f(x-1) s (n + 1 - x) / x, s = p / (1 - p).
//   f(0): t has 10 e relative, the exponent's rounding 2 e more, ex2 4 e:
//         12 t e + 4 e.  A factor adds at most 10 e (s 5 e, its
//         reciprocal 2 e, three products).
//   F(x): the sum over j <= x of f(j) (12 t + 4 + 10 j) e is at most
//         (12 t + 4 + 10 n p) e, with n p <= t; each addition rounds by
//         at most e / 2 (F < 1), and U by e.
// So |F - FP64| <= (22 t + 8 + x) e, and the walk stops for certain when
// U is farther than that from F(x) on both sides.  Returns x, or -1.
DUST2_HD int inversion(rng_state& rng, float n, const prob& q, float t) {
  const rng_state keep = rng;
  const float u = unit32(next(rng) >> 11);
  const float s = q.p * rcp32(1.0f - q.p);
  float f = ex2_32(-LOG2E * t);
  float cum = f;
  float band = std::fmaf(22 * E, t, 8 * E);
  float x = 0;
  float left = n;  // n + 1 - x of the next factor, exact
  while (u > cum + band && x < 100.0f) {
    x += 1.0f;
    f *= s * left * rcp32(x);
    left -= 1.0f;
    cum += f;
    band += E;
  }
  if (u < cum - band) {
    return static_cast<int>(x);
  }
  for (int w = 0; w < 4; ++w) {
    rng.state[w] = keep.state[w];
  }
  return -1;
}

// h(x) = (x! e^x / x^x)^2 / (2 pi), so that log x! = x log x - x +
// log(2 pi h(x)) / 2 for every x >= 0: the values for x < 16, then
// Stirling's series x + 1/6 + 1/(72 x) - 31/(6480 x^2) (the next term is
// below 2e-8 relative).  5 e.
#define DUST2_STIRLING_H                                                   \
  0x1.45f306p-3f, 0x1.2d0ea6p+0f, 0x1.1610ecp+1f, 0x1.95db22p+1f,          \
  0x1.0ade86p+2f, 0x1.4ad4f8p+2f, 0x1.8ace5ep+2f, 0x1.cac98ap+2f,          \
  0x1.0562eep+3f, 0x1.25617cp+3f, 0x1.456050p+3f, 0x1.655f5ap+3f,          \
  0x1.855e8ap+3f, 0x1.a55ddap+3f, 0x1.c55d42p+3f, 0x1.e55cbep+3f
#if defined(__CUDACC__)
__device__ const float stirling_h_dev[16] = {DUST2_STIRLING_H};
#endif
inline const float stirling_h_host[16] = {DUST2_STIRLING_H};

DUST2_HD float stirling_h(float x) {
  if (x < 16.0f) {
#if defined(__CUDA_ARCH__)
    return stirling_h_dev[static_cast<int>(x)];
#else
    return stirling_h_host[static_cast<int>(x)];
#endif
  }
  const float r = rcp32(x);
  return x + std::fmaf(std::fmaf(-31.0f / 6480, r, 1.0f / 72), r, 1.0f / 6);
}

// x log(x / m) - d for x = m + d >= 0, m > 0: with v = d / (x + m) it is
// d v + 2 x (v^3/3 + v^5/5 + ...), without cancellation for |v| < 1/4
// (through v^13; 20 e relative), and directly otherwise (100 e relative:
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

// BTRS for n p > 10.  With c = n p + 1/2 = ci + cf (in integers, cf to
// 2^-31):
//   g = (2 a / us + b) u and y = cf + g, k = ci + floor(y).  spq has
//   5 e, b 7 e, a = 0.01 p + 0.0248 b - 0.0873 > 0.08 loses at most a
//   factor 2.1 and has 20 e, t = 2 a / us 25 e, so y has
//   |u| (30 t + 12 b) e, from u (absolute 2^-32) b e, from cf 2 e: the
//   floor is certain when y is farther than that from an integer.
//   us >= 0.07 is decided on the integers exactly; v <= v_r,
//   v_r = 0.92 - 4.2 / b with 4.2 / b < 0.62: 10 e.
//   The acceptance test's left side log(v alpha / (a / us^2 + b)): 50 e,
//   and lg2's 4 e max(1, |lg2|).  Its right side is log f(k) - log f(m),
//   m = floor((n + 1) p) the mode, f the binomial probabilities: the
//   FP64 sampler forms it from table entries of log k!, here it is
//     -[D(k) - D(m)] + 1/2 log(h(m) h(n - m) / (h(k) h(n - k))),
//     D(x) = deviance(x, n p) + deviance(n - x, n q)
//   (log x! by h; the linear terms of the two deviances cancel), which
//   has no large terms: 100 e D(k) + 20 e D(m) + 30 e.  Where (n + 1) p
//   rounds to the other side of an integer, f(m) is the same to 2^-24.
// Returns k, or -1 when undecided (the generator is then at the undecided
// attempt's first uniform).
DUST2_HD int btrs(rng_state& rng, float n, const prob& q, float np) {
  const std::uint32_t ni = static_cast<std::uint32_t>(n);
  const std::uint64_t c31 = static_cast<std::uint64_t>(ni) * q.hi +
    ((static_cast<std::uint64_t>(ni) * q.lo) >> 31) + (1u << 30);
  const int ci = static_cast<int>(c31 >> 31);
  const float cf =
    static_cast<float>(static_cast<std::uint32_t>(c31) & 0x7fffffffu) *
    0x1p-31f;
  const float spq = sqrt32(np * (1.0f - q.p));
  const float b = std::fmaf(2.53f, spq, 1.15f);
  const float a = std::fmaf(0.01f, q.p, std::fmaf(0.0248f, b, -0.0873f));
  const float inv_b = rcp32(b);
  const float v_r = std::fmaf(-4.2f, inv_b, 0.92f);
  const float y_band = std::fmaf(b, 2 * E, 4 * E);
  constexpr std::uint64_t US_SQUEEZE = 0x23d70a3d70a3eull;  // 0.07 2^53, up
  constexpr std::uint64_t HALF = static_cast<std::uint64_t>(1) << 52;
  for (int attempt = 0; attempt < 1000; ++attempt) {
    const rng_state keep = rng;
    const std::uint64_t mu = next(rng) >> 11;
    const float v = unit32(next(rng) >> 11);
    const bool neg = mu < HALF;
    const std::uint64_t ad = neg ? HALF - mu : mu - HALF;
    const std::uint64_t us53 = HALF - ad;  // us 2^53; 0 when U = 0
    if (us53 == 0) {
      continue;
    }
    const float au =
      static_cast<float>(static_cast<std::uint32_t>(ad >> 21)) * 0x1p-32f;
    const float inv_us = rcp32(unit32(us53));
    const float t = 2.0f * a * inv_us;
    const float g = (t + b) * au;
    const float y = cf + (neg ? -g : g);
    const float band_y = std::fmaf(au, std::fmaf(30 * E, t, 12 * E * b),
                                   y_band);
    const float fl = std::floor(y);
    const float frac = y - fl;
    if (frac > band_y && frac < 1.0f - band_y) {
      const int k = ci + static_cast<int>(fl);
      const bool squeeze = us53 >= US_SQUEEZE;
      if (squeeze && v < v_r - 12 * E) {
        return k;
      }
      if (!squeeze || v > v_r + 12 * E) {
        const float kf = static_cast<float>(k);
        if (kf < 0.0f || kf > n) {
          continue;
        }
        const float alpha = std::fmaf(5.1f, inv_b, 2.83f) * spq;
        const float lhs =
          lg2_32(v * alpha * rcp32(std::fmaf(a * inv_us, inv_us, b)));
        const float nq = n - np;
        const float fm = std::floor(cf - 0.5f + q.p);
        const float m = static_cast<float>(ci) + fm;
        const float dk = fl + (0.5f - cf);
        const float dm = fm + (0.5f - cf);
        const float d_k = deviance(kf, np, dk) + deviance(n - kf, nq, -dk);
        const float d_m = deviance(m, np, dm) + deviance(n - m, nq, -dm);
        const float lg_h =
          lg2_32(stirling_h(m) * stirling_h(n - m) *
                 rcp32(stirling_h(kf) * stirling_h(n - kf)));
        // left side minus right side
        const float diff = std::fmaf(LN2, std::fmaf(-0.5f, lg_h, lhs),
                                     d_k - d_m);
        const float band = std::fmaf(
          100 * E, d_k, std::fmaf(4 * E, std::fabs(lhs) + std::fabs(lg_h),
                                  112 * E));
        if (diff < -band) {
          return k;
        }
        if (diff > band) {
          continue;
        }
      }
    }
    for (int w = 0; w < 4; ++w) {
      rng.state[w] = keep.state[w];
    }
    return -1;
  }
  return -1;
}

// Binomial(n, p) for a count n (nf in FP32) and a probability p <= 1/2;
// -1 when undecided.  The FP64 product selects the sampler where the FP32
// one (2 e) is too close to 10.
DUST2_HD int binomial(rng_state& rng, double n, double p, float nf,
                      const prob& q) {
  const float np = nf * q.p;
  const bool small = std::fabs(np - 10.0f) > 10.0f * 8 * E ?
    np < 10.0f : n * p < 10.0;
  return small ? inversion(rng, nf, q, nf * q.l) : btrs(rng, nf, q, np);
}

}  // namespace filter
}  // namespace random
}  // namespace dust2gpu
