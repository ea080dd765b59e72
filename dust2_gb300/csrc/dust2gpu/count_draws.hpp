// Binomial draws between counts held in FP32.
//
// The states of the stochastic compartment models are counts: integers,
// which FP32 holds exactly below 2^24.  A system may step them as FP32
// counts (system.hpp, count_update): the additions are then exact FP32
// ones and the draws' probabilities are formed in integers, so that a
// step needs no FP64 instruction.  What FP64 would compute is what is
// returned: the probability only enters through the decisions of
// binomial_filter.hpp, its distance from the FP64 probability is part of
// their bounds, and an undecided draw takes the FP64 probability and the
// FP64 sampler.
#pragma once

#include <cmath>
#include <cstdint>

#include "binomial_filter.hpp"
#include "common.hpp"
#include "distributions.hpp"
#include "math.hpp"
#include "random.hpp"

namespace dust2gpu {
namespace random {

// All counts of a step stay below this, so every sum is exact.
constexpr float COUNT_LIMIT = 16777216.0f;

// binomial(), compiled once per kernel: the rare way out of a count step.
DUST2_SAMPLER double binomial_call(rng_state& rng, double n, double p) {
  return binomial(rng, n, p);
}

DUST2_HD float binomial_count_fp64(rng_state& rng, float n, double p) {
  rng_state r = rng;
  const double x = binomial_call(r, filter::count_to_double(n), p);
  rng = r;
  return static_cast<float>(x);
}

// The probability of one draw: decided draws use q; where q is not usable
// the draw takes the FP64 probability at once.
struct draw_prob {
  filter::prob q;  // min(p, 1 - p)
  bool usable;
  bool zero;       // p is 0
  bool flip;       // p > 1/2
};

// A probability that is the same for every particle of a group, made on
// the host.
struct count_prob {
  draw_prob d;
  double p;
  bool ok;
};

inline count_prob make_count_prob(double p) {
  count_prob c{};
  c.p = p;
  c.d.zero = p == 0;
  c.d.flip = p > 0.5;
  const double pp = c.d.flip ? 1.0 - p : p;
  c.d.usable = p < 1 && pp >= 0x1p-60;
  c.ok = c.d.zero || c.d.usable;
  if (c.d.usable) {
    c.d.q = filter::make_prob(pp);
  }
  return c;
}

// binomial(rng, n, exact()) for a count n and its probability d.  A system
// with several draws per step makes them in a loop over one call of this:
// the sampler is a few hundred instructions, and one copy of it left SEIR
// at 5 blocks per SM without spilling around it (three copies 75.9 ms).
template <typename F>
DUST2_HD float draw_count(rng_state& rng, float n, const draw_prob& d,
                          const F& exact) {
  if (n == 0.0f || d.zero) {
    return 0.0f;
  }
  if (d.usable) {
    // n p too close to 10 to choose the sampler: undecided
    const float k = filter::binomial(rng, n, d.q, [] { return -1; });
    if (k >= 0.0f) {
      return d.flip ? n - k : k;
    }
  }
  return binomial_count_fp64(rng, n, exact());
}

DUST2_HD std::uint32_t mul_hi32(std::uint32_t a, std::uint32_t b) {
  return static_cast<std::uint32_t>((static_cast<std::uint64_t>(a) * b) >>
                                    32);
}

// 1 - exp(-x), x = x62 2^-62 in [2^-40, 1/2): x - x h(x),
// h = x/2! - x^2/3! + ... - x^9/10! by Horner's rule in units of 2^-32
// (the next term is below 2^-35; each product is cut to 2^-32, so h is
// within 3 2^-32 and 1 - exp(-x) within 2^-29 of itself).  -log(1 - p) is
// x.  About 40 integer instructions, against some 15 FP64 ones and the
// integer exp.
DUST2_HD filter::prob hazard_prob(std::uint64_t x62, float rel) {
  const std::uint32_t x32 = static_cast<std::uint32_t>(x62 >> 30);
  std::uint32_t h = 1184u;           // 2^32 / 10!
  h = 11836u - mul_hi32(x32, h);     // 2^32 / 9!
  h = 106522u - mul_hi32(x32, h);    // 2^32 / 8!
  h = 852176u - mul_hi32(x32, h);    // 2^32 / 7!
  h = 5965233u - mul_hi32(x32, h);   // 2^32 / 6!
  h = 35791394u - mul_hi32(x32, h);  // 2^32 / 5!
  h = 178956971u - mul_hi32(x32, h);
  h = 715827883u - mul_hi32(x32, h);
  h = 2147483648u - mul_hi32(x32, h);
  h = mul_hi32(x32, h);
  const std::uint32_t xh = static_cast<std::uint32_t>(x62 >> 31);
  const std::uint32_t xl = static_cast<std::uint32_t>(x62) & 0x7fffffffu;
  const std::uint64_t p62 = x62 -
    ((static_cast<std::uint64_t>(xh) * h) >> 1) - mul_hi32(xl, h);
  filter::prob q;
  q.hi = static_cast<std::uint32_t>(p62 >> 31);
  q.lo = static_cast<std::uint32_t>(p62) & 0x7fffffffu;
  q.p = std::fmaf(static_cast<float>(q.hi), 0x1p-31f,
                  static_cast<float>(q.lo) * 0x1p-62f);
  q.l = std::fmaf(static_cast<float>(xh), 0x1p-31f,
                  static_cast<float>(xl) * 0x1p-62f);
  q.rel = rel + 0x1p-29f;
  return q;
}

// 1 - exp(-x), x within (rel x) of x62 2^-62.  (FP64's own rounding of the
// probability, 2^-53 absolute, moves n p by less than 2^-29.)  A hazard
// outside [2^-40, 1/2) is not usable.
DUST2_HD draw_prob hazard_draw(std::uint64_t x62, float rel) {
  draw_prob d;
  d.usable = x62 - (1ull << 22) < (1ull << 61) - (1ull << 22);
  d.zero = false;
  d.flip = false;
  d.q = hazard_prob(x62, rel);
  return d;
}

}  // namespace random
}  // namespace dust2gpu
