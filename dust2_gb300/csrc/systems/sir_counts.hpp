// The two transitions of the SIR systems between FP32 counts
// (dust2gpu/count_draws.hpp): n_SI ~ Bin(S, 1 - exp(-beta I / N dt)) and
// n_IR ~ Bin(I, 1 - exp(-gamma dt)), drawn in that order.
#pragma once

#include <cmath>

#include "../dust2gpu/system.hpp"

namespace dust2gpu {
namespace systems {

struct sir_counts {
  std::uint64_t key_dt;
  std::uint64_t rate62;  // beta dt / N in units of 2^-62: 2^-32 relative
  random::count_prob recover;
  math::divisor by_N;
  double exp_gamma;      // exp(-gamma)
  bool ok;

  void prepare(double N, double beta, double gamma, double dt) {
    key_dt = math::bits_of(dt);
    by_N = math::divisor::of(N);
    exp_gamma = math::exp(-gamma);
    const double rate = beta * dt / N;
    recover = random::make_count_prob(1 - math::exp(-gamma * dt));
    ok = recover.ok && N > 0 && rate >= 0x1p-30 && rate < 1;
    rate62 = ok ? static_cast<std::uint64_t>(std::ldexp(rate, 62)) : 0;
  }

  // Prepared for this dt; ready: and the counts can be stepped.
  DUST2_HD bool prepared(double dt) const {
    return key_dt == math::bits_of(dt);
  }
  DUST2_HD bool ready(double dt) const {
    return ok && prepared(dt);
  }

  // I < 2^24 and rate < 1: a hazard of 4 or more would wrap, so it is
  // bounded in FP32 first (any hazard of 1/2 or more takes the FP64
  // probability).
  DUST2_HD void draw(random::rng_state& rng, float S, float I, double N,
                     double beta, double dt, float* n_SI,
                     float* n_IR) const {
    const std::uint32_t rate_hi = static_cast<std::uint32_t>(rate62 >> 38);
    const std::uint64_t x62 =
      I * (static_cast<float>(rate_hi) + 1.0f) < 0x1p24f ?
      static_cast<std::uint32_t>(I) * rate62 : ~0ull;
    random::draw_prob d = random::hazard_draw(x62, 0.0f);
    d.zero = I == 0.0f;
    float n = S;
    float first = 0;
    // the body holds a sampler: one copy for both draws
#pragma unroll 1
    for (int j = 0;; ++j) {
      const float k = random::draw_count(rng, n, d, [&] {
        return j == 0 ? p_SI(I, N, beta, dt) : recover.p;
      });
      if (j == 1) {
        *n_SI = first;
        *n_IR = k;
        return;
      }
      first = k;
      n = I;
      d = recover.d;
    }
  }

  // As update() forms it.
  DUST2_SAMPLER static double p_SI(float I, double N, double beta,
                                   double dt) {
    return 1 - math::exp(-beta * random::filter::count_to_double(I) / N * dt);
  }
};

}  // namespace systems
}  // namespace dust2gpu
