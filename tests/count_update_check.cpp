// Count stepping (dust2gpu/count_draws.hpp) against update(), step by
// step: the sir_cases and seir_age systems run from many random
// parameters and states, as FP32 counts and as doubles, from the same
// generators; state and generator must stay equal.  Special-function
// results of the FP32 decisions are moved by their whole error bound, up
// or down at random.  Prints: steps, steps that differ, particles that do
// not fit count stepping.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

static std::uint64_t nudge_state = 88172645463325252ull;
inline float filter_nudge(float units) {
  nudge_state ^= nudge_state << 13;
  nudge_state ^= nudge_state >> 7;
  nudge_state ^= nudge_state << 17;
  return (nudge_state & 1 ? units : -units) * 0x1p-24f;
}
#define DUST2_FILTER_NUDGE(units) filter_nudge(units)

#include "systems/seir_age.hpp"
#include "systems/sir.hpp"
#include "systems/sir_cases.hpp"

using namespace dust2gpu;

static unsigned long long steps, wrong, unfit;

template <typename T>
void run(const typename T::shared_state& shared, const double* start,
         int n_state, double dt, int n_steps, random::rng_state rng) {
  constexpr int size = count_size_of<T>();
  alignas(16) float cells[size] = {};
  const strided_counts c{cells, 1, 0};
  double x[T::n_state_max] = {}, y[T::n_state_max], g[T::n_state_max];
  for (int s = 0; s < n_state; ++s) {
    g[s] = x[s] = start[s];
  }
  bool ok = shared.counts.ready(dt);
  if constexpr (has_count_layout<T>::value) {
    ok = ok && T::count_load(g, c);
  } else {
    for (int s = 0; s < n_state; ++s) {
      ok = ok && random::filter::count_of(x[s], &c[s]);
    }
    ok = ok && T::count_fits(c);
  }
  if (!ok) {
    ++unfit;
    return;
  }
  typename T::internal_state internal{};
  random::rng_state a = rng, b = rng;
  for (int i = 0; i < n_steps; ++i) {
    T::count_update(i * dt, dt, c, shared, a);
    T::update(i * dt, dt, x, shared, internal, b, y);
    if constexpr (has_count_layout<T>::value) {
      if (i % 3 != 1) {  // stored after every step or after two
        T::count_store(g, c);
      }
    } else {
      for (int s = 0; s < n_state; ++s) {
        g[s] = random::filter::count_to_double(c[s]);
      }
    }
    bool same = true;
    for (int s = 0; s < n_state; ++s) {
      x[s] = y[s];
      same = same && (i % 3 == 1 ||
                      math::bits_of(g[s]) == math::bits_of(x[s]));
    }
    for (int w = 0; w < 4; ++w) {
      same = same && a.state[w] == b.state[w];
    }
    ++steps;
    if (!same) {
      ++wrong;
      return;
    }
  }
}

int main(int argc, char** argv) {
  const int n_cases = argc > 1 ? std::atoi(argv[1]) : 2000;
  std::uint64_t words[4];
  random::seed_state(argc > 2 ? std::atoi(argv[2]) : 1, words);
  random::rng_state r{};
  for (int w = 0; w < 4; ++w) {
    r.state[w] = words[w];
  }
  auto uni = [&](double lo, double hi) {
    return lo + (hi - lo) * random::random_real(r);
  };
  for (int i = 0; i < n_cases; ++i) {
    const double dt = i % 3 == 0 ? 1 : i % 3 == 1 ? 0.25 : uni(0.01, 2);
    const double n = std::floor(std::exp(uni(1, 16.7)));
    const double beta = i % 17 == 0 ? 0 : uni(0.01, 3);
    const double gamma = i % 13 == 0 ? uni(0.7, 4) : uni(0.01, 0.7);
    const double infected = std::floor(n * uni(0, 1) * uni(0, 1));
    {
      const double pars[] = {1, n, beta, gamma, 1e6};
      const auto s0 = systems::sir::build_shared(pars);
      auto s1 = s0;
      systems::sir::count_prepare(s1, dt);
      const double start[] = {n - infected, infected, 0, 3, 7};
      run<systems::sir>(s1, start, 5, dt, 60, r);
    }
    {
      const double pars[] = {1, n, beta, gamma};
      auto s = systems::sir_cases::build_shared(pars);
      systems::sir_cases::count_prepare(s, dt);
      const double start[] = {n - infected, infected, 0, 0};
      run<systems::sir_cases>(s, start, 4, dt, 60, r);
    }
    if (i % 8 == 0) {
      double pars[5 + 16 + 256];
      pars[0] = uni(0.5, 6);
      pars[1] = uni(0.05, 0.9);
      pars[2] = uni(0.05, 0.9);
      pars[3] = 20;
      pars[4] = 1;
      for (int a = 0; a < 16; ++a) {
        pars[5 + a] = std::floor(std::exp(uni(3, 16)));
      }
      for (int a = 0; a < 256; ++a) {
        // entries over several orders of magnitude, some zero
        pars[21 + a] = i % 16 == 0 && a % 3 == 0 ? 0 : std::exp(uni(-12, 0));
      }
      auto s = systems::seir_age::build_shared(pars);
      systems::seir_age::count_prepare(s, dt);
      double start[96] = {};
      for (int a = 0; a < 16; ++a) {
        start[a] = std::floor(pars[5 + a] * 0.8);
        start[16 + a] = std::floor(pars[5 + a] * 0.1 * uni(0, 1));
        start[32 + a] = i % 32 == 0 && a != 5 ? 0 :
          std::floor(pars[5 + a] * 0.1 * uni(0, 1));
      }
      run<systems::seir_age>(s, start, 96, dt, 60, r);
    }
    for (int k = 0; k < 7; ++k) {
      random::next(r);
    }
  }
  std::printf("%llu %llu %llu\n", steps, wrong, unfit);
  return 0;
}
