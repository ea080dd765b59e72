// Decided binomial draws whose probability is only known to within `rel`
// (dust2gpu/binomial_filter.hpp), and SEIR steps on counts whose hazards are
// such (systems/seir_age.hpp).
//
//   draws N SEED   filter::binomial with the probability moved by its whole
//                  rel, up and down, against the FP64 sampler at the
//                  probability itself: rel from 2^-29 to 1e-3, n p from 1 to
//                  1000.  Prints: draws, undecided draws with rel at most
//                  2^-24, disagreements.
//   seir N SEED    one step of seir_age with infected in one age only, by
//                  count_update and by update(): contact with an age without
//                  infected up to 10^7.6 times as strong, so that the table
//                  holds the infected age's coefficient to few bits, rounded
//                  by nearly half a unit.  Prints: steps, 0, steps that
//                  differ in state or generator.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "systems/seir_age.hpp"

using namespace dust2gpu;

static double between(random::rng_state& r, double lo, double hi) {
  return lo + (hi - lo) * random::random_real(r);
}

static bool same_state(const random::rng_state& a,
                       const random::rng_state& b) {
  return std::memcmp(a.state, b.state, sizeof(a.state)) == 0;
}

static void draws(int n_draws, random::rng_state r) {
  unsigned long long total = 0, undecided = 0, wrong = 0;
  const double rels[] = {0x1p-29, 0x1p-24, 0x1p-22, 1e-6, 1e-5, 1e-4, 1e-3};
  for (double rel : rels) {
    for (int sign = -1; sign <= 1; sign += 2) {
      for (int i = 0; i < n_draws; ++i) {
        const double mean = std::exp(between(r, 0, std::log(1000.0)));
        const double n = std::floor(std::exp(between(
          r, std::log(4 * mean + 1), std::log(16777215.0))));
        const double p = mean / n;
        auto q = random::filter::make_prob(p * (1 + sign * rel));
        q.rel = static_cast<float>(1.000001 * rel);
        random::rng_state a = r, b = r;
        const float k = random::filter::binomial(
          a, static_cast<float>(n), q, [] { return -1; });
        const double want = random::binomial_fp64(b, n, p);
        ++total;
        if (k < 0.0f) {
          undecided += rel <= 0x1p-24;
        } else {
          wrong += !(static_cast<double>(k) == want && same_state(a, b));
        }
        r = b;
      }
    }
  }
  std::printf("%llu %llu %llu\n", total, undecided, wrong);
}

static void seir(int n_steps, random::rng_state r) {
  using systems::seir_age;
  unsigned long long total = 0, wrong = 0;
  for (double units : {100.0, 300.0, 1000.0, 6433.0, 1e5, 1e7}) {
    double pars[5 + 16 + 256] = {};
    pars[0] = 2;
    pars[1] = 0.2;
    pars[2] = 0.1;
    pars[3] = 20;
    for (int a = 0; a < 16; ++a) {
      pars[5 + a] = 1.5e7;
      pars[21 + 17 * a] = 1;
    }
    auto s = seir_age::build_shared(pars);
    const double dt = 0.25, infected = 1e6, susceptible = 1.4e7;
    // contact that gives a coefficient (hazard of a step per infected) of w
    auto contact = [&](int b, double w) {
      return w / (s.beta * s.inv_N[b] * dt);
    };
    for (int a = 0; a < 16; ++a) {
      for (int b = 0; b < 16; ++b) {
        s.contact[a][b] = a == b ? contact(b, 1e-4) : 0;
      }
    }
    // age 1: a mean of 40 infections a step from the infected of age 0; age
    // 2 sets the unit
    const double top = 40 / (susceptible * infected) * 4294967296.0 / units;
    s.contact[1][1] = 0;
    s.contact[1][2] = contact(2, top);
    int e = 0;
    std::frexp(top, &e);
    const double unit = std::ldexp(1.0, e - 32);
    const double whole = std::floor(units * top * 0x1p-32 / unit);
    for (double off : {0.49, 0.51}) {
      s.contact[1][0] = contact(0, (whole + off) * unit);
      seir_age::count_prepare(s, dt);
      if (!s.counts.ready(dt)) {
        std::printf("not steppable as counts\n");
        std::exit(1);
      }
      for (int i = 0; i < n_steps; ++i) {
        double x[96] = {}, g[96];
        x[1] = susceptible;
        x[32] = infected;
        std::memcpy(g, x, sizeof(x));
        alignas(16) float cells[seir_age::count_size] = {};
        const strided_counts c{cells, 1, 0};
        if (!seir_age::count_load(g, c)) {
          std::printf("not counts\n");
          std::exit(1);
        }
        random::rng_state a = r, b = r;
        seir_age::internal_state internal{};
        seir_age::count_update(0, dt, c, s, a);
        seir_age::count_store(g, c);
        seir_age::update(0, dt, x, s, internal, b, x);
        ++total;
        wrong += !(std::memcmp(g, x, sizeof(x)) == 0 && same_state(a, b));
        r = b;
      }
    }
  }
  std::printf("%llu 0 %llu\n", total, wrong);
}

int main(int argc, char** argv) {
  if (argc != 4) {
    return 2;
  }
  std::uint64_t words[4];
  random::seed_state(std::atoi(argv[3]), words);
  random::rng_state r{};
  std::memcpy(r.state, words, sizeof(words));
  if (std::strcmp(argv[1], "draws") == 0) {
    draws(std::atoi(argv[2]), r);
  } else {
    seir(std::atoi(argv[2]), r);
  }
  return 0;
}
