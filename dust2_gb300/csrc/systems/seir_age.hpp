// Age-structured stochastic SEIR with a negative-binomial observation of
// total daily incidence (16 age groups; state S, E, I, R, cases_cumul and
// cases_inc per age, 96 entries).  Written against dust2's plugin
// contract (vignettes/writing.Rmd; structure as inst/examples/sir.cpp):
//   lambda_a = beta sum_b C[a][b] I_b / N_b,   beta = R0 gamma / rho(C)
//   per age a, in this order: n_SE ~ Bin(S_a, 1 - exp(-lambda_a dt)),
//   n_EI ~ Bin(E_a, 1 - exp(-sigma dt)), n_IR ~ Bin(I_a, 1 - exp(-gamma dt))
//   incidence counts n_EI and resets daily;
//   compare: log NegBin(observed | size, mu = sum_a cases_inc_a + 1e-6).
// rho(C) is the spectral radius of the contact matrix, found on the host
// by power iteration when parameters are read.
#pragma once

#include "../dust2gpu/system.hpp"

namespace dust2gpu {
namespace systems {

struct seir_age {
  static constexpr const char* name = "seir_age";
  // update() reads the entries of age a (and, before its loop, every I)
  // before it writes the same entries of state_next, and reads nothing
  // it has written: it is correct in place, so a particle keeps one
  // state array.
  static constexpr bool update_in_place = true;
  // 5 blocks of 128 threads per SM: 96 registers, and 160 KB of shared
  // memory for the counts.  32 groups x 8192 particles, 60 observations:
  // 4 blocks 77.1 ms, 5 72.5, 6 92.5 (the L1 cache that is left no longer
  // holds what 80 registers spill).  All 96 entries as FP32 in local
  // memory (L1 hit rate 49%) 84.0 ms, in shared memory 88.5.
  static constexpr int step_blocks_per_sm = 5;
  // Stepped by update(), the 96 doubles are a thread's own array in local
  // memory: 4 blocks of 128 threads, 128 registers.  Deterministic
  // likelihood of 4096 particles, 60 data times of 4 steps: 33.7 ms; 5
  // blocks 39.2.
  static constexpr int min_blocks_per_sm = 4;
  using real_type = double;
  using rng_state_type = random::rng_state;
  static constexpr int n_age = 16;

  // Count stepping (dust2gpu/count_draws.hpp): the hazard of age a,
  //   beta dt sum_b C[a][b] / N_b I_b,
  // as integers: the row's coefficients in units of 2^-scale with the
  // largest just below 2^32, times the counts.  A coefficient is within
  // half a unit, so the hazard is within sum_b I_b / 2 units.  16 x 16
  // 32 x 32-bit multiply-adds (about 3 cycles a warp each) in place of as
  // many FP64 ones (76 cycles).
  struct count_table {
    std::uint64_t key_dt;
    random::count_prob after[2];  // E to I, I to R
    bool ok;
    int scale[n_age];
    alignas(16) std::uint32_t k[n_age][n_age];

    DUST2_HD bool ready(real_type dt) const {
      return ok && key_dt == math::bits_of(dt);
    }
  };

  struct shared_state {
    real_type beta;
    real_type sigma;
    real_type gamma;
    real_type size;
    real_type R0;
    real_type I0;
    real_type N[n_age];
    real_type inv_N[n_age];
    real_type contact[n_age][n_age];
    count_table counts;
  };
  struct internal_state {};
  struct data_type {
    real_type incidence;
  };

  static constexpr int n_state_max = 6 * n_age;
  static constexpr real_type default_dt = 0.25;

  static constexpr parameter_info parameters[] = {
    {"R0", 1, 2, false, false},
    {"sigma", 1, 0.2, false, false},
    {"gamma", 1, 0.1, false, false},
    {"size", 1, 20, false, true},
    {"I0", 1, 1, false, false},
    {"N", n_age, 62500, false, true},
    {"contact", n_age * n_age, NAN, true, true}};
  static constexpr const char* data_names[] = {"incidence"};

  static real_type spectral_radius(const real_type (&c)[n_age][n_age]) {
    // power iteration; the contact matrix is non-negative
    std::vector<double> x(n_age, 1.0), y(n_age);
    double rho = 0;
    for (int it = 0; it < 1000; ++it) {
      double norm = 0;
      for (int a = 0; a < n_age; ++a) {
        double acc = 0;
        for (int b = 0; b < n_age; ++b) {
          acc += c[a][b] * x[b];
        }
        y[a] = acc;
        norm = std::max(norm, std::fabs(acc));
      }
      if (!(norm > 0)) {
        return 0;
      }
      for (int a = 0; a < n_age; ++a) {
        x[a] = y[a] / norm;
      }
      if (std::fabs(norm - rho) < 1e-14 * norm) {
        rho = norm;
        break;
      }
      rho = norm;
    }
    return rho;
  }

  static void derive(shared_state& s) {
    const double rho = spectral_radius(s.contact);
    s.beta = rho > 0 ? s.R0 * s.gamma / rho : 0;
    for (int a = 0; a < n_age; ++a) {
      s.inv_N[a] = 1.0 / s.N[a];
    }
  }

  static shared_state build_shared(const double* pars) {
    shared_state s{};
    s.R0 = read_par<seir_age>(pars, 0);
    s.sigma = read_par<seir_age>(pars, 1);
    s.gamma = read_par<seir_age>(pars, 2);
    s.size = read_par<seir_age>(pars, 3);
    s.I0 = read_par<seir_age>(pars, 4);
    const double* n = pars + parameter_offset<seir_age>(5);
    for (int a = 0; a < n_age; ++a) {
      s.N[a] = std::isnan(n[0]) ? parameters[5].default_value : n[a];
    }
    read_par_array<seir_age>(pars, 6, &s.contact[0][0], n_age * n_age, true);
    derive(s);
    return s;
  }

  static void update_shared(const double* pars, shared_state& s) {
    s.R0 = read_par_update<seir_age>(pars, 0, s.R0);
    s.sigma = read_par_update<seir_age>(pars, 1, s.sigma);
    s.gamma = read_par_update<seir_age>(pars, 2, s.gamma);
    s.I0 = read_par_update<seir_age>(pars, 4, s.I0);
    derive(s);
  }

  static std::vector<packing_entry> packing_state(const shared_state&) {
    return {{"S", {n_age}}, {"E", {n_age}}, {"I", {n_age}}, {"R", {n_age}},
            {"cases_cumul", {n_age}}, {"cases_inc", {n_age}}};
  }

  static int n_state(const shared_state&) {
    return 6 * n_age;
  }

  static zero_every_spec zero_every(const shared_state&) {
    auto z = zero_every_none();
    std::vector<int> idx;
    for (int a = 0; a < n_age; ++a) {
      idx.push_back(5 * n_age + a);
    }
    zero_every_add(z, 1, idx);
    return z;
  }

  static data_type build_data(const double* d) {
    return data_type{d[0]};
  }

  DUST2_HD static void initial(real_type time, const shared_state& shared,
                               internal_state& internal,
                               rng_state_type& rng_state,
                               real_type* state_next) {
    for (int a = 0; a < n_age; ++a) {
      state_next[a] = shared.N[a] - shared.I0;
      state_next[n_age + a] = 0;
      state_next[2 * n_age + a] = shared.I0;
      state_next[3 * n_age + a] = 0;
      state_next[4 * n_age + a] = 0;
      state_next[5 * n_age + a] = 0;
    }
  }

  DUST2_HD static void update(real_type time, real_type dt,
                              const real_type* state,
                              const shared_state& shared,
                              internal_state& internal,
                              rng_state_type& rng_state,
                              real_type* state_next) {
    const real_type* S = state;
    const real_type* E = state + n_age;
    const real_type* I = state + 2 * n_age;
    const real_type* R = state + 3 * n_age;
    const real_type* cum = state + 4 * n_age;
    const real_type* inc = state + 5 * n_age;
    // Every age's infection probability depends on the state at the
    // start of the step only, so all 16 are computed before the draws;
    // the prevalences x are then dead while the samplers run.
    real_type p_SE[n_age];
    {
      real_type x[n_age];
      for (int b = 0; b < n_age; ++b) {
        x[b] = I[b] * shared.inv_N[b];
      }
#pragma unroll 1
      for (int a = 0; a < n_age; ++a) {
        real_type acc = 0;
        for (int b = 0; b < n_age; ++b) {
          acc = std::fma(shared.contact[a][b], x[b], acc);
        }
        const real_type lambda = shared.beta * acc;
        p_SE[a] = 1 - math::exp(-lambda * dt);
      }
    }
    const real_type p_EI = 1 - math::exp(-shared.sigma * dt);
    const real_type p_IR = 1 - math::exp(-shared.gamma * dt);
    // the same two probabilities serve every age: prepare them once
    const auto b_EI = random::binomial_prepare(p_EI);
    const auto b_IR = random::binomial_prepare(p_IR);
    // one age per iteration, not unrolled: the body holds three samplers
#pragma unroll 1
    for (int a = 0; a < n_age; ++a) {
      const real_type n_SE = random::binomial(rng_state, S[a], p_SE[a]);
      const real_type n_EI = random::binomial(rng_state, E[a], b_EI);
      const real_type n_IR = random::binomial(rng_state, I[a], b_IR);
      state_next[a] = S[a] - n_SE;
      state_next[n_age + a] = E[a] + n_SE - n_EI;
      state_next[2 * n_age + a] = I[a] + n_EI - n_IR;
      state_next[3 * n_age + a] = R[a] + n_IR;
      state_next[4 * n_age + a] = cum[a] + n_EI;
      state_next[5 * n_age + a] = inc[a] + n_EI;
    }
  }

  static void count_prepare(shared_state& s, real_type dt) {
    count_table& c = s.counts;
    c.key_dt = math::bits_of(dt);
    c.after[0] = random::make_count_prob(1 - math::exp(-s.sigma * dt));
    c.after[1] = random::make_count_prob(1 - math::exp(-s.gamma * dt));
    c.ok = c.after[0].ok && c.after[1].ok;
    for (int a = 0; a < n_age && c.ok; ++a) {
      double row[n_age];
      double top = 0;
      for (int b = 0; b < n_age; ++b) {
        row[b] = s.beta * s.contact[a][b] * s.inv_N[b] * dt;
        c.ok = c.ok && row[b] >= 0 && row[b] < 1;
        top = std::max(top, row[b]);
      }
      int e = 0;
      std::frexp(top, &e);  // top < 2^e
      c.scale[a] = 32 - e;
      c.ok = c.ok && top > 0 && c.scale[a] >= 32 && c.scale[a] <= 62;
      if (!c.ok) {
        break;
      }
      // rounded to nearest; at most 2^32, so cut off there
      const double unit = std::ldexp(1.0, c.scale[a]);
      for (int b = 0; b < n_age; ++b) {
        const auto k = static_cast<std::uint64_t>(row[b] * unit + 0.5);
        c.k[a][b] = static_cast<std::uint32_t>(
          std::min<std::uint64_t>(k, 0xffffffffu));
      }
    }
  }

  // Stepped are S, E and I, and the I of the step's start as integers: 256
  // bytes a particle, in shared memory.  What has flowed into R and the
  // two case counts since they were last stored follows from what S, E and
  // I were then.
  static constexpr int count_size = 4 * n_age;

  // Within an age nothing exceeds the sum of its entries.
  template <typename G, typename C>
  DUST2_HD static bool count_load(const G& g, C&& c) {
    bool ok = true;
#pragma unroll
    for (int a = 0; a < n_age; ++a) {
      float sum = 0;
      for (int j = 0; j < 6; ++j) {
        float f = 0;
        ok &= random::filter::count_of(g[j * n_age + a], &f);
        sum += f;
        if (j < 3) {
          c[j * n_age + a] = f;
        }
      }
      ok &= sum < random::COUNT_LIMIT;
    }
    return ok;
  }

  template <typename G, typename C>
  DUST2_HD static void count_store(G&& g, C&& c) {
#pragma unroll
    for (int a = 0; a < n_age; ++a) {
      float was[6];
      for (int j = 0; j < 6; ++j) {
        random::filter::count_of(g[j * n_age + a], &was[j]);
      }
      const float S = c[a];
      const float E = c[n_age + a];
      const float I = c[2 * n_age + a];
      const float n_EI = (was[0] + was[1]) - (S + E);
      const float n_IR = (was[2] + n_EI) - I;
      g[a] = random::filter::count_to_double(S);
      g[n_age + a] = random::filter::count_to_double(E);
      g[2 * n_age + a] = random::filter::count_to_double(I);
      g[3 * n_age + a] = random::filter::count_to_double(was[3] + n_IR);
      g[4 * n_age + a] = random::filter::count_to_double(was[4] + n_EI);
      g[5 * n_age + a] = random::filter::count_to_double(was[5] + n_EI);
    }
  }

  // 1 - exp(-lambda_a dt) as update() forms it.
  template <typename C>
  DUST2_SAMPLER static real_type p_SE_fp64(const shared_state& shared,
                                           const C& c, int a,
                                           real_type dt) {
    real_type acc = 0;
    for (int b = 0; b < n_age; ++b) {
      const std::uint32_t I = c.quad(3 * n_age, b / 4).v[b % 4];
      const real_type x =
        random::filter::count_to_double(static_cast<float>(I)) *
        shared.inv_N[b];
      acc = std::fma(shared.contact[a][b], x, acc);
    }
    const real_type lambda = shared.beta * acc;
    return 1 - math::exp(-lambda * dt);
  }

  template <typename C>
  DUST2_HD static void count_update(real_type time, real_type dt, C&& c,
                                    const shared_state& shared,
                                    rng_state_type& rng_state) {
    const count_table& tab = shared.counts;
    std::uint32_t I_sum = 0;
#pragma unroll
    for (int q = 0; q < n_age / 4; ++q) {
      count_quad I;
      for (int j = 0; j < 4; ++j) {
        I.v[j] = static_cast<std::uint32_t>(c[2 * n_age + 4 * q + j]);
        I_sum += I.v[j];
      }
      c.quad(3 * n_age, q) = I;
    }
    const float half_sum = 0.501f * static_cast<float>(I_sum);
#pragma unroll 1
    for (int a = 0; a < n_age; ++a) {
      std::uint64_t acc = 0;
#pragma unroll
      for (int q = 0; q < n_age / 4; ++q) {
        const count_quad I = c.quad(3 * n_age, q);
        const count_quad k =
          reinterpret_cast<const count_quad*>(tab.k[a])[q];
        for (int j = 0; j < 4; ++j) {
          acc += static_cast<std::uint64_t>(k.v[j]) * I.v[j];
        }
      }
      const float S = c[a];
      const float E = c[n_age + a];
      const float I = c[2 * n_age + a];
      // a hazard of 1/2 or more is passed on as such
      const int scale = tab.scale[a];
      const std::uint64_t x62 =
        (acc >> (scale - 1)) != 0 ? ~0ull : acc << (62 - scale);
      const float units =
        std::fmaf(static_cast<float>(static_cast<std::uint32_t>(acc >> 32)),
                  0x1p32f,
                  static_cast<float>(static_cast<std::uint32_t>(acc)));
      random::draw_prob d = random::hazard_draw(
        x62, half_sum * random::filter::rcp32(units));
      d.zero = I_sum == 0;
      float n = S;
      float n_SE = 0, n_EI = 0, n_IR = 0;
#pragma unroll 1
      for (int j = 0; j < 3; ++j) {
        const float k = random::draw_count(rng_state, n, d, [&] {
          return j == 0 ? p_SE_fp64(shared, c, a, dt) : tab.after[j - 1].p;
        });
        if (j < 2) {
          d = tab.after[j].d;
        }
        n = j == 0 ? E : I;
        n_SE = j == 0 ? k : n_SE;
        n_EI = j == 1 ? k : n_EI;
        n_IR = k;
      }
      c[a] = S - n_SE;
      c[n_age + a] = E + n_SE - n_EI;
      c[2 * n_age + a] = I + n_EI - n_IR;
    }
  }

  DUST2_HD static real_type compare_data(const real_type time,
                                         const real_type* state,
                                         const data_type& data,
                                         const shared_state& shared,
                                         internal_state& internal,
                                         rng_state_type& rng_state) {
    if (math::is_nan(data.incidence)) {
      return 0;
    }
    real_type mu = 0;
    for (int a = 0; a < n_age; ++a) {
      mu += state[5 * n_age + a];
    }
    return density::negative_binomial_mu(data.incidence, shared.size,
                                         mu + 1e-6, true);
  }
};

}  // namespace systems
}  // namespace dust2gpu
