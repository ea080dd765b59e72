// Stochastic SIR with exponential observation noise: the GPU restatement
// of dust2's bundled example inst/examples/sir.cpp (same state packing,
// parameters, defaults, draw order and compare).
#pragma once

#include "../dust2gpu/system.hpp"
#include "sir_counts.hpp"

namespace dust2gpu {
namespace systems {

struct sir {
  static constexpr const char* name = "sir";
  using real_type = double;
  using rng_state_type = random::rng_state;

  struct shared_state {
    real_type N;
    real_type I0;
    real_type beta;
    real_type gamma;
    real_type exp_noise;
    sir_counts counts;
  };
  struct internal_state {};
  struct data_type {
    real_type incidence;
  };

  // 64 registers: 32 warps per SM.  The batched SIR filter, ms per run: 2
  // blocks per SM 41.3, 3 39.4, 4 39.0.
  static constexpr int step_blocks_per_sm = 4;
  static constexpr int n_state_max = 5;
  static constexpr real_type default_dt = 1;
  // state entries and the gradient of beta, gamma, I0 (sir.cpp:122-124)
  static constexpr int n_adjoint_max = 8;

  // inst/examples/sir.cpp:7-11 (parameter annotations) and :74-81.
  static constexpr parameter_info parameters[] = {
    {"I0", 1, 10, false, false},
    {"N", 1, 1000, false, true},
    {"beta", 1, 0.2, false, false},
    {"gamma", 1, 0.1, false, false},
    {"exp_noise", 1, 1e6, false, true}};
  static constexpr const char* data_names[] = {"incidence"};

  static shared_state build_shared(const double* pars) {
    shared_state s{};
    s.I0 = read_par<sir>(pars, 0);
    s.N = read_par<sir>(pars, 1);
    s.beta = read_par<sir>(pars, 2);
    s.gamma = read_par<sir>(pars, 3);
    s.exp_noise = read_par<sir>(pars, 4);
    return s;
  }

  // sir.cpp:89-93: only I0, beta and gamma can change.
  static void update_shared(const double* pars, shared_state& s) {
    s.I0 = read_par_update<sir>(pars, 0, s.I0);
    s.beta = read_par_update<sir>(pars, 2, s.beta);
    s.gamma = read_par_update<sir>(pars, 3, s.gamma);
  }

  static std::vector<packing_entry> packing_state(const shared_state&) {
    return {{"S", {}}, {"I", {}}, {"R", {}}, {"cases_cumul", {}},
            {"cases_inc", {}}};
  }

  static int n_state(const shared_state&) {
    return 5;
  }

  // sir.cpp:122-124
  static std::vector<packing_entry> packing_gradient(const shared_state&) {
    return {{"beta", {}}, {"gamma", {}}, {"I0", {}}};
  }

  static zero_every_spec zero_every(const shared_state&) {
    auto z = zero_every_none();
    zero_every_add(z, 1, {4});
    return z;
  }

  static data_type build_data(const double* d) {
    return data_type{d[0]};
  }

  DUST2_HD static void initial(real_type time, const shared_state& shared,
                               internal_state& internal,
                               rng_state_type& rng_state,
                               real_type* state_next) {
    state_next[0] = shared.N - shared.I0;
    state_next[1] = shared.I0;
    state_next[2] = 0;
    state_next[3] = 0;
    state_next[4] = 0;
  }

  DUST2_HD static void update(real_type time, real_type dt,
                              const real_type* state,
                              const shared_state& shared,
                              internal_state& internal,
                              rng_state_type& rng_state,
                              real_type* state_next) {
    const auto S = state[0];
    const auto I = state[1];
    const auto R = state[2];
    const auto cases_cumul = state[3];
    const auto cases_inc = state[4];
    const auto p_SI = p_infect(I, dt, shared);
    const auto p_IR = p_recover(dt, shared);
    const auto n_SI = random::binomial(rng_state, S, p_SI);
    const auto n_IR = random::binomial(rng_state, I, p_IR);
    state_next[0] = S - n_SI;
    state_next[1] = I + n_SI - n_IR;
    state_next[2] = R + n_IR;
    state_next[3] = cases_cumul + n_SI;
    state_next[4] = cases_inc + n_SI;
  }

  // x / N, 1 - exp(-beta I / N dt) and 1 - exp(-gamma dt), with what was
  // prepared for dt where it was (the same values).
  DUST2_HD static real_type over_N(real_type x, real_type dt,
                                   const shared_state& shared) {
    return shared.counts.prepared(dt) ?
      math::divide(x, shared.counts.by_N) : x / shared.N;
  }
  DUST2_HD static real_type p_infect(real_type I, real_type dt,
                                     const shared_state& shared) {
    return 1 - math::exp(over_N(-shared.beta * I, dt, shared) * dt);
  }
  DUST2_HD static real_type p_recover(real_type dt,
                                      const shared_state& shared) {
    return shared.counts.prepared(dt) ? shared.counts.recover.p :
      1 - math::exp(-shared.gamma * dt);
  }

  static void count_prepare(shared_state& s, real_type dt) {
    s.counts.prepare(s.N, s.beta, s.gamma, dt);
  }

  // c: S, I, R, cases_cumul, cases_inc (the last two grow by what leaves S)
  template <typename C>
  DUST2_HD static bool count_fits(const C& c) {
    return c[0] + c[1] + c[2] + c[3] + c[4] < random::COUNT_LIMIT;
  }

  template <typename C>
  DUST2_HD static void count_update(real_type time, real_type dt, C&& c,
                                    const shared_state& shared,
                                    rng_state_type& rng_state) {
    float n_SI, n_IR;
    shared.counts.draw(rng_state, c[0], c[1], shared.N, shared.beta, dt,
                       &n_SI, &n_IR);
    c[0] = c[0] - n_SI;
    c[1] = c[1] + n_SI - n_IR;
    c[2] = c[2] + n_IR;
    c[3] = c[3] + n_SI;
    c[4] = c[4] + n_SI;
  }

  DUST2_HD static real_type compare_data(const real_type time,
                                         const real_type* state,
                                         const data_type& data,
                                         const shared_state& shared,
                                         internal_state& internal,
                                         rng_state_type& rng_state) {
    const auto incidence_observed = data.incidence;
    if (math::is_nan(data.incidence)) {
      return 0;
    }
    const auto noise = random::exponential_rate(rng_state, shared.exp_noise);
    const auto incidence_modelled = state[4];
    const auto lambda = incidence_modelled + noise;
    return density::poisson(incidence_observed, lambda, true);
  }

  // The adjoint equations of the deterministic model (sir.cpp:126-210),
  // term for term: the reverse-mode derivatives of update, compare and
  // initial with respect to state and to beta, gamma, I0.
  DUST2_HD static void adjoint_initial(real_type time,
                                       const real_type* state,
                                       const real_type* adjoint,
                                       const shared_state& shared,
                                       internal_state& internal,
                                       real_type* adjoint_next) {
    const real_type adj_I = adjoint[1];
    for (int i = 0; i < 7; ++i) {
      adjoint_next[i] = adjoint[i];
    }
    adjoint_next[7] = adjoint[7] + adj_I;
  }

  // What the step back needs of the state, apart from the adjoint: the
  // engine forms it for several steps at once, one per lane.
  struct adjoint_tape {
    real_type S;
    real_type I;
    real_type p_SI;
    real_type e_SI;
  };

  DUST2_HD static adjoint_tape adjoint_prepare(real_type dt,
                                               const real_type* state,
                                               const shared_state& shared) {
    const auto I = state[1];
    return adjoint_tape{state[0], I, p_infect(I, dt, shared),
                        math::exp(over_N(-shared.beta * I * dt, dt,
                                         shared))};
  }

  DUST2_HD static void adjoint_update_tape(real_type dt,
                                           const adjoint_tape& tape,
                                           const real_type* adjoint,
                                           const shared_state& shared,
                                           real_type* adjoint_next) {
    const auto adj_S = adjoint[0];
    const auto adj_I = adjoint[1];
    const auto adj_R = adjoint[2];
    const auto adj_cases_cumul = adjoint[3];
    const auto adj_cases_inc = adjoint[4];
    const auto adj_beta = adjoint[5];
    const auto adj_gamma = adjoint[6];
    const auto adj_I0 = adjoint[7];
    const auto p_IR = p_recover(dt, shared);
    const auto adj_n_IR = -adj_I + adj_R;
    const auto adj_n_SI = adj_cases_inc + adj_cases_cumul + adj_I + -adj_S;
    const auto adj_p_IR = adj_n_IR * tape.I;
    const auto adj_p_SI = adj_n_SI * tape.S;
    const auto exp_gamma = shared.counts.prepared(dt) ?
      shared.counts.exp_gamma : math::exp(-shared.gamma);
    adjoint_next[0] = adj_n_SI * tape.p_SI + adj_S;
    adjoint_next[1] = adj_n_IR * p_IR +
      over_N(adj_p_SI * (shared.beta * dt) * tape.e_SI, dt, shared) + adj_I;
    adjoint_next[2] = adj_R;
    adjoint_next[3] = adj_cases_cumul;
    adjoint_next[4] = adj_cases_inc;
    adjoint_next[5] = adj_beta +
      over_N(adj_p_SI * tape.I * dt * tape.e_SI, dt, shared);
    adjoint_next[6] = adj_gamma + adj_p_IR * exp_gamma;
    adjoint_next[7] = adj_I0;
  }

  DUST2_HD static void adjoint_update(real_type time, real_type dt,
                                      const real_type* state,
                                      const real_type* adjoint,
                                      const shared_state& shared,
                                      internal_state& internal,
                                      real_type* adjoint_next) {
    adjoint_update_tape(dt, adjoint_prepare(dt, state, shared), adjoint,
                        shared, adjoint_next);
  }

  // The comparison's part: the derivative with respect to cases_inc.
  DUST2_HD static real_type adjoint_compare_prepare(
      const real_type* state, const data_type& data,
      const shared_state& shared) {
    const real_type noise = 1 / shared.exp_noise;
    const real_type lambda = state[4] + noise;
    return data.incidence / lambda - 1;
  }

  DUST2_HD static void adjoint_compare_tape(real_type tape,
                                            const real_type* adjoint,
                                            real_type* adjoint_next) {
    for (int i = 0; i < 8; ++i) {
      adjoint_next[i] = adjoint[i];
    }
    adjoint_next[4] = adjoint[4] + tape;
  }

  DUST2_HD static void adjoint_compare_data(real_type time,
                                            const real_type* state,
                                            const real_type* adjoint,
                                            const data_type& data,
                                            const shared_state& shared,
                                            internal_state& internal,
                                            real_type* adjoint_next) {
    adjoint_compare_tape(adjoint_compare_prepare(state, data, shared),
                         adjoint, adjoint_next);
  }
};

}  // namespace systems
}  // namespace dust2gpu
