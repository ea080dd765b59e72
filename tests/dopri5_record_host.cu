// The engine's dopri5 solver (engine/dopri5.cuh) compiled for the host, for
// tests of what it keeps between steps: the dense-output record, and resets
// that are interpolated from it.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "engine/dopri5.cuh"
#include "systems/sirode.hpp"

namespace {

namespace dp = dust2gpu::engine::dopri5;
using dust2gpu::zero_every_spec;

// `copies` times the same four variables, the last two reset every time
// unit.
template <int COPIES>
struct copies {
  static constexpr int n = 4 * COPIES;
  struct shared_state {};
  struct internal_state {};

  static void rhs(double t, const double* y, const shared_state&,
                  internal_state&, double* d) {
    for (int c = 0; c < n; c += 4) {
      const double s = std::sin(1.3 * t);
      d[c] = 0.4 * y[c] * (1 - y[c] / 10) + 0.2 * s;
      d[c + 1] = 0.3 * y[c] - 0.2 * y[c + 1];
      d[c + 2] = 0.3 * y[c];
      d[c + 3] = 2 + s;
    }
  }
  static void start(double* y) {
    for (int c = 0; c < n; c += 4) {
      y[c] = 1;
      y[c + 1] = y[c + 2] = y[c + 3] = 0;
    }
  }
  static zero_every_spec zero_every() {
    std::vector<int> index;
    for (int c = 0; c < n; c += 4) {
      index.push_back(c + 2);
      index.push_back(c + 3);
    }
    auto z = dust2gpu::zero_every_none();
    dust2gpu::zero_every_add(z, 1, index);
    return z;
  }
};

dp::control_dev control(double tol) {
  dp::control_dev c{};
  c.max_steps = 10000;
  c.atol = c.rtol = tol;
  c.step_size_min = 2.3e-16;
  c.step_size_max = 1e300;
  c.factor_safe = 0.9;
  c.facc1 = 1 / 0.2;
  c.facc2 = 1 / 10.0;
  c.beta = 0.04;
  c.constant = 0.2 - 0.04 * 0.75;
  return c;
}

template <int COPIES>
int wide(const double* times, int n_times, double tol, double* out,
         double* c4) {
  using T = copies<COPIES>;
  constexpr int NV = T::n;
  const auto c = control(tol);
  const typename T::shared_state sh{};
  typename T::internal_state internal{};
  const auto z = T::zero_every();
  double y[NV];
  T::start(y);
  dp::state<NV> st{};
  dp::scratch<NV> s{};
  dp::solver<T, NV> sol{c, sh, internal, NV, 0};
  sol.initialise(0.0, y, st, s);
  st.step_size = 0.01;  // initialise()'s depends on the number of variables
  double t = 0;
  for (int i = 0; i < n_times; ++i) {
    sol.run(t, times[i], y, z, st, s);
    t = times[i];
    std::memcpy(out + static_cast<long>(i) * NV, y, sizeof(y));
  }
  sol.settle(st, s);
  std::memcpy(c4, st.c4, sizeof(st.c4));
  return st.err;
}

}  // namespace

// Integrate `n_copies` copies (1, 8 or 10) of the four variables through
// `times`: the state at each, and the record's c4 at the end.
extern "C" int host_copies(int n_copies, const double* times, int n_times,
                           double tol, double* out, double* c4) {
  switch (n_copies) {
  case 1:
    return wide<1>(times, n_times, tol, out, c4);
  case 8:
    return wide<8>(times, n_times, tol, out, c4);
  case 10:
    return wide<10>(times, n_times, tol, out, c4);
  }
  return -1;
}

// A sirode instance integrated to `times` in one go, or (parts) with its
// solver record stored and loaded after each of them: the state at the end,
// the next step size and the squared error.
extern "C" int host_sirode(const double* pars, const double* times,
                           int n_times, int parts, double* out) {
  using T = dust2gpu::systems::sirode;
  constexpr int NV = 5;
  const auto c = control(1e-6);
  const auto sh = T::build_shared(pars);
  const auto z = T::zero_every(sh);
  typename T::internal_state internal{};
  dust2gpu::random::rng_state r{};
  double y[NV];
  T::initial(0.0, sh, internal, r, y);
  dp::state<NV> st{};
  dp::scratch<NV> s{};
  dp::solver<T, NV> sol{c, sh, internal, NV, 0};
  sol.initialise(0.0, y, st, s);
  double t = 0;
  for (int i = 0; i < n_times; ++i) {
    sol.run(t, times[i], y, z, st, s);
    t = times[i];
    if (parts) {
      sol.settle(st, s);
      // as load_ode leaves what is not stored
      st.pending = false;
      st.clear_c4();
      st.has_log_error = false;
      st.log_error = 0;
      s = dp::scratch<NV>{};
    }
  }
  sol.settle(st, s);
  std::memcpy(out, y, sizeof(y));
  out[5] = st.step_size;
  std::memcpy(out + 6, st.c4, sizeof(st.c4));
  return st.err;
}

namespace {

// Rejected steps at the kick, and more after it.
struct kicked {
  struct shared_state {};
  struct internal_state {};
  static void rhs(double t, const double* y, const shared_state&,
                  internal_state&, double* d) {
    d[0] = t < 5 ? 0.1 * y[0] : -200 * std::sin(40 * t) * y[0];
    d[1] = y[0] - 0.3 * y[1];
  }
};

}  // namespace

// Integrate until the solver gives up (max_steps, or ssmin), one attempt at
// a time.  got: t0, t1, h and c1 .. c5 as settled afterwards; want: those of
// the last accepted step, taken when it was made, with c5 of the last
// attempt.  Returns the error, or -1 without one by time 12; *n_rejected
// counts the attempts rejected at the end.
extern "C" int host_give_up(int max_steps, double ssmin, double* got,
                            double* want, int* n_rejected) {
  constexpr int NV = 2;
  auto c = control(1e-6);
  c.max_steps = max_steps;
  c.step_size_min = ssmin;
  const kicked::shared_state sh{};
  kicked::internal_state internal{};
  double y[NV] = {1, 0};
  dp::state<NV> st{};
  dp::scratch<NV> s{};
  dp::solver<kicked, NV> sol{c, sh, internal, NV, 0};
  sol.initialise(0.0, y, st, s);
  auto put = [](const dp::state<NV>& x, double* out) {
    out[0] = x.t0;
    out[1] = x.t1;
    out[2] = x.h;
    for (int i = 0; i < NV; ++i) {
      out[3 + i] = x.c1[i];
      out[5 + i] = x.c2[i];
      out[7 + i] = x.c3[i];
      out[9 + i] = x.c4[i];
      out[11 + i] = x.c5[i];
    }
  };
  put(st, want);
  const double end = 12;
  double t = 0;
  while (t < end) {
    bool reject = false;
    double h = st.step_size;
    *n_rejected = 0;
    for (;;) {
      const double trial = t + h > end ? end - t : h;
      const int res = sol.attempt(t, end, y, h, reject, st, s);
      if (res < 0) {
        sol.settle(st, s);
        put(st, got);
        return st.err;
      }
      if (res > 0) {
        auto settled = st;
        sol.settle(settled, s);
        put(settled, want);
        break;
      }
      ++*n_rejected;
      for (int i = 0; i < NV; ++i) {
        want[11 + i] = dp::dense_c5(trial, st.dydt[i], s.k3[i], s.k4[i],
                                    s.k5[i], s.k6[i], s.k2[i]);
      }
    }
  }
  return -1;
}
