// Dormand-Prince 5(4) integrator for one particle, run by one thread.
//
// A restatement of dust2's solver (inst/include/dust2/continuous/
// solver.hpp) for register-resident state:
//   try_step            7-stage FSAL step, dense-output coefficient c5 and
//                       the RMS error estimate                  (:96-149)
//   step                accept/reject loop with the PI controller, error
//                       checks and truncation at t_end; the step size is
//                       not updated after a truncated step     (:153-229)
//   run                 integration to t_end, honouring critical times
//                       and zero_every resets                  (:232-262)
//   initialise          Hairer's initial step size             (:265-324)
//   update_interpolation, apply_zero_every(_final)   (:335-352, :437-492)
// The Butcher tableau and Shampine's dense-output weights are the
// published Dormand-Prince (1980) / Shampine (1986) coefficients.
//
// GB300's FP64 pipe is the bound, so the FP64 instructions of a step are
// cut where the rounding may change within the solver's tolerance: the
// stage sums are fused multiply-add chains over h-scaled weights, the
// controller works with the mean square of the error instead of its root
// (powers of half the exponent, through the engine's exp and log in integer
// fixed point), the dense output's coefficients are formed when an output
// asks for them, and the divisions of the error norm, the controller, the
// initial step size and the interpolation point are multiplications by the
// engine's reciprocal.  Everything else (controller logic, truncation,
// zero_every) computes the reference's values.  On 65,536 instances of the
// batched sirode workload: 325 FP64 operations and 217 FP64 instructions an
// attempted step (552 and 352 with coefficients formed at every step, a
// root, and weights scaled where that is more), pipe 83% busy, 8.1 ms a
// launch (12.8).  65,536 of them with 28 outputs: 11.3 -> 7.1 ms a run, 300
// of them 2.82 -> 1.65 ms, where one warp's chain is what takes the time.
#pragma once

#include <cmath>

#include "../dust2gpu/common.hpp"
#include "../dust2gpu/math.hpp"
#include "../dust2gpu/system.hpp"

namespace dust2gpu {
namespace engine {
namespace dopri5 {

constexpr double C2 = 0.2;
constexpr double C3 = 0.3;
constexpr double C4 = 0.8;
constexpr double C5 = 8.0 / 9.0;
constexpr double A21 = 0.2;
constexpr double A31 = 3.0 / 40.0;
constexpr double A32 = 9.0 / 40.0;
constexpr double A41 = 44.0 / 45.0;
constexpr double A42 = -56.0 / 15.0;
constexpr double A43 = 32.0 / 9.0;
constexpr double A51 = 19372.0 / 6561.0;
constexpr double A52 = -25360.0 / 2187.0;
constexpr double A53 = 64448.0 / 6561.0;
constexpr double A54 = -212.0 / 729.0;
constexpr double A61 = 9017.0 / 3168.0;
constexpr double A62 = -355.0 / 33.0;
constexpr double A63 = 46732.0 / 5247.0;
constexpr double A64 = 49.0 / 176.0;
constexpr double A65 = -5103.0 / 18656.0;
constexpr double A71 = 35.0 / 384.0;
constexpr double A73 = 500.0 / 1113.0;
constexpr double A74 = 125.0 / 192.0;
constexpr double A75 = -2187.0 / 6784.0;
constexpr double A76 = 11.0 / 84.0;
constexpr double E1 = 71.0 / 57600.0;
constexpr double E3 = -71.0 / 16695.0;
constexpr double E4 = 71.0 / 1920.0;
constexpr double E5 = -17253.0 / 339200.0;
constexpr double E6 = 22.0 / 525.0;
constexpr double E7 = -1.0 / 40.0;
constexpr double D1 = -12715105075.0 / 11282082432.0;
constexpr double D3 = 87487479700.0 / 32700410799.0;
constexpr double D4 = -10690763975.0 / 1880347072.0;
constexpr double D5 = 701980252875.0 / 199316789632.0;
constexpr double D6 = -1453857185.0 / 822651844.0;
constexpr double D7 = 69997945.0 / 29380423.0;

// Solver controls as seen by a kernel.
struct control_dev {
  int max_steps;
  double atol;
  double rtol;
  double step_size_min;
  double step_size_max;
  double factor_safe;
  double facc1;   // 1 / factor_min
  double facc2;   // 1 / factor_max
  double beta;
  double constant;
  const double* critical;  // sorted critical times
  int n_critical;
  double* step_times;      // [particle][cap] when recording, else null
  int* n_step_times;       // [particle]
  int step_times_cap;
};

// Per-particle solver state, held in registers during a kernel.
template <int NV>
struct state {
  double dydt[NV];
  double c1[NV];
  double c2[NV];
  double c3[NV];
  double c4[NV];
  double c5[NV];
  double t0;
  double t1;
  double h;          // last.h
  double step_size;
  double mean_square;  // dust2's error, squared
  int n_steps;
  int n_steps_accepted;
  int n_steps_rejected;
  int err;           // error code (0 = none)
  // The dense-output record of the last accepted step is formed when it is
  // needed (settle, interpolate_reset).  Until then c1 holds y before the step,
  // c2 its change and c3 the derivative before it; the stages are still in
  // scratch (k3 .. k6, and the derivative after it in k2).  c4_set has a
  // bit for each entry of c4 that interpolate_reset has written since.
  static constexpr int c4_words = (NV + 31) / 32;
  bool pending;
  std::uint32_t c4_set[c4_words];
  // While has_log_error, log_error is that of mean_square (below 1e-8,
  // log_floor).
  bool has_log_error;
  double log_error;

  DUST2_HD void clear_c4() {
#pragma unroll
    for (int w = 0; w < c4_words; ++w) {
      c4_set[w] = 0;
    }
  }
  DUST2_HD void mark_c4(int i) {
#pragma unroll
    for (int w = 0; w < c4_words; ++w) {
      if (w == i / 32) {
        c4_set[w] |= 1u << (i % 32);
      }
    }
  }
  DUST2_HD bool c4_marked(int i) const {
    return (c4_set[i / 32] >> (i % 32)) & 1;
  }
};

template <int NV>
struct scratch {
  double y_next[NV];
  double y_stiff[NV];
  double k2[NV];
  double k3[NV];
  double k4[NV];
  double k5[NV];
  double k6[NV];
};

DUST2_HD double square(double x) {
  return x * x;
}

// std::min / std::max semantics (NaN handling differs from fmin/fmax).
DUST2_HD double ref_min(double a, double b) {
  return (b < a) ? b : a;
}

DUST2_HD double ref_max(double a, double b) {
  return (a < b) ? b : a;
}

// ref_max(|a|, |b|) with the comparison on the bits (a NaN counts as
// larger than any number; the caller's result is then NaN either way).
DUST2_HD double max_abs(double a, double b) {
  const std::uint64_t ua = math::bits_of(a) & 0x7fffffffffffffffull;
  const std::uint64_t ub = math::bits_of(b) & 0x7fffffffffffffffull;
  return math::from_bits(ua < ub ? ub : ua);
}

DUST2_HD double clamp(double x, double lo, double hi) {
  return ref_max(ref_min(x, hi), lo);
}

// t / period, exactly: for a period that is a power of two (the usual
// daily reset has period 1) the quotient is t times the exact reciprocal,
// the same correctly rounded value as the division; other periods divide.
DUST2_HD double div_period(double t, double period) {
  const std::uint64_t b = math::bits_of(period);
  const std::uint64_t e = b >> 52;  // sign and biased exponent
  if ((b & 0x000fffffffffffffull) == 0 && e >= 2 && e <= 2045) {
    // an exponent subtraction where both are normal
    const std::uint64_t tb = math::bits_of(t);
    const std::uint64_t te = (tb >> 52) & 0x7ff;
    const std::uint64_t qe = te + 1023 - e;
    if (te - 1 < 2046 && qe - 1 < 2046) {
      return math::from_bits(tb + ((1023 - e) << 52));
    }
    return t * math::from_bits((2046 - e) << 52);
  }
  return math::divide_call(t, period);
}

// 1/x through the engine's reciprocal (an FP32 seed and two Newton steps,
// within an ulp) where that is accurate, |x| in [2^-99, 2^99]; a division
// elsewhere.  Four FP64 instructions instead of a division's sequence.
DUST2_HD double recip(double x) {
  const std::uint64_t e = (math::bits_of(x) >> 52) & 0x7ff;
  return e - (1023 - 99) <= 198 ? math::rcp(x) : math::divide_call(1.0, x);
}

// Systems whose state always has n_state_max entries may declare
// `static constexpr bool fixed_n_state = true`.  The solver's loops over
// variables then have no test of the number of variables: with one, the
// compiler kept every stage sum of sirode's S, I, R and two case counts
// (45 FP64 instructions a step) although the rhs reads S and I only.
template <class T, class = void>
struct has_fixed_n_state : std::false_type {};
template <class T>
struct has_fixed_n_state<T, std::void_t<decltype(T::fixed_n_state)>>
  : std::integral_constant<bool, T::fixed_n_state> {};

// A system whose variables are shared out over lanes (each integrates its
// own) sums the error norms over them: T::lane_sum(internal, x), the same
// value in every lane.  T::holds(internal, i) says whether a lane's entry i
// is a variable; the others pad it, with value and rate 0.
template <class T, class = void>
struct has_lane_sum : std::false_type {};
template <class T>
struct has_lane_sum<T, std::void_t<decltype(&T::lane_sum)>>
  : std::true_type {};

// The last coefficient of the dense output, and its value at u (v = 1 - u).
// Called, so that they are evaluated for the entry being reset: expanded
// under the test of the reset mask they were evaluated ahead of it, for
// every entry at every step (117 of 293 FP64 instructions of a sirode step
// between daily outputs, which resets nothing by interpolation).
DUST2_MATH_CORE double dense_c5(double h, double k1, double k3, double k4,
                                double k5, double k6, double k7) {
  double acc = D1 * k1;
  acc = std::fma(D3, k3, acc);
  acc = std::fma(D4, k4, acc);
  acc = std::fma(D5, k5, acc);
  acc = std::fma(D6, k6, acc);
  return h * std::fma(D7, k7, acc);
}

DUST2_MATH_CORE double dense_value(double c1, double c2, double c3, double c4,
                                   double c5, double u, double v) {
  return c1 + u * (c2 + v * (c3 + u * (c4 + v * c5)));
}

// A system may say that the rate of entry i is always that of an earlier
// entry j negated: T::opposite_rate(i) is j, or -1.  Its error estimate is
// then the other's negated, the same bits.
template <class T, class = void>
struct has_opposite_rates : std::false_type {};
template <class T>
struct has_opposite_rates<T, std::void_t<decltype(&T::opposite_rate)>>
  : std::true_type {};

template <typename T, int NV>
struct solver {
  const control_dev& ctl;
  const typename T::shared_state& shared;
  typename T::internal_state& internal;
  int n_var;
  int particle;
  // Special state after the n_var integrated variables: read by the rhs,
  // carried unchanged through every stage (solver.hpp:236-239, 274-276).
  int n_special = 0;
  // 1 / n_var for the error norm's mean
  double inv_n_var = 1.0 / n_var;
  // the controller's constants: its logarithms are of the mean square, so
  // twice those of the error
  double log_safe = math::log(ctl.factor_safe);
  double log_floor = 2 * math::log(1e-4);
  double half_constant = 0.5 * ctl.constant;
  double half_beta = 0.5 * ctl.beta;
  double inv_facc1 = 1 / ctl.facc1;
  double inv_facc2 = 1 / ctl.facc2;

  // Whether entry i is one of the integrated variables.
  DUST2_HD bool on(int i) const {
    return has_fixed_n_state<T>::value || i < n_var;
  }

  // log(max(mean_square, 1e-8)), given log_ms = log(mean_square)
  DUST2_HD double floored_log(double mean_square, double log_ms) const {
    return math::gt_nonneg(1e-8, mean_square) ? log_floor : log_ms;
  }

  // The inverse of the scale of entry i's errors; 0 for padding, which has
  // no scale when atol is 0.
  DUST2_HD double inv_scale(int i, double abs_y) const {
    const double r = recip(std::fma(ctl.rtol, abs_y, ctl.atol));
    if constexpr (has_lane_sum<T>::value) {
      return T::holds(internal, i) ? r : 0.0;
    } else {
      return r;
    }
  }

  DUST2_HD double total(double x) const {
    if constexpr (has_lane_sum<T>::value) {
      return T::lane_sum(internal, x);
    } else {
      return x;
    }
  }

  DUST2_HD void copy_special(const double* y, double* dst) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (i >= n_var && i < n_var + n_special) {
        dst[i] = y[i];
      }
    }
  }

  DUST2_HD void rhs(double t, const double* y, double* dydt) {
    T::rhs(t, y, shared, internal, dydt);
  }

  // The stages as chains of fused multiply-adds: y + h (a_1 k_1 + ... +
  // a_j k_j) is j + 1 FP64 instructions per variable, or j with weights
  // scaled by h once per step, where the stage is short or (the last) of
  // all variables.  The rounding differs from the reference's expression,
  // within the solver's tolerance.  Returns the mean square of the scaled
  // errors.
  DUST2_HD double try_step(double t, double h, const double* y,
                           state<NV>& st, scratch<NV>& s) {
    const double* k1 = st.dydt;
    const double t_next = t + h;
    const double b21 = h * A21;
    const double b31 = h * A31, b32 = h * A32;
    const double b71 = h * A71, b73 = h * A73, b74 = h * A74, b75 = h * A75,
      b76 = h * A76;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) s.y_next[i] = std::fma(b21, k1[i], y[i]);
    }
    rhs(t + C2 * h, s.y_next, s.k2);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        s.y_next[i] = std::fma(b32, s.k2[i], std::fma(b31, k1[i], y[i]));
      }
    }
    rhs(t + C3 * h, s.y_next, s.k3);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        double acc = A41 * k1[i];
        acc = std::fma(A42, s.k2[i], acc);
        acc = std::fma(A43, s.k3[i], acc);
        s.y_next[i] = std::fma(h, acc, y[i]);
      }
    }
    rhs(t + C4 * h, s.y_next, s.k4);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        double acc = A51 * k1[i];
        acc = std::fma(A52, s.k2[i], acc);
        acc = std::fma(A53, s.k3[i], acc);
        acc = std::fma(A54, s.k4[i], acc);
        s.y_next[i] = std::fma(h, acc, y[i]);
      }
    }
    rhs(t + C5 * h, s.y_next, s.k5);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        double acc = A61 * k1[i];
        acc = std::fma(A62, s.k2[i], acc);
        acc = std::fma(A63, s.k3[i], acc);
        acc = std::fma(A64, s.k4[i], acc);
        acc = std::fma(A65, s.k5[i], acc);
        s.y_stiff[i] = std::fma(h, acc, y[i]);
      }
    }
    rhs(t_next, s.y_stiff, s.k6);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        double acc = std::fma(b71, k1[i], y[i]);
        acc = std::fma(b73, s.k3[i], acc);
        acc = std::fma(b74, s.k4[i], acc);
        acc = std::fma(b75, s.k5[i], acc);
        s.y_next[i] = std::fma(b76, s.k6[i], acc);
      }
    }
    rhs(t_next, s.y_next, s.k2);
    double err = 0.0;  // of the estimates over h
    double estimate[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        double acc = E1 * k1[i];
        acc = std::fma(E3, s.k3[i], acc);
        acc = std::fma(E4, s.k4[i], acc);
        acc = std::fma(E5, s.k5[i], acc);
        acc = std::fma(E6, s.k6[i], acc);
        acc = std::fma(E7, s.k2[i], acc);
        if constexpr (has_opposite_rates<T>::value) {
          // an entry whose rate is that of an earlier one, negated
          const int j = T::opposite_rate(i);
          acc = j >= 0 ? -estimate[j >= 0 ? j : 0] : acc;
        }
        estimate[i] = acc;
        const double sk = acc * inv_scale(i, max_abs(y[i], s.y_next[i]));
        err = std::fma(sk, sk, err);
      }
    }
    return total(err) * inv_n_var * (h * h);
  }

  // The record of an accepted step: what settle and dense_output need and
  // the next trial step overwrites.  Forming c3, c4 and c5 of every entry
  // at every step took 45 of a sirode step's 351 FP64 instructions, where
  // only the entry being reset is ever interpolated.
  DUST2_HD void update_interpolation(double t, double h, const double* y,
                                     state<NV>& st, scratch<NV>& s) {
    st.t0 = t;
    st.t1 = t + h;
    st.h = h;
    st.pending = true;
    st.clear_c4();
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        st.c1[i] = y[i];
        st.c2[i] = s.y_next[i] - y[i];
        st.c3[i] = st.dydt[i];
      }
    }
  }

  // Coefficients 3 and 4 of entry i of a pending record; `after` is the
  // derivative after its step.
  DUST2_HD double coefficient3(int i, const state<NV>& st) const {
    return std::fma(st.h, st.c3[i], -st.c2[i]);
  }
  DUST2_HD double coefficient4(int i, const state<NV>& st, double c3,
                               double after) const {
    return st.c4_marked(i) ? st.c4[i] :
      std::fma(-st.h, after, st.c2[i]) - c3;
  }

  // Coefficients 3 to 5 of entry i of a pending record.
  DUST2_HD void coefficients(int i, const state<NV>& st,
                             const scratch<NV>& s, double* c3, double* c4,
                             double* c5) const {
    *c3 = coefficient3(i, st);
    *c4 = coefficient4(i, st, *c3, s.k2[i]);
    *c5 = dense_c5(st.h, st.c3[i], s.k3[i], s.k4[i], s.k5[i], s.k6[i],
                   s.k2[i]);
  }

  // Complete the record, before it is stored.
  DUST2_HD void settle(state<NV>& st, const scratch<NV>& s) const {
    if (!st.pending) {
      return;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        double c3, c4, c5;
        coefficients(i, st, s, &c3, &c4, &c5);
        st.c3[i] = c3;
        st.c4[i] = c4;
        st.c5[i] = c5;
      }
    }
    st.pending = false;
  }

  // The record when the solver gives up after a rejected step: that step
  // has overwritten the stages.  The accepted step's coefficients are
  // completed (the derivative after it is st.dydt), and c5 is the rejected
  // step's, as the reference forms it in every trial step (solver.hpp
  // try_step); st.t1 holds that step's size.
  DUST2_HD void keep_after_rejection(state<NV>& st,
                                     const scratch<NV>& s) const {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        if (st.pending) {
          const double c3 = coefficient3(i, st);
          st.c4[i] = coefficient4(i, st, c3, st.dydt[i]);
          st.c3[i] = c3;
        }
        st.c5[i] = dense_c5(st.t1, st.dydt[i], s.k3[i], s.k4[i], s.k5[i],
                            s.k6[i], s.k2[i]);
      }
    }
    st.t1 = st.t0 + st.h;
    st.pending = false;
  }

  DUST2_HD void record_step_time(double t) {
    if (ctl.step_times != nullptr) {
      int& n = ctl.n_step_times[particle];
      if (n < ctl.step_times_cap) {
        ctl.step_times[static_cast<long>(particle) * ctl.step_times_cap + n] =
          t;
      }
      n++;
    }
  }

  // One pass of step's accept/reject loop (solver.hpp:161-226): the error
  // checks, truncation at t_end, one trial step and its acceptance.
  // Returns 1 when the step was accepted (t then holds the new time), 0
  // when it was rejected (h shrunk, reject set; try again) and -1 on an
  // error (st.err set, t unchanged).
  DUST2_HD int attempt(double& t, double t_end, double* y, double& h,
                       bool& reject, state<NV>& st, scratch<NV>& s) {
    const int err = st.n_steps > ctl.max_steps ? ERR_ODE_TOO_MANY_STEPS :
      h < ctl.step_size_min ? ERR_ODE_STEP_TOO_SMALL :
      h <= fabs(t) * 2.220446049250313e-16 ? ERR_ODE_STEP_VANISHED : 0;
    if (err != 0) {
      st.err = err;
      if (reject) {
        keep_after_rejection(st, s);
      }
      return -1;
    }
    const bool truncated = t + h > t_end;
    if (truncated) {
      h = t_end - t;
    }
    const double mean_square = try_step(t, h, y, st, s);
    st.n_steps++;
    // The controller's powers through one logarithm and one exponential
    // of the engine (integer fixed point, no FP64 instruction):
    // safe fac_old^beta / err^c = exp(log safe + beta log fac_old -
    // c log err), the factor of the step size, with the logarithms of
    // err^2; log 0 = -Inf, and NaN and Inf propagate as through pow.
    const double log_err = math::log(mean_square);
    if (mean_square <= 1) {
      update_interpolation(t, h, y, st, s);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (on(i)) {
          st.dydt[i] = s.k2[i];
          y[i] = s.y_next[i];
        }
      }
      st.n_steps_accepted++;
      record_step_time(truncated ? t_end : t + h);
      if (!truncated) {
        // log fac_old is the last step's log err, or the floor's
        const double log_old = st.has_log_error ? st.log_error :
          floored_log(st.mean_square, math::log(st.mean_square));
        const double log_fac = std::fma(-half_constant, log_err,
                                        half_beta * log_old) + log_safe;
        const double h_new =
          h * clamp(math::exp(log_fac), inv_facc1, inv_facc2);
        const double h_max = reject ? h : ctl.step_size_max;
        st.step_size = ref_min(h_new, h_max);
        st.mean_square = mean_square;
        st.log_error = floored_log(mean_square, log_err);
        st.has_log_error = true;
      }
      t = truncated ? t_end : t + h;
      return 1;
    }
    reject = true;
    st.t1 = h;  // until the next accepted step, or keep_after_rejection
    if (st.n_steps_accepted >= 1) {
      st.n_steps_rejected++;
    }
    h *= ref_max(inv_facc1, math::exp(std::fma(-half_constant, log_err,
                                               log_safe)));
    return 0;
  }

  // One accepted step (solver.hpp:153-229); returns the new time.
  DUST2_HD double step(double t, double t_end, double* y, state<NV>& st,
                       scratch<NV>& s) {
    bool reject = false;
    double h = st.step_size;
    while (attempt(t, t_end, y, h, reject, st, s) == 0) {
    }
    return t;
  }

  // Dense output of the last step for the zero_every entries of `mask`,
  // written into c4[0..] in index order (the reference uses c4 as its
  // scratch buffer, solver.hpp:456-458) and then subtracted from y.
  DUST2_HD void interpolate_reset(const zero_every_spec& z, int e,
                                  double t_reset, double* y, state<NV>& st,
                                  const scratch<NV>& s) {
    const double u = (t_reset - st.t0) * recip(st.h);
    const double v = 1 - u;
    int r = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i) && z.has(e, i)) {
        double c3 = st.c3[i], c4 = st.c4[i], c5 = st.c5[i];
        if (st.pending) {
          coefficients(i, st, s, &c3, &c4, &c5);
        }
        const double val = dense_value(st.c1[i], st.c2[i], c3, c4, c5, u, v);
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          if (q == r) {
            st.c4[q] = val;
          }
        }
        st.mark_c4(r);
        ++r;
      }
    }
    r = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i) && z.has(e, i)) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          if (q == r) {
            y[i] -= st.c4[q];
          }
        }
        ++r;
      }
    }
  }

  DUST2_HD void apply_zero_every(double t, double* y, const zero_every_spec& z,
                                 state<NV>& st, const scratch<NV>& s) {
    if (z.n == 0 || st.h == 0) {
      return;
    }
    for (int e = 0; e < z.n; ++e) {
      const double period = z.period[e];
      const double n = math::floor_bits(div_period(t, period));
      const double m = math::floor_bits(div_period(st.t0, period));
      if (n > m) {
        const double t_reset = n * period;
        if (t_reset == t) {
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            if (on(i) && z.has(e, i)) {
              y[i] = 0;
            }
          }
        } else {
          interpolate_reset(z, e, t_reset, y, st, s);
        }
      }
    }
  }

  DUST2_HD void apply_zero_every_final(double t, double* y,
                                       const zero_every_spec& z,
                                       state<NV>& st, const scratch<NV>& s) {
    if (z.n == 0 || st.h == 0) {
      return;
    }
    for (int e = 0; e < z.n; ++e) {
      const double period = z.period[e];
      if (st.h > period) {
        const int n = static_cast<int>(ceil(div_period(t, period)));
        const int m = static_cast<int>(ceil(div_period(st.t0, period)));
        if (n > m) {
          const double t_reset = (n - 1) * period;
          interpolate_reset(z, e, t_reset, y, st, s);
        }
      }
    }
  }

  // solver.hpp:232-262
  DUST2_HD double run(double t, double t_end, double* y,
                      const zero_every_spec& z, state<NV>& st,
                      scratch<NV>& s) {
    if (n_special > 0) {
      copy_special(y, s.y_next);
      copy_special(y, s.y_stiff);
    }
    if (ctl.n_critical == 0) {
      while (t < t_end && st.err == 0) {
        apply_zero_every(t, y, z, st, s);
        t = step(t, t_end, y, st, s);
      }
    } else {
      int tc = 0;
      while (tc < ctl.n_critical && ctl.critical[tc] <= t) {
        ++tc;
      }
      double t_end_i = (tc == ctl.n_critical || ctl.critical[tc] >= t_end) ?
        t_end : ctl.critical[tc];
      while (t < t_end && st.err == 0) {
        apply_zero_every(t, y, z, st, s);
        t = step(t, t_end_i, y, st, s);
        if (t >= t_end_i && t < t_end) {
          ++tc;
          t_end_i = (tc == ctl.n_critical || ctl.critical[tc] >= t_end) ?
            t_end : ctl.critical[tc];
        }
      }
    }
    if (st.err == 0) {
      apply_zero_every_final(t, y, z, st, s);
    }
    return t;
  }

  // solver.hpp:265-324 (the interpolation record `last` is kept, as the
  // reference keeps it across re-initialisation).
  DUST2_HD void initialise(double t, const double* y, state<NV>& st,
                           scratch<NV>& s) {
    st.step_size = 0;
    st.mean_square = 0;
    st.has_log_error = false;
    st.n_steps = 0;
    st.n_steps_accepted = 0;
    st.n_steps_rejected = 0;
    if (ctl.step_times != nullptr) {
      ctl.n_step_times[particle] = 0;
    }
    record_step_time(t);
    if (st.pending) {
      // c4 needs the derivative after the record's step, which may be
      // wanted once the stages are gone (keep_after_rejection)
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (on(i)) {
          st.c4[i] = coefficient4(i, st, coefficient3(i, st), s.k2[i]);
          st.mark_c4(i);
        }
      }
    }
    double* f0 = st.dydt;
    double* f1 = s.y_stiff;  // not the stages of a pending record
    double* y1 = s.y_next;
    double inv_sk[NV];
    if (n_special > 0) {
      copy_special(y, y1);
    }
    rhs(t, y, f0);
    double norm_f = 0.0;
    double norm_y = 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        inv_sk[i] = inv_scale(i, fabs(y[i]));
        const double f = f0[i] * inv_sk[i];
        const double g = y[i] * inv_sk[i];
        norm_f = std::fma(f, f, norm_f);
        norm_y = std::fma(g, g, norm_y);
      }
    }
    norm_f = total(norm_f);
    norm_y = total(norm_y);
    double h = (norm_f <= 1e-10 || norm_y <= 1e-10) ?
      1e-6 : sqrt(norm_y / norm_f) * 0.01;
    h = ref_min(h, ctl.step_size_max);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        y1[i] = std::fma(h, f0[i], y[i]);
      }
    }
    rhs(t + h, y1, f1);
    double der2 = 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (on(i)) {
        const double f = (f1[i] - f0[i]) * inv_sk[i];
        der2 = std::fma(f, f, der2);
      }
    }
    der2 = sqrt(total(der2)) / h;
    const double order = 5;
    const double der12 = ref_max(fabs(der2), sqrt(norm_f));
    const double h1 = (der12 <= 1e-15) ?
      ref_max(1e-6, fabs(h) * 1e-3) :
      math::exp(math::log(0.01 / der12) / order);
    h = ref_min(100 * fabs(h), h1);
    if (!isfinite(h)) {
      st.err = ERR_ODE_INITIAL_STEP;
      return;
    }
    h = ref_max(h, ctl.step_size_min * 100);
    h = ref_min(h, ctl.step_size_max);
    st.step_size = h;
  }
};

}  // namespace dopri5
}  // namespace engine
}  // namespace dust2gpu
