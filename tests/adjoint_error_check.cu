// The adjoint kernels (engine/unfilter.cuh) on a system whose comparison
// fails at given data times: by a thread per particle, and by 8 and 32 lanes
// per particle.  For each prints code, value and log-likelihood of every
// particle.
#include <cstdio>
#include <vector>

#include "engine/unfilter.cuh"

using namespace dust2gpu;

struct picky {
  using real_type = double;
  using rng_state_type = random::rng_state;
  static constexpr int n_state_max = 1;
  static constexpr int n_adjoint_max = 2;
  static constexpr int n_output = 0;
  struct shared_state {
    double rate;
  };
  struct internal_state {};
  struct data_type {
    double y;
  };
  struct adjoint_tape {
    double x;
  };
  DUST2_HD static void update(double, double dt, const double* x,
                              const shared_state& shared, internal_state&,
                              random::rng_state&, double* next) {
    next[0] = x[0] + shared.rate * dt;
  }
  // negative data: an invalid draw, of which the error records the datum
  DUST2_HD static double compare_data(double, const double* x,
                                      const data_type& d,
                                      const shared_state&, internal_state&,
                                      random::rng_state& rng) {
    if (d.y < 0) {
      random::binomial(rng, -d.y, 2.0);
      return 0;
    }
    return x[0] * d.y;
  }
  DUST2_HD static adjoint_tape adjoint_prepare(double, const double* x,
                                               const shared_state&) {
    return adjoint_tape{x[0]};
  }
  DUST2_HD static void adjoint_update_tape(double dt, const adjoint_tape&,
                                           const double* adj,
                                           const shared_state&,
                                           double* next) {
    next[0] = adj[0];
    next[1] = adj[1] + dt * adj[0];
  }
  DUST2_HD static void adjoint_update(double, double dt, const double* x,
                                      const double* adj,
                                      const shared_state& shared,
                                      internal_state&, double* next) {
    adjoint_update_tape(dt, adjoint_prepare(dt, x, shared), adj, shared,
                        next);
  }
  DUST2_HD static double adjoint_compare_prepare(const double*,
                                                 const data_type& d,
                                                 const shared_state&) {
    return d.y;
  }
  DUST2_HD static void adjoint_compare_tape(double tape, const double* adj,
                                            double* next) {
    next[0] = adj[0] + tape;
    next[1] = adj[1];
  }
  DUST2_HD static void adjoint_compare_data(double, const double* x,
                                            const double* adj,
                                            const data_type& d,
                                            const shared_state& shared,
                                            internal_state&, double* next) {
    adjoint_compare_tape(adjoint_compare_prepare(x, d, shared), adj, next);
  }
  DUST2_HD static void adjoint_initial(double, const double*,
                                       const double* adj,
                                       const shared_state&, internal_state&,
                                       double* next) {
    next[0] = adj[0];
    next[1] = adj[1];
  }
};

template <typename V>
V* managed(std::size_t n) {
  V* p = nullptr;
  if (cudaMallocManaged(reinterpret_cast<void**>(&p), n * sizeof(V)) !=
      cudaSuccess) {
    std::printf("no device\n");
    std::exit(2);
  }
  for (std::size_t i = 0; i < n; ++i) {
    p[i] = V{};
  }
  return p;
}

int main() {
  constexpr int N = 5, stride = 32, n_times = 70;
  const int fails[][2] = {{-1, -1}, {0, 3}, {45, 47}, {33, 69}, {69, 69}};
  for (const auto& f : fails) {
    engine::system_view<picky> v{};
    v.state = managed<double>(stride);
    v.rng = managed<std::uint64_t>(4 * stride);
    auto* shared = managed<picky::shared_state>(1);
    shared[0].rate = 0.5;
    v.shared = shared;
    auto* zero = managed<zero_every_spec>(1);
    v.zero_every = zero;
    auto* tiles = managed<engine::tile>(1);
    tiles[0] = engine::tile{0, 0, N, 0};
    v.tiles = tiles;
    v.stride = stride;
    v.n_state = 1;
    v.deterministic = true;
    v.any_error = managed<int>(1);
    auto* active = managed<int>(1);
    active[0] = 1;
    auto* step = managed<int>(n_times);
    auto* back = managed<int>(n_times);
    auto* times = managed<double>(n_times);
    auto* data = managed<picky::data_type>(n_times);
    for (int i = 0; i < n_times; ++i) {
      step[i] = i + 1;
      back[i] = 1;
      times[i] = i + 1;
      data[i].y = i == f[0] || i == f[1] ? -(i + 1.0) : 1.0;
    }
    auto* hist = managed<double>((n_times + 1) * stride);
    auto* ll = managed<double>(stride);
    auto* gradient = managed<double>(N);
    for (int lanes : {1, 8, 32}) {
      v.errors = managed<particle_error>(stride);
      for (int k = 0; k < N; ++k) {
        v.state[k] = k;
      }
      if (lanes == 1) {
        engine::k_unfilter_adjoint<picky><<<1, 256>>>(
          v, active, step, n_times, n_times, 0, n_times, times, 1, data, 1,
          hist, ll, gradient, 1, engine::unfilter_save{});
      } else if (lanes == 8) {
        engine::k_unfilter_adjoint_lanes<picky, 8><<<2, 32>>>(
          v, active, step, back, N, n_times, n_times, 0, n_times, times, 1,
          data, 1, hist, ll, gradient, 1, engine::unfilter_save{});
      } else {
        engine::k_unfilter_adjoint_lanes<picky, 32><<<N, 32>>>(
          v, active, step, back, N, n_times, n_times, 0, n_times, times, 1,
          data, 1, hist, ll, gradient, 1, engine::unfilter_save{});
      }
      if (cudaDeviceSynchronize() != cudaSuccess) {
        std::printf("failed\n");
        return 2;
      }
      for (int k = 0; k < N; ++k) {
        std::printf("%d %d %d %g %.17g %.17g\n", f[0], lanes,
                    v.errors[k].code, v.errors[k].v0, ll[k], gradient[k]);
      }
    }
  }
  return 0;
}
