// A system whose parameters take nearly all of the 48 KB of static shared
// memory that a kernel may have: the kernels that step it compile.
#include "engine/discrete.cuh"

using namespace dust2gpu;

struct large {
  using real_type = double;
  using rng_state_type = random::rng_state;
  static constexpr int n_state_max = 2;
  static constexpr int n_output = 0;
  struct shared_state {
    double table[SHARED_DOUBLES];
  };
  struct internal_state {};
  DUST2_HD static void update(double, double dt, const double* x,
                              const shared_state& shared, internal_state&,
                              random::rng_state& rng, double* next) {
    next[0] = x[0] + random::normal(rng, 0, 1) * dt;
    next[1] = x[1] + shared.table[static_cast<int>(x[0]) & 1023];
  }
};

template __global__ void engine::k_run<large>(engine::system_view<large>,
                                              double, double, int);
template __global__ void engine::k_simulate<large>(
  engine::system_view<large>, const engine::run_segment*, int, double, int,
  const int*, int, double*);
