// Sizes that a likelihood server's memory plan is made of: per session, per
// observation and per particle, for a system given by -DSYSTEM.
#include <cstdio>

#include "engine/served.cuh"
#include "systems/seir_age.hpp"
#include "systems/sir_cases.hpp"

int main() {
  using namespace dust2gpu;
  using T = systems::SYSTEM;
  std::printf("%zu %zu %zu\n",
              sizeof(T::shared_state) + sizeof(zero_every_spec),
              sizeof(T::data_type) + sizeof(engine::obs_step),
              // state twice, generator, three weights, index, error
              2 * T::n_state_max * sizeof(double) + 4 * 8 + 3 * 8 + 4 +
              sizeof(particle_error));
  return 0;
}
