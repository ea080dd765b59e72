// Which mixed-time systems the filter integrates with several lanes per
// particle (engine/filter.cuh has_lanes, no_resets).  Prints one digit per
// question.
#include <cstdio>

#include "engine/filter.cuh"
#include "systems/malaria.hpp"
#include "systems/sirode.hpp"

using namespace dust2gpu;

template <int SPECIAL, int OUTPUT>
struct declares_lanes {
  static constexpr int n_special = SPECIAL;
  static constexpr int n_output = OUTPUT;
  template <int L>
  struct lanes {};
};

int main() {
  auto z = zero_every_none();
  auto reset = z;
  zero_every_add(reset, 7, {1});
  std::printf("%d%d%d%d%d%d%d%d\n",
              engine::has_lanes<systems::malaria>::value,
              engine::has_lanes<systems::sirode>::value,
              engine::has_lanes<declares_lanes<1, 0>>::value,
              engine::has_lanes<declares_lanes<0, 0>>::value,
              engine::has_lanes<declares_lanes<2, 0>>::value,
              engine::has_lanes<declares_lanes<1, 1>>::value,
              engine::no_resets({z, z}), engine::no_resets({z, reset, z}));
  return 0;
}
