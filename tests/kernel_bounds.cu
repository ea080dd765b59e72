// Blocks per SM that the systems' kernels are compiled for: those that step
// counts, and the others.
#include <cstdio>

#include "engine/discrete.cuh"
#include "systems/seir_age.hpp"
#include "systems/sir.hpp"
#include "systems/sir_cases.hpp"
#include "systems/walk.hpp"

using namespace dust2gpu;

template <typename T>
void print() {
  std::printf("%d %d\n", engine::step_blocks_of<T>::value,
              engine::min_blocks_of<T>::value);
}

int main() {
  print<systems::sir>();
  print<systems::sir_cases>();
  print<systems::seir_age>();
  print<systems::walk>();
  return 0;
}
