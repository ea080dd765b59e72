// System-independent kernels of the likelihood server (engine/served.cuh):
// request start and end-of-tick bookkeeping.
#include <cmath>

#include "engine/device.cuh"
#include "engine/filter.cuh"
#include "engine/served.cuh"

namespace dust2gpu {
namespace engine {

// Reset the filter state of the listed slots (filter.hpp:156-175: ll = 0)
// and mark them running from their first observation.
__global__ void k_served_begin(served_start_list list, filter_view f,
                               int* active, int* obs, int* starting,
                               int* slot_error) {
  const int i = threadIdx.x;
  if (i >= list.n) {
    return;
  }
  const int g = list.slot[i];
  active[g] = 1;
  starting[g] = 1;
  obs[g] = 0;
  f.ll[g] = 0;
  f.gkey[g] = ordered_key(-INFINITY);
  f.gnz[g] = 0;
  f.gflag[g] = 0;
  f.mode[g] = MODE_KEEP;
  slot_error[g] = 0;
}

// After a tick: each running slot moves to its next observation and stops
// after its last; the "starting" marks of the tick are cleared.
__global__ void k_served_advance(int* active, const served_slot* slots,
                                 int* obs, int* starting, int n_slots) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_slots) {
    return;
  }
  starting[g] = 0;
  if (!active[g]) {
    return;
  }
  const int o = obs[g] + 1;
  obs[g] = o;
  if (o >= slots[g].n_obs) {
    active[g] = 0;
  }
}

}  // namespace engine
}  // namespace dust2gpu
