// The FP32 decisions of the binomial samplers (dust2gpu/binomial_filter.hpp)
// against the FP64 samplers, draw by draw.  Compiled for the host by
// tests/test_binomial_filter.py (with every special-function result moved
// by its whole error bound, up or down at random) and, with nvcc, for the
// device.  Prints: draws, undecided draws, disagreements.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#if !defined(__CUDACC__)
static std::uint64_t nudge_state = 88172645463325252ull;
inline float filter_nudge(float units) {
  nudge_state ^= nudge_state << 13;
  nudge_state ^= nudge_state >> 7;
  nudge_state ^= nudge_state << 17;
  return (nudge_state & 1 ? units : -units) * 0x1p-24f;
}
#define DUST2_FILTER_NUDGE(units) filter_nudge(units)
#endif

#include "dust2gpu/distributions.hpp"

using namespace dust2gpu;

struct tally {
  unsigned long long draws, undecided, wrong;
};

DUST2_HD void check(random::rng_state& rng, double n, double p, int n_draws,
                    tally& t) {
  const bool flip = p > 0.5;
  const double pp = flip ? 1.0 - p : p;
  for (int i = 0; i < n_draws; ++i) {
    random::rng_state a = rng;
    t.draws++;
    float nf;
    float k = -1.0f;
    if (random::filter::count_of(n, &nf)) {
      k = random::filter::binomial(a, nf, random::filter::make_prob(pp),
                                   [&] { return n * pp < 10.0 ? 1 : 0; });
    }
    random::rng_state b = rng;
    const double want = random::binomial_fp64(b, n, pp);
    if (k < 0.0f) {
      t.undecided++;
      // the FP64 sampler takes over from where the filter stopped
      const double x = random::binomial_fp64(a, n, pp);
      k = static_cast<float>(x);
    }
    bool same = static_cast<double>(k) == want &&
      math::bits_of(random::filter::count_to_double(k)) ==
      math::bits_of(want);
    for (int w = 0; w < 4; ++w) {
      same = same && a.state[w] == b.state[w];
    }
    t.wrong += same ? 0 : 1;
    rng = b;
  }
}

// The case of index i: counts from 1 to 2^24 - 1 and probabilities so that
// n p covers inversion, the boundary at 10 and rejection up to n / 2.
DUST2_HD void pick(random::rng_state& r, double* n, double* p) {
  const double ln = random::random_real(r) * 24;
  double nn = math::floor_bits(math::exp(ln * 0.6931471805599453));
  *n = nn < 1 ? 1 : nn > 16777215 ? 16777215 : nn;
  const double kind = random::random_real(r);
  double mean;
  if (kind < 0.4) {
    mean = 10 * random::random_real(r);
  } else if (kind < 0.5) {
    mean = 10 + 1e-5 * (random::random_real(r) - 0.5);
  } else if (kind < 0.7) {
    mean = 10 + 40 * random::random_real(r);
  } else {
    mean = *n * random::random_real(r) * random::random_real(r);
  }
  double q = mean / *n;
  if (q < 1e-9) {
    q = 1e-9;
  }
  if (q > 1 - 1e-9) {
    q = random::random_real(r) * 0.5 + 1e-9;
  }
  *p = q;
}

DUST2_HD random::rng_state start(std::uint64_t seed) {
  random::rng_state r{};
  for (int w = 0; w < 4; ++w) {
    std::uint64_t z = (seed += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    r.state[w] = z ^ (z >> 31);
  }
  return r;
}

#if defined(__CUDACC__)

__global__ void k_check(std::uint64_t seed, int n_cases, int n_draws,
                        tally* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  random::rng_state r = start(seed + 7919ull * i);
  tally t{};
  for (int c = 0; c < n_cases; ++c) {
    double n, p;
    pick(r, &n, &p);
    check(r, n, p, n_draws, t);
  }
  atomicAdd(&out->draws, t.draws);
  atomicAdd(&out->undecided, t.undecided);
  atomicAdd(&out->wrong, t.wrong);
}

int main(int argc, char** argv) {
  const int blocks = argc > 1 ? std::atoi(argv[1]) : 8;
  const int n_draws = argc > 2 ? std::atoi(argv[2]) : 16;
  tally* dev = nullptr;
  tally t{};
  if (cudaMalloc(&dev, sizeof(tally)) != cudaSuccess ||
      cudaMemset(dev, 0, sizeof(tally)) != cudaSuccess) {
    std::printf("no device\n");
    return 2;
  }
  k_check<<<blocks, 128>>>(1, 64, n_draws, dev);
  if (cudaMemcpy(&t, dev, sizeof(tally), cudaMemcpyDeviceToHost) !=
      cudaSuccess) {
    std::printf("failed\n");
    return 2;
  }
  std::printf("%llu %llu %llu\n", t.draws, t.undecided, t.wrong);
  return 0;
}

#else

int main(int argc, char** argv) {
  const int n_cases = argc > 1 ? std::atoi(argv[1]) : 20000;
  const int n_draws = argc > 2 ? std::atoi(argv[2]) : 100;
  random::rng_state r = start(argc > 3 ? std::atoi(argv[3]) : 1);
  tally t{};
  for (int c = 0; c < n_cases; ++c) {
    double n, p;
    pick(r, &n, &p);
    check(r, n, p, n_draws, t);
  }
  // single counts and whole ranges of small ones
  for (int n = 1; n <= 64; ++n) {
    for (int j = 1; j < 20; ++j) {
      check(r, n, 0.05 * j, n_draws, t);
    }
  }
  std::printf("%llu %llu %llu\n", t.draws, t.undecided, t.wrong);
  return 0;
}

#endif
