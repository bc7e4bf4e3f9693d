// The segment lengths of the column walks: the same choice as a search over every
// length (the rule's own formula), from few of them.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../chllmodel_b200/csrc/sweep_unit.cuh"

// Evaluations of the rule: next_segment's steps.
static unsigned steps(uint32_t n) {
  unsigned k = 0;
  for (uint32_t s = 1; s; s = chll::next_segment(n, s)) ++k;
  return k;
}

static uint32_t every_length(uint64_t cols, uint32_t n, uint64_t threads, double start) {
  double best = 1e300;
  uint32_t seg = 0;
  for (uint32_t s = 1; s <= n; ++s) {
    const uint64_t tasks = cols * ((n + s - 1) / s);
    const double cost = (double)((tasks + threads - 1) / threads) * (s + start);
    if (cost < best) {
      best = cost;
      seg = s;
    }
  }
  return seg;
}

static double every_walk(uint32_t units, uint32_t ncols, uint32_t planes, uint32_t threads,
                         uint32_t* seg) {
  double best = (double)((units + threads - 1) / threads);
  *seg = 0;
  for (uint32_t s = 2; s <= planes; ++s) {
    const uint64_t tasks = (uint64_t)ncols * ((planes + s - 1) / s);
    const double cost = (double)((tasks + threads - 1) / threads) *
                        ((double)s * chll::kWalkStep + chll::kWalkPrime);
    if (cost < best) {
      best = cost;
      *seg = s;
    }
  }
  return best;
}

int main() {
  std::mt19937_64 rng(11);
  int bad = 0;
  const uint32_t planes[] = {1, 2, 3, 4, 5, 16, 17, 64, 101, 128, 129, 480, 1000, 4097, 65535};
  for (uint32_t n : planes) {
    if (steps(n) > 2 * std::sqrt((double)n) + 1) {
      std::printf("wrong: %u steps for %u planes\n", steps(n), n);
      ++bad;
    }
    for (int t = 0; t < (n > 5000 ? 60 : 400); ++t) {
      const uint32_t cols = 1 + (uint32_t)std::exp2((rng() % 1800) / 100.0);
      const uint32_t threads = 32u * (1 + (uint32_t)(rng() % 4000));
      for (double start : {0.33, 0.5})
        bad += chll::cheapest_segment(cols, n, threads, start) != every_length(cols, n, threads, start);
      uint32_t a = 0, b = 0;
      const double ca = chll::walk_pass_cost(cols * n, cols, n, true, threads, -1, &a);
      const double cb = every_walk(cols * n, cols, n, threads, &b);
      bad += ca != cb || a != b;
    }
    // a fixed length: that one, or the unit loop where there is no such length
    for (int force : {1, 2, 7, 64}) {
      uint32_t a = 9;
      chll::walk_pass_cost(n * 8, 8, n, true, 256, force, &a);
      bad += a != (force >= 2 && (uint32_t)force <= n ? (uint32_t)force : 0u);
    }
  }
  std::printf("%d wrong\n", bad);
  return bad != 0;
}
