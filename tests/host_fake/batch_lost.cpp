// The tuner and trials whose waits give up: their leftover arrivals do not stay in
// the meeting words, they are not taken for the fastest, and a batch none of whose
// trials ran to its end is refused.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/chll_mod.h"
#include "fake_cuda.h"
#include "stubs.h"

static const int kReplicas = 16, kWords = 48 * kReplicas;
static int bad = 0, runs = 0;
static unsigned lose = 0;  // launches of this many threads per CTA give up; 1: every launch

static void expect(bool ok, const char* what) {
  if (!ok) {
    std::printf("wrong: %s (%s)\n", what, chll_last_error());
    ++bad;
  }
}

static std::function<void()> batch_launch(const fake::Launch& l) {
  if (l.kernel.find("batch_kernel") == std::string::npos) return nullptr;
  char* const states = *static_cast<char**>(l.args[1]);
  unsigned long long* const words = *static_cast<unsigned long long**>(l.args[2]);
  const unsigned threads = l.block.x;
  return [=] {
    ++runs;
    // replica 0's status word (behind d, step and nflip)
    unsigned* const status = reinterpret_cast<unsigned*>(states + 24);
    if (*status) return;
    for (int w = 0; w < kWords; ++w) expect(words[w] == 0, "meeting words are clear at a launch");
    if (lose == 1 || lose == threads) {
      *status = 1;
      words[0] = (1ull << 40) + 17;
    }
  };
}

int main() {
  fake::bind = batch_launch;
  std::vector<chll_replica_spec> specs(kReplicas);
  for (int r = 0; r < kReplicas; ++r) {
    std::memset(&specs[r], 0, sizeof(specs[r]));
    specs[r].ni = specs[r].nj = specs[r].nk = 8;
    specs[r].boundary = CHLL_PERIODIC;
    specs[r].kT = specs[r].K = specs[r].eps = 1.0;
  }
  chll_batch* b = nullptr;
  expect(chll_batch_create(specs.data(), kReplicas, &b) == CHLL_OK, "create");
  std::vector<double> m(16 * kReplicas);
  int threads = 0;
  // every trial takes the same time: without the lost ones 256 is the first
  lose = 128;
  expect(chll_batch_autotune(b, 3, &threads, nullptr, nullptr) == CHLL_OK, "autotune");
  expect(threads == 256, "a lost trial is not the fastest");
  lose = 0;
  expect(chll_batch_run(b, 4, 2, 0) == CHLL_OK, "run");
  expect(chll_batch_moments(b, m.data()) == CHLL_OK, "moments");
  // no trial runs to its end: refused, the shape and the state kept
  lose = 1;
  expect(chll_batch_autotune(b, 3, &threads, nullptr, nullptr) == CHLL_EDEVICE, "all lost");
  lose = 0;
  int32_t kept = 0;
  expect(chll_batch_get_tuning(b, &kept, nullptr, nullptr, nullptr) == CHLL_OK && kept == 256,
         "the shape is kept");
  expect(chll_batch_run(b, 4, 2, 0) == CHLL_OK, "run");
  expect(chll_batch_moments(b, m.data()) == CHLL_OK, "moments");
  // a copy back that fails is reported
  fake::fail_copy = 3;  // the two of the snapshot, then the shape's map
  expect(chll_batch_autotune(b, 3, nullptr, nullptr, nullptr) == CHLL_ECUDA, "no copy");
  chll_batch_destroy(b);
  std::printf("%d runs, %d wrong\n", runs, bad);
  return bad != 0 || runs < 10;
}
