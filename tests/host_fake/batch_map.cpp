// chll_batch_run replays a captured launch: every address that it was given is
// still allocated when it runs, whatever launch shapes were prepared in between.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/chll_mod.h"
#include "fake_cuda.h"
#include "stubs.h"

static int bad = 0, runs = 0;
static unsigned ctas = 0;  // of the last launch

static std::function<void()> batch_launch(const fake::Launch& l) {
  if (l.kernel.find("batch_kernel") == std::string::npos) return nullptr;
  std::vector<const void*> ptrs;
  for (int a : {0, 1, 2, 3, 5}) ptrs.push_back(*static_cast<void**>(l.args[a]));
  const size_t map_bytes = sizeof(int2) * l.grid.x * *static_cast<int*>(l.args[4]);
  const unsigned grid = l.grid.x;
  return [=] {
    ++runs;
    ctas = grid;
    for (const void* p : ptrs) bad += !fake::live(p);
    if (!fake::live(ptrs[3], map_bytes)) {
      ++bad;
      return;
    }
    const int2* map = static_cast<const int2*>(ptrs[3]);
    // one wave: every replica, each in one run of CTAs
    std::vector<int> seen(16, 0);
    for (size_t e = 0; e < map_bytes / sizeof(int2); ++e) {
      if (map[e].x < -1 || map[e].x >= 16 || map[e].y < -1 || map[e].y >= 16) {
        ++bad;
      } else if (e == 0 || map[e].x != map[e - 1].x) {
        if (map[e].x >= 0) ++seen[map[e].x];
        if (map[e].x >= 0 && map[e].y >= 0) ++seen[map[e].y];
      }
    }
    for (int n : seen) bad += n != 1;
  };
}

static chll_batch* make(bool pair) {
  std::vector<chll_replica_spec> specs(16);
  for (int r = 0; r < 16; ++r) {
    std::memset(&specs[r], 0, sizeof(specs[r]));
    specs[r].ni = specs[r].nj = specs[r].nk = 32;
    specs[r].boundary = CHLL_PERIODIC;
    specs[r].kT = specs[r].K = specs[r].eps = 1.0;
    specs[r].replica = (uint32_t)r;
  }
  chll_batch* b = nullptr;
  if (chll_batch_create(specs.data(), 16, &b) != CHLL_OK) std::printf("create: %s\n", chll_last_error());
  chll_batch_set_pairing(b, pair);
  return b;
}

static void expect(bool ok, const char* what) {
  if (!ok) {
    std::printf("wrong: %s (%s)\n", what, chll_last_error());
    ++bad;
  }
}

// a larger map prepared between two runs of one shape
static void larger_map(chll_batch* b) {
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "first run");
  expect(chll_batch_set_tuning(b, 128, 0) == CHLL_OK, "set_tuning");
  expect(chll_batch_info(b, nullptr, nullptr, nullptr, nullptr) == CHLL_OK, "info");
  expect(chll_batch_set_tuning(b, 256, 0) == CHLL_OK, "set_tuning back");
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "second run");
}

// and by the tuner
static void tuned(chll_batch* b) {
  expect(chll_batch_set_tuning(b, 512, 0) == CHLL_OK, "set_tuning");
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "first run");
  expect(chll_batch_autotune(b, 2, nullptr, nullptr, nullptr) == CHLL_OK, "autotune");
  expect(chll_batch_set_tuning(b, 512, 0) == CHLL_OK, "set_tuning");
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "second run");
}

// a shape whose map cannot be allocated, then the shape before it
static void no_memory(chll_batch* b) {
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "first run");
  expect(chll_batch_set_tuning(b, 128, 0) == CHLL_OK, "set_tuning");
  fake::fail_malloc = 1;
  expect(chll_batch_info(b, nullptr, nullptr, nullptr, nullptr) == CHLL_ENOMEM, "no memory");
  expect(chll_batch_set_tuning(b, 256, 0) == CHLL_OK, "set_tuning back");
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "second run");
}

// the same where the new map's copy fails: the old shape's map is uploaded again
static void no_copy(chll_batch* b) {
  expect(chll_batch_set_tuning(b, 128, 0) == CHLL_OK, "set_tuning");
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "first run");
  expect(chll_batch_set_tuning(b, 256, 0) == CHLL_OK, "set_tuning");
  fake::fail_copy = 2;  // the map's copy goes through, the descriptors' does not
  expect(chll_batch_info(b, nullptr, nullptr, nullptr, nullptr) == CHLL_ECUDA, "no copy");
  expect(chll_batch_set_tuning(b, 128, 0) == CHLL_OK, "set_tuning back");
  expect(chll_batch_run(b, 10, 5, 0) == CHLL_OK, "second run");
  expect(ctas == 148 * 4, "the launch is the old shape's");
}

int main(int argc, char** argv) {
  fake::bind = batch_launch;
  const std::string what = argc > 1 ? argv[1] : "";
  for (int pair : {0, 1}) {
    chll_batch* b = make(pair);
    if (what == "larger_map") larger_map(b);
    if (what == "tuned") tuned(b);
    if (what == "no_memory") no_memory(b);
    if (what == "no_copy") no_copy(b);
    chll_batch_destroy(b);
  }
  std::printf("%d runs, %d wrong\n", runs, bad);
  return bad != 0 || runs < 4;
}
