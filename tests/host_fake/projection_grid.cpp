// The projection's launch up to the largest planes a lattice can have (fewer than 2^31
// slots per colour): at least one CTA, no more than the device holds.
#include <cstdio>

#include "fake_cuda.h"
#include "stubs.h"

int main() {
  int bad = 0, launches = 0;
  unsigned ctas = 0;
  fake::bind = [&](const fake::Launch& l) -> std::function<void()> {
    ++launches;
    ctas = l.grid.x;
    return nullptr;
  };
  const int shapes[][3] = {{4, 3, 2}, {480, 480, 480}, {4, 1 << 20, 1}, {4, (1 << 30) - 64, 1},
                           {4, (1 << 30) - 32, 1}, {4, (1 << 30) - 1, 1}};
  for (const auto& s : shapes) {
    chll::LatticeView L;
    L.col[0] = L.col[1] = nullptr;
    L.ni = s[0];
    L.nj = s[1];
    L.nk = s[2];
    L.hx = s[0] / 2;
    L.periodic = 0;
    ctas = 0;
    chll::launch_projection(L, 1, 0, 0, 1, 4, nullptr, nullptr);
    if (ctas < 1 || ctas > 148 * 6) {
      std::printf("wrong: %u CTAs for %d x %d x %d\n", ctas, s[0], s[1], s[2]);
      ++bad;
    }
  }
  return bad != 0;
}
