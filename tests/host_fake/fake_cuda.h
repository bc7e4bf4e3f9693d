// A CUDA runtime on the host for tests of the library's host paths: device
// memory is host memory whose blocks are remembered (and never handed out
// twice), launches are what a test binds them to, a captured graph replays them,
// and a call can be made to fail.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <functional>
#include <string>
#include <vector>

namespace fake {

struct Launch {
  std::string kernel;  // mangled name
  dim3 grid, block;
  void** args;
};

// Turns a launch into what it does when it runs (at once, or whenever the graph
// that captured it is launched).  Arguments are copied here: args ends with the
// call.  Unbound launches do nothing.
extern std::function<std::function<void()>(const Launch&)> bind;

// Whether [p, p + bytes) lies in one block that has not been freed.
bool live(const void* p, size_t bytes = 1);

// The n-th next allocation (copy) fails, 1 = the next one; 0: none.
extern int fail_malloc, fail_copy;

}  // namespace fake
