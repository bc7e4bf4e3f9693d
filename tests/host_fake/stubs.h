// Device work that a host path reaches in these tests and that does nothing here.
#pragma once
#include <cstdint>

#include "../../chllmodel_b200/csrc/sweep.cuh"

namespace chll {
__attribute__((weak)) void sweep_prepare() {}
}  // namespace chll
