#include "fake_cuda.h"

#include <cstdlib>
#include <cstring>
#include <map>

namespace fake {

std::function<std::function<void()>(const Launch&)> bind;
int fail_malloc = 0, fail_copy = 0;

namespace {

std::map<const char*, size_t> blocks;  // live ones; freed memory stays unused
// kernels register before main
std::map<const void*, std::string>& kernels() {
  static std::map<const void*, std::string> k;
  return k;
}
bool capturing = false;
std::vector<std::function<void()>> captured;

struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
std::vector<Config> configs;

bool fails(int& countdown) { return countdown > 0 && --countdown == 0; }

cudaError_t launch(const void* func, dim3 grid, dim3 block, void** args) {
  if (grid.x == 0 || grid.y == 0 || grid.z == 0 || block.x == 0) return cudaErrorInvalidConfiguration;
  std::function<void()> f = bind ? bind({kernels()[func], grid, block, args}) : nullptr;
  if (!f) return cudaSuccess;
  if (capturing)
    captured.push_back(f);
  else
    f();
  return cudaSuccess;
}

}  // namespace

bool live(const void* p, size_t bytes) {
  const char* c = static_cast<const char*>(p);
  auto it = blocks.upper_bound(c);
  if (it == blocks.begin()) return false;
  --it;
  return c + bytes <= it->first + it->second;
}

}  // namespace fake

using namespace fake;

struct FakeGraph {
  std::vector<std::function<void()>> nodes;
};

extern "C" {

// what nvcc's host code registers
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
  kernels()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  configs.push_back({grid, block, smem, stream});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = configs.back().grid;
  *block = configs.back().block;
  *smem = configs.back().smem;
  *static_cast<cudaStream_t*>(stream) = configs.back().stream;
  configs.pop_back();
  return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t, cudaStream_t) {
  return launch(f, g, b, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, c->gridDim, c->blockDim, args);
}

cudaError_t cudaMalloc(void** p, size_t n) {
  if (fails(fail_malloc)) return cudaErrorMemoryAllocation;
  const size_t bytes = (n + 255) / 256 * 256;
  *p = std::aligned_alloc(256, bytes ? bytes : 256);
  std::memset(*p, 0xa5, bytes);
  blocks[static_cast<char*>(*p)] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (p && !blocks.erase(static_cast<char*>(p))) return cudaErrorInvalidValue;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (fails(fail_copy)) return cudaErrorInvalidValue;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  return cudaMemcpyAsync(d, s, n, k, nullptr);
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof(*a));
  a->type = live(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = true;
  captured.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  *g = reinterpret_cast<cudaGraph_t>(new FakeGraph{captured});
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(new FakeGraph(*reinterpret_cast<FakeGraph*>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (auto& f : reinterpret_cast<FakeGraph*>(e)->nodes) f();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<FakeGraph*>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete reinterpret_cast<FakeGraph*>(e);
  return cudaSuccess;
}

// one B200: 148 SMs, kernels of 128 registers
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads,
                                                                  size_t, unsigned) {
  *n = 512 / threads;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }

cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "an error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  static char streams[64];
  static int n = 0;
  *s = reinterpret_cast<cudaStream_t>(&streams[n++ % 64]);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  static char event;
  *e = reinterpret_cast<cudaEvent_t>(&event);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) {
  return cudaErrorNotSupported;
}
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorNotSupported; }

}  // extern "C"
