// Conversions between the caller's natural-order arrays and the red/black
// float4 lattice, and the on-device random initial state.
//
// The reference keeps nx, ny, nz (FP64) and s (int32) as four F-order
// (i fastest) arrays (chll/chll.py:57-61, chll_mod.f90:43-45).  The lattice
// here is one float4 (nx, ny, nz, s) per site split by colour, so a half-sweep
// reads each colour as one coalesced 128-bit stream.  One thread per natural
// site: reads are coalesced, and the writes of a warp land in two contiguous
// runs (one per colour).
//
// The kernels that fill a lattice walk the padded rows and write the padding
// slots' zeros themselves: clearing the lattice first wrote it twice (256^3 from
// device memory: 45 of 134 us; the copy alone is 82 at the measured bandwidth).
#include "chll_common.cuh"
#include "sweep.cuh"

namespace chll {

namespace {

// x / d for 32-bit x as the high word of one 64-bit product with
// floor(2^64 / d) + 1 (Lemire, Kaser, Kurz, "Faster remainder by direct
// computation", 2019).
struct ExactDiv {
  uint32_t d;
  uint64_t m;
  __host__ explicit ExactDiv(uint32_t divisor)
      : d(divisor), m(divisor > 1 ? ~0ull / divisor + 1 : 0) {}
  __device__ __forceinline__ uint32_t div(uint32_t x) const {
    return d > 1 ? (uint32_t)__umul64hi(m, x) : x;
  }
};

// The elements a kernel walks: nj * nk rows of `width` sites (ni, or ni padded
// to the storage rows' 2 hx; fewer than 2^32 in all).
struct Rows {
  uint64_t count;
  ExactDiv by_width, by_nj;
  __host__ Rows(const LatticeView& L, int width)
      : count((uint64_t)width * L.nj * L.nk), by_width((uint32_t)width), by_nj((uint32_t)L.nj) {}
};

struct Site {
  int i, c;         // x coordinate, colour
  uint32_t row;     // j + nj * k
  uint32_t slot;
};

__device__ __forceinline__ Site site_of(const LatticeView& L, const Rows& R, uint64_t e) {
  Site s;
  s.row = R.by_width.div((uint32_t)e);
  s.i = (int)((uint32_t)e - s.row * R.by_width.d);
  const uint32_t k = R.by_nj.div(s.row), j = s.row - k * R.by_nj.d;
  s.c = (int)(((uint32_t)s.i + j + k) & 1u);
  s.slot = s.row * (uint32_t)L.hx + ((uint32_t)s.i >> 1);
  return s;
}

__device__ __forceinline__ size_t natural(const LatticeView& L, const Site& s) {
  return (size_t)s.row * (size_t)L.ni + (size_t)s.i;
}

__global__ void pack_f64_kernel(LatticeView L, Rows R, const double* __restrict__ nx,
                                const double* __restrict__ ny, const double* __restrict__ nz,
                                const int* __restrict__ s) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < R.count;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const Site x = site_of(L, R, t);
    const size_t e = natural(L, x);
    colour_array(L, x.c)[x.slot] =
        x.i < L.ni ? make_float4((float)nx[e], (float)ny[e], (float)nz[e], (float)s[e])
                   : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

__global__ void unpack_f64_kernel(LatticeView L, Rows R, double* __restrict__ nx,
                                  double* __restrict__ ny, double* __restrict__ nz,
                                  int* __restrict__ s) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < R.count;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const Site x = site_of(L, R, t);
    const size_t e = natural(L, x);
    const float4 v = colour_array(L, x.c)[x.slot];
    nx[e] = v.x;
    ny[e] = v.y;
    nz[e] = v.z;
    s[e] = (int)v.w;
  }
}

__global__ void pack_f4_kernel(LatticeView L, Rows R, const float4* __restrict__ src) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < R.count;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const Site x = site_of(L, R, t);
    const size_t e = natural(L, x);
    colour_array(L, x.c)[x.slot] = x.i < L.ni ? src[e] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

__global__ void unpack_f4_kernel(LatticeView L, Rows R, float4* __restrict__ dst) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < R.count;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const Site x = site_of(L, R, t);
    const size_t e = natural(L, x);
    dst[e] = colour_array(L, x.c)[x.slot];
  }
}

// Directors uniform on the sphere (cos(theta) = 2u-1, phi = 2*pi*u', as the
// reference drivers' init_random, scripts/pdanneal.py:5-16) and s = -1 with
// probability 1/2 (chll/chll.py:84-90).  site0: index of the view's first
// site in the whole lattice (a z-slab draws its global sites' values).
__global__ void init_random_kernel(LatticeView L, Rows R, uint32_t key0, uint32_t key1,
                                   uint32_t replica, uint64_t site0) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < R.count;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const Site x = site_of(L, R, t);
    const size_t e = natural(L, x);
    Ctr4 c = {{(uint32_t)(e + site0), 0xffffffffu, replica, kStreamInit}};
    const Ctr4 r = philox4x32_10(c, key0, key1);
    const float ct = 2.0f * u01(r.v[0]) - 1.0f;
    const float st = sqrtf(fmaxf(0.f, 1.0f - ct * ct));
    float sp, cp;
    sincospif(2.0f * u01(r.v[1]), &sp, &cp);
    const float s = (u01(r.v[2]) < 0.5f) ? -1.0f : 1.0f;
    colour_array(L, x.c)[x.slot] =
        x.i < L.ni ? make_float4(st * cp, st * sp, ct, s) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

unsigned int grid_for(size_t n) {
  const size_t b = (n + 255) / 256;
  return (unsigned int)(b < 148 * 16 ? (b ? b : 1) : 148 * 16);
}

}  // namespace

void launch_pack_f64(const LatticeView& L, const double* nx, const double* ny, const double* nz,
                     const int* s, cudaStream_t stream) {
  const Rows R(L, padded_ni(L.ni));
  pack_f64_kernel<<<grid_for(R.count), 256, 0, stream>>>(L, R, nx, ny, nz, s);
}

void launch_unpack_f64(const LatticeView& L, double* nx, double* ny, double* nz, int* s,
                       cudaStream_t stream) {
  const Rows R(L, L.ni);
  unpack_f64_kernel<<<grid_for(R.count), 256, 0, stream>>>(L, R, nx, ny, nz, s);
}

void launch_pack_f4(const LatticeView& L, const float4* xyzs, cudaStream_t stream) {
  const Rows R(L, padded_ni(L.ni));
  pack_f4_kernel<<<grid_for(R.count), 256, 0, stream>>>(L, R, xyzs);
}

void launch_unpack_f4(const LatticeView& L, float4* xyzs, cudaStream_t stream) {
  const Rows R(L, L.ni);
  unpack_f4_kernel<<<grid_for(R.count), 256, 0, stream>>>(L, R, xyzs);
}

void launch_init_random(const LatticeView& L, uint32_t key0, uint32_t key1, uint32_t replica,
                        cudaStream_t stream, uint64_t site0) {
  const Rows R(L, padded_ni(L.ni));
  init_random_kernel<<<grid_for(R.count), 256, 0, stream>>>(L, R, key0, key1, replica, site0);
}

}  // namespace chll
