// What the resident launches share: many passes over one lattice in one
// cooperative launch whose CTAs meet at a grid barrier between passes (the
// sweeps of resident.cu, the gradient quench of adjoint.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "chll_common.cuh"
#include "chll_physics.cuh"
#include "sweep.cuh"
#include "sweep_unit.cuh"

namespace chll {

constexpr int kResThreads = 512;  // most threads per CTA, and per SM (128 registers each)

// A wait gives up at its kWaitPolls-th poll.  A lattice with a smaller limit starts
// the count at kWaitPolls less its limit, in kernels of their own (LIMITED): a start
// or a limit from the arguments costs the usual ones up to 3% (128^3 sweeps 23.2 and
// 23.6 us, the quench of 64^3 3.58 and 3.66, open 4.30 and 4.45).
inline uint32_t first_poll(uint32_t wait_limit) {
  return kWaitPolls - std::min(wait_limit, kWaitPolls);
}

// One word per pass, three in rotation, 128 bytes apart: director accepts in
// bits 0-25, flips in bits 26-51, arrived CTAs in bits 52-63.  The word of pass
// q is cleared by the first CTA once the barrier of pass q + 1 is through --
// every CTA has then read it for the last time -- and that CTA's release at
// pass q + 2 puts the clear before any arrival at pass q + 3, its next use.
constexpr int kWordStride = 16;
constexpr int kCountBits = 26;
constexpr unsigned long long kCountMask = (1ull << kCountBits) - 1;
constexpr int kArriveShift = 2 * kCountBits;

// Thread 0 of every CTA adds the CTA's counts and arrival to the pass's word
// (release: the CTA's stores, ordered before it by the CTA barrier, are
// visible to whoever acquires the word) ...
__device__ __forceinline__ void grid_arrive(unsigned long long* w, unsigned long long counts,
                                            uint32_t nct) {
  if (nct == 1) return;
  const unsigned long long add = counts + (1ull << kArriveShift);
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(add) : "memory");
}

// ... and waits until every CTA has (acquire).  Returns the word, or the CTA's
// own counts of a grid of one CTA; ok = false if the wait ran out.
__device__ __forceinline__ unsigned long long grid_wait(unsigned long long* w,
                                                        unsigned long long counts, uint32_t nct,
                                                        uint32_t polls, bool& ok) {
  if (nct == 1) return counts;
  unsigned long long v;
  do {
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w) : "memory");
    if ((uint32_t)(v >> kArriveShift) == nct) return v;
  } while (++polls < kWaitPolls);
  ok = false;
  return v;
}

// Thread 0 of the CTA that arrives last at the launch's last word: nobody waits
// for that one, so all three can be cleared for the next launch.
__device__ __forceinline__ void clear_words(unsigned long long* words) {
  for (int w = 0; w < 3; ++w) words[w * kWordStride] = 0;
}

// One unit per thread: the thread keeps both colours' unit g (the 4-site x-block
// q of row (j, k)) in registers for the whole launch.  The other colour's pair
// then is the x-row pair of walk_task, so a pass loads the +-y and +-z pairs and
// one x neighbour, at addresses fixed for the launch.  ni a multiple of 4, or
// open boundaries (a padding slot reads as the zero of a missing neighbour).
template <bool P>
struct OwnBlock {
  uint32_t g, u, o0;        // unit, its slot, parity of colour 0's sites in the row
  uint32_t yp, ym, zp, zm;  // slots of the neighbour pairs
  uint32_t xm, xp;          // the x neighbours outside the block: below, above
  bool has, hyp, hym, hzp, hzm, hxm, hxp;
  bool v[4];                // sites 4q .. 4q+3 inside the lattice
  float4 n[2][2];           // [colour][slot of the pair]

  __device__ __forceinline__ OwnBlock(const LatticeView& L, const SweepGeom& G) {
    g = blockIdx.x * blockDim.x + threadIdx.x;
    has = g < G.units;
    const uint32_t hx = (uint32_t)L.hx, nj = (uint32_t)L.nj, nk = (uint32_t)L.nk;
    const uint32_t plane = hx * nj;
    const uint32_t row = G.by_Q.div(g), q = g - row * G.Q;
    const uint32_t k = G.by_nj.div(row), j = row - k * nj;
    o0 = (j + k) & 1u;
    u = 2 * g;
    hyp = P || j + 1 < nj;
    hym = P || j > 0;
    hzp = P || k + 1 < nk;
    hzm = P || k > 0;
    hxm = P || q > 0;
    hxp = P || q + 1 < G.Q;
    yp = j + 1 < nj ? u + hx : u - (nj - 1) * hx;
    ym = j > 0 ? u - hx : u + (nj - 1) * hx;
    zp = k + 1 < nk ? u + plane : u - (nk - 1) * plane;
    zm = k > 0 ? u - plane : u + (nk - 1) * plane;
    xm = q > 0 ? u - 1 : u + hx - 1;
    xp = q + 1 < G.Q ? u + 2 : u - 2 * q;
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = has && 4 * q + t < (uint32_t)L.ni;
    n[0][0] = n[0][1] = n[1][0] = n[1][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const UnitSlots s = ld_unit(L.col[c] + u);
        n[c][0] = s.a;
        n[c][1] = s.b;
      }
    }
  }

  // Colour C's sites are 4q+1, 4q+3 rather than 4q, 4q+2.
  template <int C>
  __device__ __forceinline__ bool odd() const {
    return (o0 ^ C) != 0;
  }

  // The neighbours of colour C's two sites; has only.
  template <int C>
  __device__ __forceinline__ void neighbours(const LatticeView& L, Nbrs& nb0, Nbrs& nb1) const {
    const float4* oth = L.col[C ^ 1];
    const bool o = odd<C>();
    nbr_units<kLoadCoherentOrdered>(hyp, oth + yp, nb0.b[2], nb1.b[2]);
    nbr_units<kLoadCoherentOrdered>(hym, oth + ym, nb0.b[3], nb1.b[3]);
    nbr_units<kLoadCoherentOrdered>(hzp, oth + zp, nb0.b[4], nb1.b[4]);
    nbr_units<kLoadCoherentOrdered>(hzm, oth + zm, nb0.b[5], nb1.b[5]);
    float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
    if (o ? hxp : hxm) e = ld4_other<kLoadCoherentOrdered>(oth + (o ? xp : xm));
    const float4 xa = n[C ^ 1][0], xb = n[C ^ 1][1];
    nb0.b[0] = o ? xb : xa;
    nb0.b[1] = o ? xa : e;
    nb1.b[0] = o ? e : xb;
    nb1.b[1] = o ? xb : xa;
  }
};

// One site of each colour per thread, for lattices of at most half a unit per
// thread: slot h of both colour arrays.  In the row, colour C's site has the other
// colour's slot h as one x neighbour (+x where its parity is even) and slot h - 1
// or h + 1 as the other; the slots h of the rows beside are its y and z
// neighbours.  Half of OwnBlock's serial arithmetic per pass: with the grid barrier
// sweeps of 32^3 4.2 against 4.7 us, 48^3 4.7 against 5.1.
template <bool P>
struct OwnSite {
  uint32_t h, g, o0;        // slot, unit, parity of colour 0's site in the row
  uint32_t yp, ym, zp, zm;  // slots of the neighbours
  uint32_t xm, xp;          // slots h - 1, h + 1 (wrapped)
  bool has, hyp, hym, hzp, hzm, hxm, hxp;
  bool v[2];                // sites 2h, 2h+1 of the row inside the lattice
  float4 n[2];              // [colour]

  __device__ __forceinline__ OwnSite(const LatticeView& L, const SweepGeom& G)
      : OwnSite(L, G, blockIdx.x * blockDim.x + threadIdx.x) {}
  __device__ __forceinline__ OwnSite(const LatticeView& L, const SweepGeom& G, uint32_t slot) {
    h = slot;
    g = h >> 1;
    const uint32_t hx = (uint32_t)L.hx, nj = (uint32_t)L.nj, nk = (uint32_t)L.nk;
    const uint32_t plane = hx * nj, wide = P ? (uint32_t)L.ni / 2 : hx;
    const uint32_t row = G.by_Q.div(g), r = h - row * hx;
    has = g < G.units && r < wide;  // periodic: a padding slot is nobody's neighbour
    const uint32_t k = G.by_nj.div(row), j = row - k * nj;
    o0 = (j + k) & 1u;
    hyp = P || j + 1 < nj;
    hym = P || j > 0;
    hzp = P || k + 1 < nk;
    hzm = P || k > 0;
    hxm = P || r > 0;
    hxp = P || r + 1 < wide;
    yp = j + 1 < nj ? h + hx : h - (nj - 1) * hx;
    ym = j > 0 ? h - hx : h + (nj - 1) * hx;
    zp = k + 1 < nk ? h + plane : h - (nk - 1) * plane;
    zm = k > 0 ? h - plane : h + (nk - 1) * plane;
    xm = r > 0 ? h - 1 : h + wide - 1;
    xp = r + 1 < wide ? h + 1 : h - r;
    v[0] = has && 2 * r < (uint32_t)L.ni;
    v[1] = has && 2 * r + 1 < (uint32_t)L.ni;
    n[0] = n[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has) {
      n[0] = ld4_other<kLoadCoherentOrdered>(L.col[0] + h);
      n[1] = ld4_other<kLoadCoherentOrdered>(L.col[1] + h);
    }
  }

  template <int C>
  __device__ __forceinline__ bool odd() const {
    return (o0 ^ C) != 0;
  }

  template <int C>
  __device__ __forceinline__ bool valid() const {
    return odd<C>() ? v[1] : v[0];
  }

  // The neighbours of colour C's site; has only.
  template <int C>
  __device__ __forceinline__ void neighbours(const LatticeView& L, Nbrs& nb) const {
    const float4* oth = L.col[C ^ 1];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool o = odd<C>();
    nb.b[2] = hyp ? ld4_other<kLoadCoherentOrdered>(oth + yp) : zero;
    nb.b[3] = hym ? ld4_other<kLoadCoherentOrdered>(oth + ym) : zero;
    nb.b[4] = hzp ? ld4_other<kLoadCoherentOrdered>(oth + zp) : zero;
    nb.b[5] = hzm ? ld4_other<kLoadCoherentOrdered>(oth + zm) : zero;
    const float4 e = (o ? hxp : hxm) ? ld4_other<kLoadCoherentOrdered>(oth + (o ? xp : xm)) : zero;
    nb.b[0] = o ? e : n[C ^ 1];
    nb.b[1] = o ? n[C ^ 1] : e;
  }

  template <int C>
  __device__ __forceinline__ void store(const LatticeView& L) const {
    asm volatile("st.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(L.col[C] + h), "f"(n[C].x),
                 "f"(n[C].y), "f"(n[C].z), "f"(n[C].w)
                 : "memory");
  }
};

// A site as published to the threads of other CTAs: the director, and the
// chirality's sign beside a number.  One 128-bit access of device scope, so a
// reader that finds the number it waits for has the whole site.
constexpr uint32_t kTagMask = 0x7fffffffu;

__device__ __forceinline__ uint4 ld_word(const uint4* p) {
  unsigned long long lo, hi;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0,%1}, t;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

__device__ __forceinline__ void st_word(uint4* p, const float4& n, uint32_t tag) {
  const uint32_t w = (__float_as_uint(n.w) & 0x80000000u) | (tag & kTagMask);
  const unsigned long long lo = (unsigned long long)__float_as_uint(n.x) |
                                ((unsigned long long)__float_as_uint(n.y) << 32);
  const unsigned long long hi =
      (unsigned long long)__float_as_uint(n.z) | ((unsigned long long)w << 32);
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1,%2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               ::"l"(p), "l"(lo), "l"(hi)
               : "memory");
}

// Streaming multiprocessors of the current device (kResThreads threads of a
// resident launch each).
inline uint32_t resident_sms() {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int>& slot = cache[dev & 63];
  int n = slot.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
    slot.store(n, std::memory_order_relaxed);
  }
  return (uint32_t)n;
}

// Whether OwnBlock (OwnSite) holds the lattice: a unit (site of each colour) per
// thread.  An OwnSite wraps a padded row, an OwnBlock does not.
inline bool one_unit_each(const LatticeView& L, uint32_t units) {
  return units <= resident_sms() * kResThreads && (L.ni % 4 == 0 || !L.periodic);
}
inline bool one_site_each(uint32_t units, uint32_t per_sm = kResThreads) {
  return 2 * units <= resident_sms() * per_sm;
}

// Threads per CTA and CTAs for `items` threads: up to 256 one CTA (two warps per
// scheduler), whose barrier is its own; else spread over the SMs in CTAs of whole
// warps.
inline void resident_shape(uint32_t items, uint32_t& block, uint32_t& ctas,
                           uint32_t per_sm = kResThreads) {
  const uint32_t sms = resident_sms();
  const uint32_t share = items <= 256 ? items : (items + sms - 1) / sms;
  block = std::min<uint32_t>(per_sm, (share + 31) / 32 * 32);
  ctas = std::min((items + block - 1) / block, sms * (per_sm / block));
}

template <class KERNEL, class ARGS>
cudaError_t launch_cooperative(KERNEL kernel, uint32_t ctas, uint32_t block, cudaStream_t stream,
                               const ARGS& args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(block);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

}  // namespace chll
