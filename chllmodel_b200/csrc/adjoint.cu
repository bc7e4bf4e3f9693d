// Adjoint of the lattice energy: dE/dn_i for every director and dE/d(eps,K,h).
//
// Total energy (each bond once, the sweep's boundary):
//   E = sum_<ij>, j=i+e_a [ eps*(1 - c^2) - K*c*X*sbar ] - h*sum_i s_i,
//   c = n_i.n_j,  X = (n_i x n_j).e_a = n_i.(n_j x e_a),  sbar = (s_i+s_j)/2.
// This is the bond sum behind the reference's local energy (chll_mod.f90:
// 363-412): the local energy of a site is the sum of the bonds touching it.
// Per bond, seen from site i with neighbour b in direction sigma*e_a
// (sigma = -1 forward, +1 backward):
//   dE_b/dn_i = -2*eps*c*b + sigma*K*sbar*(X*b + c*(b x e_a)),
// with c = n_i.b and X = (n_i x b).e_a.  The director gradient is optionally
// projected on the tangent plane, g - (g.n) n/|n|^2 (the torque direction).
// Coupling derivatives (FP64): dE/deps = sum(1-c^2), dE/dK = -sum(c*X*sbar),
// dE/dh = -sum(s), together with E itself.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "chll_common.cuh"
#include "moments.cuh"
#include "resident.cuh"
#include "sweep.cuh"
#include "sweep_unit.cuh"

namespace chll {

namespace {

constexpr int kGradThreads = 256;

// Slot t of colour `col` -> lattice site (i, j, k), with 32-bit divisions by
// multiplication (a colour holds < 2^31 slots); false for a padding slot.
__device__ __forceinline__ bool slot_site(const LatticeView& L, const MomentGeom& M, int col,
                                          uint32_t t, int& i, int& j, int& k) {
  const uint32_t r = M.by_hx.div(t);
  const int h = (int)(t - r * (uint32_t)L.hx);
  k = (int)M.by_nj.div(r);
  j = (int)(r - (uint32_t)k * (uint32_t)L.nj);
  i = 2 * h + ((col + j + k) & 1);
  return i < L.ni;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Adds one bond's dE/dn_i to (gx,gy,gz).  AXIS: 0,1,2; sigma = -1 forward.
template <int AXIS>
__device__ __forceinline__ void bond_grad(const float4& n, const float4& b, float sigma,
                                          const Coupling& cp, float& gx, float& gy, float& gz) {
  const float c = n.x * b.x + n.y * b.y + n.z * b.z;
  float X, ex, ey, ez;  // X = (n x b).e_a; (ex,ey,ez) = b x e_a
  if (AXIS == 0) {
    X = n.y * b.z - n.z * b.y;
    ex = 0.f; ey = b.z; ez = -b.y;
  } else if (AXIS == 1) {
    X = n.z * b.x - n.x * b.z;
    ex = -b.z; ey = 0.f; ez = b.x;
  } else {
    X = n.x * b.y - n.y * b.x;
    ex = b.y; ey = -b.x; ez = 0.f;
  }
  const float sbar = 0.5f * (n.w + b.w);
  const float a = -2.f * cp.eps * c;
  const float w = sigma * cp.K * sbar;
  gx += a * b.x + w * (X * b.x + c * ex);
  gy += a * b.y + w * (X * b.y + c * ey);
  gz += a * b.z + w * (X * b.z + c * ez);
}

// dE/dn of one site from its six neighbours (+x, -x, +y, -y, +z, -z; zero
// past an open boundary), optionally projected on the tangent plane.
__device__ __forceinline__ float4 site_grad(const float4& n, const float4& bxp, const float4& bxm,
                                            const float4& byp, const float4& bym,
                                            const float4& bzp, const float4& bzm,
                                            const Coupling& cp, int project) {
  float gx = 0.f, gy = 0.f, gz = 0.f;
  bond_grad<0>(n, bxp, -1.f, cp, gx, gy, gz);
  bond_grad<0>(n, bxm, +1.f, cp, gx, gy, gz);
  bond_grad<1>(n, byp, -1.f, cp, gx, gy, gz);
  bond_grad<1>(n, bym, +1.f, cp, gx, gy, gz);
  bond_grad<2>(n, bzp, -1.f, cp, gx, gy, gz);
  bond_grad<2>(n, bzm, +1.f, cp, gx, gy, gz);
  if (project) {
    const float nn = n.x * n.x + n.y * n.y + n.z * n.z;
    const float gn = (gx * n.x + gy * n.y + gz * n.z) / nn;
    gx -= gn * n.x;
    gy -= gn * n.y;
    gz -= gn * n.z;
  }
  return make_float4(gx, gy, gz, 0.f);
}

// FP64 sums of one site: its forward bonds (+x, +y, +z, each bond of the
// lattice once; hx, hy, hz = present) and its field term.
__device__ __forceinline__ void site_sums(const float4& n, const float4& bx, const float4& by,
                                          const float4& bz, bool hx, bool hy, bool hz,
                                          const CouplingD& cd, double acc[4]) {
  const double nx = n.x, ny = n.y, nz = n.z, s = n.w;
  const float4 fw[3] = {bx, by, bz};
  const bool hf[3] = {hx, hy, hz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!hf[a]) continue;
    const float4 b = fw[a];
    const double c = nx * b.x + ny * b.y + nz * b.z;
    const double X = (a == 0) ? ny * b.z - nz * b.y
                   : (a == 1) ? nz * b.x - nx * b.z
                              : nx * b.y - ny * b.x;
    const double sbar = 0.5 * (s + (double)b.w);
    const double nem = 1.0 - c * c;
    const double chi = -c * X * sbar;
    acc[0] += cd.eps * nem + cd.K * chi;
    acc[1] += nem;
    acc[2] += chi;
  }
  acc[0] -= cd.g * s;
  acc[3] -= s;
}

// Block sums of the four FP64 accumulators into partials; the last block to
// finish (ticket) adds the partials into out4 with all its threads (blocks
// strided over the threads, then warp shuffles and the warps in order: a
// fixed order for a given grid, so the sums are reproducible).
__device__ __forceinline__ void finish_sums(const double acc[4], double* __restrict__ partials,
                                            unsigned int* __restrict__ ticket,
                                            double* __restrict__ out4) {
  __shared__ double s_part[kGradThreads / 32][4];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const double v = warp_sum(acc[m]);
    if (lane == 0) s_part[warp][m] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int w = 0; w < kGradThreads / 32; ++w) v += s_part[w][threadIdx.x];
    partials[(size_t)blockIdx.x * 4 + threadIdx.x] = v;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
#pragma unroll
    for (int m = 0; m < 4; ++m) v[m] += __ldcg(&partials[(size_t)b * 4 + m]);  // L2
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const double w = warp_sum(v[m]);
    if (lane == 0) s_part[warp][m] = w;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int w = 0; w < kGradThreads / 32; ++w) t += s_part[w][threadIdx.x];
    out4[threadIdx.x] = t;
  }
  if (threadIdx.x == 0) *ticket = 0;
}

// One slot per thread: colour arrays that are 16-byte aligned but not 32
// (caller-provided arrays of chll_energy_grad_noalloc; every slot is read as
// one float4).
__global__ void __launch_bounds__(kGradThreads)
    energy_grad_site_kernel(LatticeView L, MomentGeom M, CouplingD cd, float4* __restrict__ grad_rb,
                       int project,
                       double* __restrict__ partials, unsigned int* __restrict__ ticket,
                       double* __restrict__ out4) {
  Coupling cp;  // FP32 couplings of the per-site gradient
  cp.eps = (float)cd.eps;
  cp.K = (float)cd.K;
  cp.g = (float)cd.g;
  cp.inv_kT = 0.f;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};  // E, dE/deps, dE/dK, dE/dh
  const uint64_t total = 2 * (uint64_t)M.per_colour;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const int col = e >= M.per_colour;
    const uint32_t t = (uint32_t)e - (col ? M.per_colour : 0u);
    int i, j, k;
    if (!slot_site(L, M, col, t, i, j, k)) {
      if (grad_rb) grad_rb[e] = zero;
      continue;
    }
    const float4 n = colour_array(L, col)[t];
    int ip = i + 1, im = i - 1, jp = j + 1, jm = j - 1, kp = k + 1, km = k - 1;
    bool hip = ip < L.ni, him = im >= 0, hjp = jp < L.nj, hjm = jm >= 0, hkp = kp < L.nk,
         hkm = km >= 0;
    if (L.periodic) {
      if (!hip) ip = 0;
      if (!him) im = L.ni - 1;
      if (!hjp) jp = 0;
      if (!hjm) jm = L.nj - 1;
      if (!hkp) kp = 0;
      if (!hkm) km = L.nk - 1;
      hip = him = hjp = hjm = hkp = hkm = true;
    }
    const float4 bxp = hip ? site_at(L, ip, j, k) : zero;
    const float4 bxm = him ? site_at(L, im, j, k) : zero;
    const float4 byp = hjp ? site_at(L, i, jp, k) : zero;
    const float4 bym = hjm ? site_at(L, i, jm, k) : zero;
    const float4 bzp = hkp ? site_at(L, i, j, kp) : zero;
    const float4 bzm = hkm ? site_at(L, i, j, km) : zero;

    if (grad_rb) grad_rb[e] = site_grad(n, bxp, bxm, byp, bym, bzp, bzm, cp, project);
    site_sums(n, bxp, byp, bzp, hip, hjp, hkp, cd, acc);
  }

  finish_sums(acc, partials, ticket, out4);
}

// Two sites per thread on the sweep's unit gather (256-bit accesses): colour
// 0's units, then colour 1's.  Needs 32-byte aligned colour and gradient
// arrays (unit_view_aligned).
template <int C, bool PERIODIC>
__device__ __forceinline__ void grad_units(const LatticeView& L, const SweepGeom& G,
                                           const Coupling& cp, const CouplingD& cd,
                                           float4* __restrict__ grad_c, int project,
                                           double acc[4]) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t g = blockIdx.x * kGradThreads + threadIdx.x; g < G.units;
       g += gridDim.x * kGradThreads) {
    UnitNbhd U;
    gather_unit<C, PERIODIC, PERIODIC>(L, G, g, U);
    float4 g0 = zero, g1 = zero;
    if (U.v0) {
      if (grad_c)
        g0 = site_grad(U.n0, U.nb0.b[0], U.nb0.b[1], U.nb0.b[2], U.nb0.b[3], U.nb0.b[4],
                       U.nb0.b[5], cp, project);
      site_sums(U.n0, U.nb0.b[0], U.nb0.b[2], U.nb0.b[4], U.fx0, U.fy, U.fz, cd, acc);
    }
    if (U.v1) {
      if (grad_c)
        g1 = site_grad(U.n1, U.nb1.b[0], U.nb1.b[1], U.nb1.b[2], U.nb1.b[3], U.nb1.b[4],
                       U.nb1.b[5], cp, project);
      site_sums(U.n1, U.nb1.b[0], U.nb1.b[2], U.nb1.b[4], U.fx1, U.fy, U.fz, cd, acc);
    }
    if (grad_c) st_unit(grad_c + (U.cen - L.col[C]), g0, g1);
  }
}

template <bool PERIODIC>
__global__ void __launch_bounds__(kGradThreads)
    energy_grad_unit_kernel(LatticeView L, SweepGeom G, CouplingD cd,
                            float4* __restrict__ grad_rb, uint32_t per_colour, int project,
                            double* __restrict__ partials, unsigned int* __restrict__ ticket,
                            double* __restrict__ out4) {
  Coupling cp;  // FP32 couplings of the per-site gradient
  cp.eps = (float)cd.eps;
  cp.K = (float)cd.K;
  cp.g = (float)cd.g;
  cp.inv_kT = 0.f;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};  // E, dE/deps, dE/dK, dE/dh
  grad_units<0, PERIODIC>(L, G, cp, cd, grad_rb, project, acc);
  grad_units<1, PERIODIC>(L, G, cp, cd, grad_rb ? grad_rb + per_colour : nullptr, project, acc);
  finish_sums(acc, partials, ticket, out4);
}

// ---------------------------------------------------------------------------
// The adjoint of caller arrays in natural order (i fastest): directors n
// (N x 3) and chiralities s (N), FP32, as the autograd wrapper has them.
//
// The path through a red/black lattice read and wrote the state five more times
// (records packed together, a cleared lattice, the red/black copy, the
// gradient unpacked and its fourth column cut off); here a call reads each
// array once and writes the (N x 3) gradient once: 28 B per site.
//
// A thread walks one column (i, j) over a run of planes and carries its site
// and the two z neighbours in registers, with the FP64 forms of its site from
// the step before (the conversions are a quarter-rate pipe: 12 per site instead
// of 16).  A warp holds 32 consecutive columns of the flattened plane, so a
// load of a component is three whole lines per warp whatever ni is, and the x
// neighbours come from the lanes beside; the ends of a warp or a row load
// theirs.
// ---------------------------------------------------------------------------
struct NaturalGeom {
  uint32_t ni, nj, nk;
  uint32_t plane;      // ni * nj, columns
  uint32_t cols;       // columns rounded up to whole warps
  uint32_t seg, nseg;  // planes per task, tasks per column
};

struct Site64 {
  double x, y, z, s;
};

__device__ __forceinline__ Site64 to64(const float4& v) {
  return {(double)v.x, (double)v.y, (double)v.z, (double)v.w};
}

// Site e of fewer than 2^32: 32-bit indices, widened once per address.
__device__ __forceinline__ float4 natural_site(const float* __restrict__ n,
                                               const float* __restrict__ s, uint32_t e) {
  const float* const p = n + 3ull * e;
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(s + e));
}

// One forward bond's FP64 terms: acc[0] the sum of 1 - c^2, acc[1] that of
// c X (s + s').
template <int AXIS>
__device__ __forceinline__ void bond_sums64(const Site64& n, const Site64& b, double acc[3]) {
  const double c = n.x * b.x + n.y * b.y + n.z * b.z;
  const double X = AXIS == 0 ? n.y * b.z - n.z * b.y
                 : AXIS == 1 ? n.z * b.x - n.x * b.z
                             : n.x * b.y - n.y * b.x;
  acc[0] += 1.0 - c * c;
  acc[1] += c * X * (n.s + b.s);
}

// One bond's dE/dn_i as coefficients of the neighbour and of b x e_a:
// (-2 eps c + w X) b + (w c) (b x e_a) with w = sigma K sbar, in half the
// instructions of bond_grad's term by term form (m2eps = -2 eps, kw = sigma
// K / 2).  Adds the second part to g and returns the first one's coefficient,
// so that the smaller parts are summed before the larger ones.  A bond that is
// not there (has) has zero coefficients.
template <int AXIS, bool ALWAYS>
__device__ __forceinline__ float bond_grad_part(const float4& n, const float4& b, bool has,
                                                float m2eps, float kw, float& gx, float& gy,
                                                float& gz) {
  const float c = n.x * b.x + n.y * b.y + n.z * b.z;
  const float X = AXIS == 0 ? n.y * b.z - n.z * b.y
                : AXIS == 1 ? n.z * b.x - n.x * b.z
                            : n.x * b.y - n.y * b.x;
  const float w = kw * (n.w + b.w);
  const float q = ALWAYS || has ? w * c : 0.f;
  if (AXIS == 0) {
    gy += q * b.z;
    gz -= q * b.y;
  } else if (AXIS == 1) {
    gz += q * b.x;
    gx -= q * b.z;
  } else {
    gx += q * b.y;
    gy -= q * b.x;
  }
  const float p = w * X + m2eps * c;
  return ALWAYS || has ? p : 0.f;
}

__device__ __forceinline__ void add_scaled(float p, const float4& b, float& gx, float& gy,
                                           float& gz) {
  gx += p * b.x;
  gy += p * b.y;
  gz += p * b.z;
}

// A neighbour that is not there is read as the site itself, so that no load is
// conditional, and its bond left out.
template <bool GRAD, bool PER>
__global__ void __launch_bounds__(kGradThreads)
    natural_grad_kernel(NaturalGeom G, const float* __restrict__ n, const float* __restrict__ s,
                        CouplingD cd, float* __restrict__ grad, int project,
                        double* __restrict__ partials) {
  const float m2eps = -2.f * (float)cd.eps, kw = 0.5f * (float)cd.K;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t ntasks = (uint64_t)G.cols * G.nseg;
  double acc[3] = {0.0, 0.0, 0.0};  // bond_sums64's two, then the sum of s
  for (uint64_t t = blockIdx.x * (uint64_t)kGradThreads + threadIdx.x; t < ntasks;
       t += (uint64_t)gridDim.x * kGradThreads) {
    // whole warps share a segment: the same planes in every lane
    const uint32_t sg = (uint32_t)(t / G.cols);
    const uint32_t p0 = (uint32_t)(t - (uint64_t)sg * G.cols);
    const bool has = p0 < G.plane;
    const uint32_t p = has ? p0 : G.plane - 1;
    const uint32_t j = p / G.ni, i = p - j * G.ni;
    const uint32_t k0 = sg * G.seg, k1 = min(k0 + G.seg, G.nk);
    const bool hxp = PER || i + 1 < G.ni, hxm = PER || i > 0;
    const bool hyp = PER || j + 1 < G.nj, hym = PER || j > 0;
    // columns of the in-plane neighbours
    const uint32_t cxp = i + 1 < G.ni ? p + 1 : (PER ? p - i : p);
    const uint32_t cxm = i > 0 ? p - 1 : (PER ? p + (G.ni - 1) : p);
    const uint32_t cyp = j + 1 < G.nj ? p + G.ni : (PER ? i : p);
    const uint32_t cym = j > 0 ? p - G.ni : (PER ? p + (G.nj - 1) * G.ni : p);
    // whose x neighbours are not in the lanes beside
    const bool lxp = lane == 31 || p0 + 1 >= G.plane || i + 1 == G.ni;
    const bool lxm = lane == 0 || i == 0;
    const uint32_t last = (G.nk - 1) * G.plane;  // first site of the last plane
    uint32_t base = k0 * G.plane;                // of this plane
    float4 c = natural_site(n, s, base + p);
    float4 zm = c;
    if (GRAD)
      zm = natural_site(n, s, (k0 > 0 ? base - G.plane : (PER ? last : base)) + p);
    Site64 c64 = to64(c);
    for (uint32_t k = k0; k < k1; ++k, base += G.plane) {
      const bool hzp = PER || k + 1 < G.nk, hzm = PER || k > 0;
      if (k + 2 < G.nk) {  // the plane after the next: the lines no thread has read yet
        const uint32_t e = base + 2 * G.plane + p;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(n + 3ull * e));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(s + e));
      }
      const float4 zp =
          natural_site(n, s, (k + 1 < G.nk ? base + G.plane : (PER ? 0u : base)) + p);
      const float4 yp = natural_site(n, s, base + cyp);
      float4 ym = yp;
      if (GRAD) ym = natural_site(n, s, base + cym);
      float4 xp, xm = c;
      xp.x = __shfl_down_sync(0xffffffffu, c.x, 1);
      xp.y = __shfl_down_sync(0xffffffffu, c.y, 1);
      xp.z = __shfl_down_sync(0xffffffffu, c.z, 1);
      xp.w = __shfl_down_sync(0xffffffffu, c.w, 1);
      if (lxp) xp = natural_site(n, s, base + cxp);
      if (GRAD) {
        xm.x = __shfl_up_sync(0xffffffffu, c.x, 1);
        xm.y = __shfl_up_sync(0xffffffffu, c.y, 1);
        xm.z = __shfl_up_sync(0xffffffffu, c.z, 1);
        xm.w = __shfl_up_sync(0xffffffffu, c.w, 1);
        if (lxm) xm = natural_site(n, s, base + cxm);
      }
      const Site64 zp64 = to64(zp);
      if (has) {
        if (GRAD) {
          float gx = 0.f, gy = 0.f, gz = 0.f;
          const float pxp = bond_grad_part<0, PER>(c, xp, hxp, m2eps, -kw, gx, gy, gz);
          const float pxm = bond_grad_part<0, PER>(c, xm, hxm, m2eps, kw, gx, gy, gz);
          const float pyp = bond_grad_part<1, PER>(c, yp, hyp, m2eps, -kw, gx, gy, gz);
          const float pym = bond_grad_part<1, PER>(c, ym, hym, m2eps, kw, gx, gy, gz);
          const float pzp = bond_grad_part<2, PER>(c, zp, hzp, m2eps, -kw, gx, gy, gz);
          const float pzm = bond_grad_part<2, PER>(c, zm, hzm, m2eps, kw, gx, gy, gz);
          add_scaled(pxp, xp, gx, gy, gz);
          add_scaled(pxm, xm, gx, gy, gz);
          add_scaled(pyp, yp, gx, gy, gz);
          add_scaled(pym, ym, gx, gy, gz);
          add_scaled(pzp, zp, gx, gy, gz);
          add_scaled(pzm, zm, gx, gy, gz);
          if (project) {
            const float nn = c.x * c.x + c.y * c.y + c.z * c.z;
            const float gn = (gx * c.x + gy * c.y + gz * c.z) / nn;
            gx -= gn * c.x;
            gy -= gn * c.y;
            gz -= gn * c.z;
          }
          float* out = grad + 3ull * (base + p);
          out[0] = gx;
          out[1] = gy;
          out[2] = gz;
        }
        if (hxp) bond_sums64<0>(c64, to64(xp), acc);
        if (hyp) bond_sums64<1>(c64, to64(yp), acc);
        if (hzp) bond_sums64<2>(c64, zp64, acc);
        acc[2] += c64.s;
      }
      zm = c;
      c = zp;
      c64 = zp64;
    }
  }
  __shared__ double s_part[kGradThreads / 32][3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double v = warp_sum(acc[m]);
    if (lane == 0) s_part[threadIdx.x >> 5][m] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int w = 0; w < kGradThreads / 32; ++w)
      for (int m = 0; m < 3; ++m) v[m] += s_part[w][m];
    double* out = partials + (size_t)blockIdx.x * 4;  // E, dE/d(eps, K, h)
    out[1] = v[0];
    out[2] = -0.5 * v[1];
    out[3] = -v[2];
    out[0] = cd.eps * out[1] + cd.K * out[2] + cd.g * out[3];
  }
}

// The CTA partials summed in a fixed order: E, then dE/d(eps, K, h).
__global__ void __launch_bounds__(kGradThreads)
    natural_sums_kernel(const double* __restrict__ partials, uint32_t rows,
                        double* __restrict__ energy, double* __restrict__ derivs) {
  __shared__ double s_part[kGradThreads / 32][4];
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  wait_prerequisite_grids();
  for (uint32_t b = threadIdx.x; b < rows; b += kGradThreads) {
#pragma unroll
    for (int m = 0; m < 4; ++m) v[m] += __ldcg(&partials[(size_t)b * 4 + m]);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const double w = warp_sum(v[m]);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5][m] = w;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int w = 0; w < kGradThreads / 32; ++w) t += s_part[w][threadIdx.x];
    if (threadIdx.x == 0) *energy = t;
    else derivs[threadIdx.x - 1] = t;
  }
}

// Every product and sum of a quench step is an explicit fmaf / __fmul_rn /
// __fadd_rn, so that the pass kernel and the resident forms round alike: a quench
// amplifies a rounding along the lattice's soft modes, and forms that contracted
// differently would end in different states of one lattice.

// x0 y0 + x1 y1 + x2 y2; SECOND: the second product is the rounded one of the
// first two.
template <bool SECOND>
__device__ __forceinline__ float quench_dot(float x0, float y0, float x1, float y1, float x2,
                                            float y2) {
  const float t = SECOND ? fmaf(x0, y0, __fmul_rn(x1, y1)) : fmaf(x1, y1, __fmul_rn(x0, y0));
  return fmaf(x2, y2, t);
}

// One bond's dE/dn_i (bond_grad) added to g.
template <int AXIS, bool SECOND>
__device__ __forceinline__ void quench_bond(const float4& n, const float4& b, float m2eps, float sk,
                                            float g[3], bool second = SECOND) {
  constexpr int p = (AXIS + 1) % 3, q = (AXIS + 2) % 3;
  const float nv[3] = {n.x, n.y, n.z}, bv[3] = {b.x, b.y, b.z};
  const float c = SECOND || second ? quench_dot<true>(n.x, b.x, n.y, b.y, n.z, b.z)
                                   : quench_dot<false>(n.x, b.x, n.y, b.y, n.z, b.z);
  const float X = fmaf(nv[p], bv[q], -__fmul_rn(nv[q], bv[p]));
  const float a = __fmul_rn(m2eps, c);
  const float w = __fmul_rn(sk, __fmul_rn(0.5f, __fadd_rn(n.w, b.w)));
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    // component t of X b + c (b x e_a)
    const float e = t == p ? bv[q] : -bv[p];
    const float u = t == AXIS ? __fmul_rn(X, bv[t]) : fmaf(X, bv[t], __fmul_rn(c, e));
    g[t] = __fadd_rn(g[t], fmaf(a, bv[t], __fmul_rn(w, u)));
  }
}

// One site of a zero-temperature gradient quench: n moves against its
// tangent-projected energy gradient, n <- normalise(n - eta (I - n n^T) dE/dn),
// with the neighbours nb (+x, -x, +y, -y, +z, -z) held fixed.  Which product of a
// bond's dot product is rounded on its own differs between the boundaries and,
// for -z, between a unit's sites (second: the unit's second one).  The physics does
// not ask for it: these are the roundings of the pass kernel as it was first
// compiled, kept so that a quench still ends in the state it ended in before.
template <bool P>
__device__ __forceinline__ float4 quench_site(float4 n, const Nbrs& nb, const Coupling& cp,
                                              float eta, bool second) {
  const float m2eps = __fmul_rn(-2.f, cp.eps);
  float g[3] = {0.f, 0.f, 0.f};
  quench_bond<0, true>(n, nb.b[0], m2eps, -cp.K, g);
  quench_bond<0, true>(n, nb.b[1], m2eps, cp.K, g);
  quench_bond<1, P>(n, nb.b[2], m2eps, -cp.K, g);
  quench_bond<1, P>(n, nb.b[3], m2eps, cp.K, g);
  quench_bond<2, P>(n, nb.b[4], m2eps, -cp.K, g);
  quench_bond<2, P>(n, nb.b[5], m2eps, cp.K, g, second);
  const float nn = quench_dot<true>(n.x, n.x, n.y, n.y, n.z, n.z);
  const float gn = __fdiv_rn(quench_dot<true>(g[0], n.x, g[1], n.y, g[2], n.z), nn);
  const float x = fmaf(-eta, fmaf(-gn, n.x, g[0]), n.x);
  const float y = fmaf(-eta, fmaf(-gn, n.y, g[1]), n.y);
  const float z = fmaf(-eta, fmaf(-gn, n.z, g[2]), n.z);
  const float rn = rsqrtf(quench_dot<true>(x, x, y, y, z, z));
  n.x = __fmul_rn(x, rn);
  n.y = __fmul_rn(y, rn);
  n.z = __fmul_rn(z, rn);
  return n;
}

// One colour of the quench: every site of colour C moves with the other
// colour fixed, so the two colours alternate like the Metropolis half-sweeps.
// A thread takes the sweep's unit of two same-colour sites (gather_unit,
// 256-bit accesses).  Chiralities are not changed.
template <int C, bool PERIODIC>
__global__ void __launch_bounds__(kGradThreads) quench_pass_kernel(LatticeView L, SweepGeom G,
                                                                   Coupling cp, float eta) {
  for (uint32_t g = blockIdx.x * kGradThreads + threadIdx.x; g < G.units;
       g += gridDim.x * kGradThreads) {
    UnitNbhd U;
    gather_unit<C, PERIODIC, PERIODIC>(L, G, g, U);
    if (U.v0) U.n0 = quench_site<PERIODIC>(U.n0, U.nb0, cp, eta, false);
    if (U.v1) U.n1 = quench_site<PERIODIC>(U.n1, U.nb1, cp, eta, true);
    st_unit(U.cen, U.n0, U.n1);
  }
}

// The same steps in one cooperative launch (resident.cuh): a step is a pass of
// each colour with a barrier after it.  For lattices of one CTA, whose barrier is
// the CTA's own, and for those of more units than threads.
struct QuenchArgs {
  LatticeView L;
  SweepGeom G;
  Coupling cp;
  float eta;
  Control* ctl;
  unsigned long long* words;
  int nsteps;
  uint32_t first_poll;
};

struct NoOwn {
  __device__ __forceinline__ NoOwn(const LatticeView&, const SweepGeom&) {}
};

// SITE: one site of each colour per thread (one CTA); else the unit loop.
template <bool P, bool SITE, bool LIMITED>
__global__ void __launch_bounds__(kResThreads, 1)
    quench_resident_kernel(const __grid_constant__ QuenchArgs A) {
  __shared__ int s_ok;
  if (A.ctl->status) return;  // an earlier wait ran out: the words are not to be trusted
  const bool lead = threadIdx.x == 0;
  std::conditional_t<SITE, OwnSite<P>, NoOwn> B(A.L, A.G);
  uint32_t slot = 0;
  auto pass = [&](auto colour) {
    constexpr int C = decltype(colour)::value;
    if constexpr (SITE) {
      if (!B.has) return;
      Nbrs nb;
      B.template neighbours<C>(A.L, nb);
      if (B.template valid<C>())
        B.n[C] = quench_site<P>(B.n[C], nb, A.cp, A.eta, (B.h & 1u) != 0);
      B.template store<C>(A.L);
    } else {
      for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < A.G.units;
           g += gridDim.x * blockDim.x) {
        UnitNbhd U;
        gather_unit<C, P, P, false, kLoadCoherentOrdered>(A.L, A.G, g, U);
        if (U.v0) U.n0 = quench_site<P>(U.n0, U.nb0, A.cp, A.eta, false);
        if (U.v1) U.n1 = quench_site<P>(U.n1, U.nb1, A.cp, A.eta, true);
        st_unit(U.cen, U.n0, U.n1);
      }
    }
  };
  // false in every thread if the wait ran out
  auto meet = [&]() {
    __syncthreads();  // the CTA's stores before thread 0's release
    if (lead) {
      bool ok = true;
      grid_arrive(A.words + slot * kWordStride, 0, gridDim.x);
      grid_wait(A.words + slot * kWordStride, 0, gridDim.x, LIMITED ? A.first_poll : 0u, ok);
      if (blockIdx.x == 0) A.words[(slot == 0 ? 2 : slot - 1) * kWordStride] = 0;
      if (!ok) set_status(A.ctl, 4u);
      s_ok = ok;
    }
    slot = slot == 2 ? 0 : slot + 1;
    __syncthreads();
    return s_ok != 0;
  };
  for (int s = 0; s < A.nsteps; ++s) {
    pass(std::integral_constant<int, 0>());
    if (!meet()) return;
    pass(std::integral_constant<int, 1>());
    if (s + 1 < A.nsteps && !meet()) return;
  }
  if (lead && gridDim.x > 1) {
    const unsigned long long old = atomicAdd(A.words + slot * kWordStride, 1ull << kArriveShift);
    if ((uint32_t)(old >> kArriveShift) == gridDim.x - 1) clear_words(A.words);
  }
}

// The same without the grid barrier, for lattices of up to a site of each colour
// (N = 1) or a unit (N = 2) per thread: a thread waits for its neighbours' sites,
// as flow.cu's sweeps.  Those of its own CTA, most of an x-y neighbourhood, come
// through shared memory and a CTA barrier; the others are published words.  What
// bounds a pass is a word's way to L2 and back, and beyond a site per thread the
// words' bandwidth.  us per step on one B200, with the grid barrier and here:
//
//   periodic   16^3   30^3   32^3   48^3   64^3    open  33x31x17  48^3   65x63x61
//   barrier    3.41   4.13   3.49   3.95   5.49          3.58      4.14   5.77
//   here       1.81   1.96   1.78   2.11   3.58          2.18      2.25   4.44
//
// (With the z neighbours' chiralities loaded in every pass, 16 bytes apart, as the
// other remote ones' still are, a unit each: 64^3 4.35 against 4.25, 65x63x61 4.72.)
// T threads per SM: 512 with 128 registers, and periodic up to 896 with 72, where a
// site each is still faster than a unit each though 100 bytes spill.  Spills wait
// behind the polls: a form with a kilobyte of them took 18.8 us at 64^3.
constexpr int kQuenchWide = 896;  // threads of 72 registers per SM

struct QuenchFlowArgs {
  QuenchArgs Q;
  uint4* xch;
  uint32_t* epoch;
  uint32_t per_colour;
};

__device__ __forceinline__ float4 as_site(const uint4& w) {
  return make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z),
                     __uint_as_float(w.w));
}
__device__ __forceinline__ uint4 as_word(const float4& n) {
  return make_uint4(__float_as_uint(n.x), __float_as_uint(n.y), __float_as_uint(n.z),
                    __float_as_uint(n.w));
}

template <bool P, int N, int T, bool LIMITED>
struct QuenchFlow {
  using Own = std::conditional_t<N == 1, OwnSite<P>, OwnBlock<P>>;
  const QuenchFlowArgs& A;
  float4 (&sites)[2][N * T];
  volatile int& lost;
  Own B;
  float zs[2][2][N];  // [colour][+z, -z]: the neighbours' chiralities, which do not change

  __device__ __forceinline__ QuenchFlow(const QuenchFlowArgs& a, float4 (&s)[2][N * T],
                                        volatile int& l)
      : A(a), sites(s), lost(l), B(a.Q.L, a.Q.G) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int t = 0; t < N; ++t) {
        zs[c][0][t] = B.has && B.hzp ? A.Q.L.col[c ^ 1][B.zp + t].w : 0.f;
        zs[c][1][t] = B.has && B.hzm ? A.Q.L.col[c ^ 1][B.zm + t].w : 0.f;
      }
    }
  }

  __device__ __forceinline__ uint32_t slot() const {
    if constexpr (N == 1) return B.h;
    else return B.u;
  }
  template <int C>
  __device__ __forceinline__ float4& own(int t) {
    if constexpr (N == 1) return B.n[C];
    else return B.n[C][t];
  }

  // The neighbours of colour C's sites, the other CTAs' as published with `tag`.
  template <int C>
  __device__ __forceinline__ void neighbours(uint32_t tag, Nbrs (&nb)[N]) {
    const uint4* const words = A.xch + (C ? 0u : A.per_colour);
    const uint32_t first = blockIdx.x * blockDim.x * N, span = blockDim.x * N;
    const bool o = B.template odd<C>();
    const uint32_t at[5] = {B.yp, B.ym, B.zp, B.zm, o ? B.xp : B.xm};
    const bool in[5] = {B.hyp, B.hym, B.hzp, B.hzm, o ? B.hxp : B.hxm};
    bool open[5];
    uint4 w[5][N];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const uint32_t l = at[i] - first;
      open[i] = in[i] && l >= span;
#pragma unroll
      for (int t = 0; t < (i < 4 ? N : 1); ++t)
        w[i][t] = in[i] && l < span ? as_word(sites[C ^ 1][l + t]) : make_uint4(0, 0, 0, 0);
    }
    uint32_t polls = LIMITED ? A.Q.first_poll : 0u;
    bool again;
    do {
#pragma unroll
      for (int i = 0; i < 5; ++i) {
#pragma unroll
        for (int t = 0; t < (i < 4 ? N : 1); ++t)
          if (open[i]) w[i][t] = ld_word(words + at[i] + t);
      }
      again = false;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        bool there = true;
#pragma unroll
        for (int t = 0; t < (i < 4 ? N : 1); ++t)
          there = there && ((w[i][t].w ^ tag) & kTagMask) == 0;
        if (there) open[i] = false;
        again = again || open[i];
      }
      if (again && ++polls % 1024 == 0) {
        if (polls >= kWaitPolls || *(volatile unsigned int*)&A.Q.ctl->status) lost = 1;
        again = !lost;  // a lost launch runs to its end without waiting
      }
    } while (again);
#pragma unroll
    for (int t = 0; t < N; ++t) {
      w[2][t].w = __float_as_uint(zs[C][0][t]);
      w[3][t].w = __float_as_uint(zs[C][1][t]);
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {  // the other published sites are a CTA's border rows
      if (i != 2 && i != 3 && in[i] && at[i] - first >= span) {
#pragma unroll
        for (int t = 0; t < (i < 4 ? N : 1); ++t)
          w[i][t].w = __float_as_uint(A.Q.L.col[C ^ 1][at[i] + t].w);
      }
    }
#pragma unroll
    for (int t = 0; t < N; ++t) {
#pragma unroll
      for (int i = 0; i < 4; ++i) nb[t].b[2 + i] = as_site(w[i][t]);
    }
    const float4 e = as_site(w[4][0]), xa = own<C ^ 1>(0);
    if constexpr (N == 1) {
      nb[0].b[0] = o ? e : xa;
      nb[0].b[1] = o ? xa : e;
    } else {
      const float4 xb = own<C ^ 1>(1);
      nb[0].b[0] = o ? xb : xa;
      nb[0].b[1] = o ? xa : e;
      nb[1].b[0] = o ? e : xb;
      nb[1].b[1] = o ? xb : xa;
    }
  }

  // Colour 0's first neighbours, from the lattice.
  __device__ __forceinline__ void start(Nbrs (&nb)[N]) {
    if constexpr (N == 1) B.template neighbours<0>(A.Q.L, nb[0]);
    else B.template neighbours<0>(A.Q.L, nb[0], nb[1]);
  }

  template <int C>
  __device__ __forceinline__ void move(uint32_t tag, const Nbrs (&nb)[N]) {
    if (B.has) {
#pragma unroll
      for (int t = 0; t < N; ++t) {
        float4& n = own<C>(t);
        const bool second = N == 1 ? (slot() & 1u) != 0 : t == 1;
        if (N == 1 ? (B.template odd<C>() ? B.v[1] : B.v[0])
                   : (B.template odd<C>() ? B.v[N * t + 1] : B.v[N * t]))
          n = quench_site<P>(n, nb[t], A.Q.cp, A.Q.eta, second);
        st_word(A.xch + (C ? A.per_colour : 0u) + slot() + t, n, tag);
        sites[C][threadIdx.x * N + t] = n;
      }
    }
    __syncthreads();
  }

  template <int C>
  __device__ __forceinline__ void store() {
    if constexpr (N == 1) B.template store<C>(A.Q.L);
    else st_unit(A.Q.L.col[C] + B.u, B.n[C][0], B.n[C][1]);
  }
};

template <bool P, int N, int T, bool LIMITED>
__global__ void __launch_bounds__(T, 1)
    quench_flow_kernel(const __grid_constant__ QuenchFlowArgs A) {
  __shared__ float4 sites[2][N * T];
  __shared__ volatile int s_lost;
  Control* const ctl = A.Q.ctl;
  const uint32_t base = *(volatile uint32_t*)A.epoch;
  if (threadIdx.x == 0) s_lost = *(volatile unsigned int*)&ctl->status ? 1 : 0;
  __syncthreads();
  const bool stale = s_lost;  // an earlier wait ran out: the words are not to be trusted
  __syncthreads();
  if (stale) return;
  QuenchFlow<P, N, T, LIMITED> F(A, sites, s_lost);
  const bool has = F.B.has;
  for (int s = 0; s < A.Q.nsteps; ++s) {
    Nbrs nb[N];
    if (has) {
      if (s)
        F.template neighbours<0>(base + (uint32_t)s, nb);
      else
        F.start(nb);
    }
    F.template move<0>(base + (uint32_t)s + 1u, nb);
    if (has) F.template neighbours<1>(base + (uint32_t)s + 1u, nb);
    F.template move<1>(base + (uint32_t)s + 1u, nb);
  }
  if (has && !s_lost) {
    F.template store<0>();
    F.template store<1>();
  }
  if (threadIdx.x != 0) return;
  if (s_lost) {
    set_status(ctl, 4u);
    atomicAdd(A.epoch, (uint32_t)A.Q.nsteps + 2u);  // what was published is never read again
  } else if (atomicAdd(A.Q.words, 1ull) == gridDim.x - 1) {
    *A.epoch = base + (uint32_t)A.Q.nsteps;
    *A.Q.words = 0;
  }
}

using QuenchKernel = void (*)(const QuenchArgs);
template <bool LIMITED>
QuenchKernel quench_resident(bool periodic, bool site) {
  if (site)
    return periodic ? quench_resident_kernel<true, true, LIMITED>
                    : quench_resident_kernel<false, true, LIMITED>;
  return periodic ? quench_resident_kernel<true, false, LIMITED>
                  : quench_resident_kernel<false, false, LIMITED>;
}

// n: sites (1) or a unit (2) per thread.
using QuenchFlowKernel = void (*)(const QuenchFlowArgs);
template <bool LIMITED>
QuenchFlowKernel quench_flow(bool periodic, int n, bool wide) {
  if (wide) return quench_flow_kernel<true, 1, kQuenchWide, LIMITED>;
  if (n == 1)
    return periodic ? quench_flow_kernel<true, 1, kResThreads, LIMITED>
                    : quench_flow_kernel<false, 1, kResThreads, LIMITED>;
  return periodic ? quench_flow_kernel<true, 2, kResThreads, LIMITED>
                  : quench_flow_kernel<false, 2, kResThreads, LIMITED>;
}

// CTAs of `kernel` (kGradThreads threads) resident on the current device, one
// wave of a grid-stride launch; cached per device ordinal (threads that race
// on the first query store the same value).
template <class Kernel>
int resident_ctas(Kernel kernel, std::atomic<int> cache[16]) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int>& slot = cache[dev & 15];
  int res = slot.load(std::memory_order_relaxed);
  if (res == 0) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kGradThreads, 0);
    res = std::max(1, sms) * std::max(1, per_sm);
    slot.store(res, std::memory_order_relaxed);
  }
  return res;
}

}  // namespace

int energy_grad_max_blocks() { return kGradMaxBlocks; }

void launch_quench_pass(const LatticeView& L, const CouplingD& cd, float eta, int colour,
                        cudaStream_t stream) {
  Coupling cp;
  cp.eps = (float)cd.eps;
  cp.K = (float)cd.K;
  cp.g = (float)cd.g;
  cp.inv_kT = 0.f;
  static std::atomic<int> resident[16];
  const int res = resident_ctas(quench_pass_kernel<0, true>, resident);
  const SweepGeom G = make_geom(L);
  size_t blocks = ((size_t)G.units + kGradThreads - 1) / kGradThreads;
  if (blocks > (size_t)res) blocks = (size_t)res;
  if (blocks == 0) blocks = 1;
  const unsigned int nb = (unsigned int)blocks;
  if (L.periodic) {
    if (colour == 0) quench_pass_kernel<0, true><<<nb, kGradThreads, 0, stream>>>(L, G, cp, eta);
    else quench_pass_kernel<1, true><<<nb, kGradThreads, 0, stream>>>(L, G, cp, eta);
  } else {
    if (colour == 0) quench_pass_kernel<0, false><<<nb, kGradThreads, 0, stream>>>(L, G, cp, eta);
    else quench_pass_kernel<1, false><<<nb, kGradThreads, 0, stream>>>(L, G, cp, eta);
  }
}

// Sites (1) or a unit (2) per thread of quench_flow_kernel; 0: not that form.  With
// kQuenchWide threads per SM a site each takes periodic lattices up to 64^3 (3.58
// against 4.25 us with a unit each, 56^3 2.82 against 3.70, and 54^3, whose rows are
// padded, 3.0 against the unit loop's 5.4); the open kernel spills more there and is
// slower (4.6 against 4.3).
int quench_flow_sites(const LatticeView& L) {
  const uint32_t units = make_geom(L).units;
  if (2 * units <= 256) return 0;
  if (one_site_each(units, L.periodic ? kQuenchWide : kResThreads)) return 1;
  return one_unit_each(L, units) ? 2 : 0;
}

// Against a launch per pass, us per step (periodic): 8^3 1.1 and 7.5, 64^3 3.6 and
// 8.4, 96^3 12.4 and 16.6, 128^3 24.4 and 25.0; from 160^3 on the launches win (45.2
// and 41.3: their loads are the read-only ones).
bool quench_resident_pays(const LatticeView& L) { return make_geom(L).units <= (1u << 19); }

cudaError_t launch_quench_resident(const LatticeView& L, const CouplingD& cd, float eta,
                                   Control* ctl, unsigned long long* words, void* xch, int nsteps,
                                   uint32_t wait_limit, cudaStream_t stream) {
  QuenchArgs A;
  A.L = L;
  A.G = make_geom(L);
  A.cp.eps = (float)cd.eps;
  A.cp.K = (float)cd.K;
  A.cp.g = (float)cd.g;
  A.cp.inv_kT = 0.f;
  A.eta = eta;
  A.ctl = ctl;
  A.words = words;
  A.nsteps = nsteps;
  A.first_poll = first_poll(wait_limit);
  if (const int n = quench_flow_sites(L)) {
    QuenchFlowArgs F;
    F.Q = A;
    F.xch = static_cast<uint4*>(xch);
    F.epoch = reinterpret_cast<uint32_t*>(words + 3 * kWordStride);
    F.per_colour = 2 * A.G.units;
    const bool wide = n == 1 && !one_site_each(A.G.units);
    const auto kernel = A.first_poll ? quench_flow<true>(L.periodic, n, wide)
                                     : quench_flow<false>(L.periodic, n, wide);
    uint32_t threads, grid;
    resident_shape(n == 1 ? 2 * A.G.units : A.G.units, threads, grid,
                   wide ? kQuenchWide : kResThreads);
    return launch_cooperative(kernel, grid, threads, stream, F);
  }
  const bool site = 2 * A.G.units <= 256;
  uint32_t block, ctas;
  resident_shape(site ? 2 * A.G.units : A.G.units, block, ctas);
  return launch_cooperative(A.first_poll ? quench_resident<true>(L.periodic, site)
                                         : quench_resident<false>(L.periodic, site),
                            ctas, block, stream, A);
}

cudaError_t launch_natural_grad(int ni, int nj, int nk, int periodic, const float* n,
                                const float* s, const CouplingD& cd, float* grad, int project,
                                double* partials, double* energy, double* derivs,
                                cudaStream_t stream) {
  static std::atomic<int> resident[2][16];
  const uint32_t ctas = (uint32_t)std::min(
      kGradMaxBlocks, grad ? resident_ctas(natural_grad_kernel<true, false>, resident[1])
                           : resident_ctas(natural_grad_kernel<false, false>, resident[0]));
  NaturalGeom G;
  G.ni = (uint32_t)ni;
  G.nj = (uint32_t)nj;
  G.nk = (uint32_t)nk;
  G.plane = G.ni * G.nj;
  G.cols = (G.plane + 31) / 32 * 32;
  // Planes per task: the fewest steps on the busiest thread, a task's first
  // loads counted as half a step.
  G.seg = cheapest_segment(G.cols, G.nk, (uint64_t)ctas * kGradThreads, 0.5);
  G.nseg = (G.nk + G.seg - 1) / G.seg;
  const uint64_t need = ((uint64_t)G.cols * G.nseg + kGradThreads - 1) / kGradThreads;
  const uint32_t blocks = (uint32_t)std::min<uint64_t>(need, ctas);
  auto kernel = grad ? (periodic ? natural_grad_kernel<true, true> : natural_grad_kernel<true, false>)
                     : (periodic ? natural_grad_kernel<false, true>
                                 : natural_grad_kernel<false, false>);
  kernel<<<blocks, kGradThreads, 0, stream>>>(G, n, s, cd, grad, project, partials);
  // scheduled while the kernel before it drains
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(kGradThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, natural_sums_kernel, (const double*)partials, blocks, energy,
                            derivs);
}

void launch_energy_grad(const LatticeView& L, const CouplingD& cp, float4* grad_rb, int project,
                        double* partials, unsigned int* ticket, double* out4,
                        cudaStream_t stream) {
  const size_t total = 2 * (size_t)L.nk * L.nj * L.hx;
  const bool units = unit_view_aligned(L) && ((uintptr_t)grad_rb % 32) == 0;
  static std::atomic<int> resident[16];
  const int res = units ? resident_ctas(energy_grad_unit_kernel<true>, resident) : kGradMaxBlocks;
  size_t blocks = ((units ? total / 4 : total) + kGradThreads - 1) / kGradThreads;
  if (blocks > (size_t)std::min(res, kGradMaxBlocks)) blocks = std::min(res, kGradMaxBlocks);
  if (blocks == 0) blocks = 1;
  const unsigned int nb = (unsigned int)blocks;
  if (units) {
    const SweepGeom G = make_geom(L);
    const uint32_t pc = (uint32_t)(total / 2);
    if (L.periodic)
      energy_grad_unit_kernel<true><<<nb, kGradThreads, 0, stream>>>(L, G, cp, grad_rb, pc, project,
                                                                     partials, ticket, out4);
    else
      energy_grad_unit_kernel<false><<<nb, kGradThreads, 0, stream>>>(
          L, G, cp, grad_rb, pc, project, partials, ticket, out4);
  } else {
    energy_grad_site_kernel<<<nb, kGradThreads, 0, stream>>>(L, make_moment_geom(L), cp, grad_rb,
                                                             project, partials, ticket, out4);
  }
}

}  // namespace chll
