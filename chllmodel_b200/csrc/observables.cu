// FP64 observables of one red/black lattice and the reference measurement
// row: the sums that moments.cuh lists, and the reference's etot()
// (chll_mod.f90:414-456): x and y periodic, z open, and the +y dot product's x
// component read from the diagonal neighbour (ip1, jp1, k) as chll_mod.f90:438.
//
// A thread walks a column of 4-site x-blocks (both colours' units at one slot)
// over a run of planes.  Its four sites are converted to FP64 once and serve as
// the +z neighbours of the step before, as each other's +x neighbours, and a
// step loads the +y row's block and one site beyond the block: 9.3 conversions
// and 42 FP64 operations per site where one thread per site with all its
// neighbours took 18 and 59 (and twice the other instructions).  Before and
// after, us: 64^3 11.7, 8.3; 128^3 26.7, 18.0; 256^3 157, 86; 480^3 1004, 508
// (the read of the state alone: 41 and 271 us at 256^3 and 480^3).  The FP64 pipe
// is half busy; the rest is the waits of twelve warps per SM.  Sixteen at 128
// registers took 505 us at 480^3 but 10.1 at 64^3, twenty at 96 spill (690 us).
//
// Reduction: warp shuffle -> CTA partial in scratch -> the last CTA to finish
// sums the partials in a fixed order, so results are bit-reproducible.
#include <algorithm>
#include <atomic>

#include "chll_common.cuh"
#include "moments.cuh"
#include "sweep.cuh"
#include "sweep_unit.cuh"

namespace chll {

namespace {

constexpr int kObsThreads = 128;
constexpr int kObsCtasPerSm = 3;  // 168 registers: the block and its neighbours in FP64
constexpr int kObsMaxBlocks = 148 * 4;

struct ObsWalk {
  uint32_t Q, ncols;   // blocks per row and per plane
  uint32_t seg, ntasks;  // planes per task, tasks
};

struct Site64 {
  double x, y, z, s;
};

__device__ __forceinline__ Site64 to64(const float4& v) {
  return {(double)v.x, (double)v.y, (double)v.z, (double)v.w};
}

// The four sites 4q .. 4q+3 of a row from the units at its slot of both
// colours; c: colour of site 4q.
__device__ __forceinline__ void load_block(const LatticeView& L, uint32_t c, uint32_t u,
                                           float4 v[4]) {
  const UnitSlots a = ld_unit_nc(colour_array(L, (int)c) + u);
  const UnitSlots b = ld_unit_nc(colour_array(L, (int)c ^ 1) + u);
  v[0] = a.a;
  v[1] = b.a;
  v[2] = a.b;
  v[3] = b.b;
}

// Sums over bonds of 1 - dot^2 and of dot * cross * (s + s').
struct BondAcc {
  double nem, chi;
  __device__ __forceinline__ void add(double dot, double cross, double ss) {
    nem += 1.0 - dot * dot;
    chi += dot * cross * ss;
  }
};

// PER: periodic boundaries.  PAD: rows whose last block may hold padding.
template <bool PER, bool PAD>
__global__ void __launch_bounds__(kObsThreads, kObsCtasPerSm)
    observables_kernel(LatticeView L, MomentGeom M, ObsWalk W, CouplingD cp,
                       const Control* __restrict__ ctl,
                       double* __restrict__ partials, unsigned int* __restrict__ ticket,
                       double* __restrict__ row, long long step) {
  // bonds of the energy and the reference etot, of the energy alone, of etot
  // alone (x and y wrap there, z is open, the +y dot product is its own)
  BondAcc both = {0.0, 0.0}, own = {0.0, 0.0}, ref = {0.0, 0.0};
  double acc[kObsMoments];
#pragma unroll
  for (int m = 0; m < kObsMoments; ++m) acc[m] = 0.0;

  const uint32_t hx = (uint32_t)L.hx, nj = (uint32_t)L.nj, nk = (uint32_t)L.nk;
  const uint32_t plane = hx * nj;
  for (uint32_t t = blockIdx.x * kObsThreads + threadIdx.x; t < W.ntasks;
       t += gridDim.x * kObsThreads) {
    const uint32_t sg = t / W.ncols, col = t - sg * W.ncols;
    const uint32_t j = col / W.Q, q = col - j * W.Q;
    const uint32_t k0 = sg * W.seg, k1 = min(k0 + W.seg, nk);
    const uint32_t jp = j + 1 < nj ? j + 1 : 0;
    const bool has_yp = PER || j + 1 < nj;
    // slot offsets of the +y row's block and of the site after the block (the
    // row's first site after its last)
    const uint32_t oy = j + 1 < nj ? hx : (uint32_t)(-(int32_t)(j * hx));
    const uint32_t ox = q + 1 < W.Q ? 2u : (uint32_t)(-(int32_t)(2 * q));
    const bool row_end = q + 1 == W.Q;
    const uint32_t nv = PAD && row_end ? (uint32_t)L.ni - 4 * q : 4u;  // sites of the block
    uint32_t u = (k0 * nj + j) * hx + 2 * q;
    uint32_t c = (j + k0) & 1u, cy = (jp + k0) & 1u;
    Site64 d[4];
    {
      float4 v[4];
      load_block(L, c, u, v);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[i] = to64(v[i]);
    }
    for (uint32_t k = k0; k < k1; ++k) {
      const bool ref_zp = (uint32_t)M.kglob0 + k + 1 < (uint32_t)M.nkg;  // z is open in etot
      const bool has_zp = PER || ref_zp;
      const bool wrap_z = k + 1 == nk && !M.zhalo;
      float4 v[4], w[4];
      if (k + 2 < nk) {  // the plane after the next: the lines no thread has read yet
        asm volatile("prefetch.global.L1 [%0];" ::"l"(L.col[0] + (u + 2 * plane)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(L.col[1] + (u + 2 * plane)));
      }
      if (has_zp) {
        const uint32_t cz = wrap_z ? j & 1u : c ^ 1u;
        load_block(L, cz, wrap_z ? u - k * plane : u + plane, v);
      }
      load_block(L, cy, u + oy, w);
      const Site64 xe = to64(ld4(colour_array(L, (int)c) + (u + ox)));
      const double te = (double)__ldg(&colour_array(L, (int)cy)[u + oy + ox].x);
      double wx[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) wx[i] = (double)w[i].x;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (PAD && (uint32_t)i >= nv) break;
        const bool end = row_end && (PAD ? (uint32_t)i + 1 == nv : i == 3);
        const Site64 n = d[i];
        // +x
        Site64 X = i < 3 ? d[i < 3 ? i + 1 : 3] : xe;
        double tx = i < 3 ? wx[i < 3 ? i + 1 : 3] : te;
        if (PAD && end) {
          X = xe;
          tx = te;
        }
        const double dx = n.x * X.x + n.y * X.y + n.z * X.z;
        const double cx = n.y * X.z - n.z * X.y;
        if (!PER && end)
          ref.add(dx, cx, n.s + X.s);
        else
          both.add(dx, cx, n.s + X.s);
        // +y, and with the x component of the +x +y neighbour (chll_mod.f90:438)
        const double wy = (double)w[i].y, wz = (double)w[i].z, ss = n.s + (double)w[i].w;
        const double part = n.y * wy + n.z * wz;
        const double cyc = n.z * wx[i] - n.x * wz;
        if (has_yp) own.add(n.x * wx[i] + part, cyc, ss);
        ref.add(n.x * tx + part, cyc, ss);
        acc[2] += n.s;
        acc[3] += n.x * n.x;
        acc[4] += n.y * n.y;
        acc[5] += n.z * n.z;
        acc[6] += n.x * n.y;
        acc[7] += n.x * n.z;
        acc[8] += n.y * n.z;
      }
      // +z: the next step's block
      if (has_zp) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const Site64 n = d[i];
          const Site64 Z = d[i] = to64(v[i]);
          if (PAD && (uint32_t)i >= nv) continue;
          const double dz = n.x * Z.x + n.y * Z.y + n.z * Z.z;
          const double cz = n.x * Z.y - n.y * Z.x;
          if (ref_zp)
            both.add(dz, cz, n.s + Z.s);
          else
            own.add(dz, cz, n.s + Z.s);
        }
      }
      u += plane;
      c ^= 1u;
      cy ^= 1u;
    }
  }
  const double field = cp.g * acc[2], hk = 0.5 * cp.K;
  acc[0] = cp.eps * (both.nem + own.nem) - hk * (both.chi + own.chi) - field;
  acc[1] = cp.eps * (both.nem + ref.nem) - hk * (both.chi + ref.chi) - field;

  __shared__ double s_part[kObsThreads / 32][kObsMoments];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < kObsMoments; ++m) {
    const double v = warp_sum_d(acc[m]);
    if (lane == 0) s_part[warp][m] = v;
  }
  __syncthreads();
  if (threadIdx.x < kObsMoments) {
    double v = 0.0;
    for (int w = 0; w < kObsThreads / 32; ++w) v += s_part[w][threadIdx.x];
    partials[(size_t)blockIdx.x * kObsMoments + threadIdx.x] = v;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // The partials summed by the whole CTA: thread t takes blocks t, t + 256,
  // ... (L2 reads, all in flight at once), then warp shuffles and the warps in
  // order -- a fixed order for a given grid, so the result is reproducible.
  double v[kObsMoments];
#pragma unroll
  for (int m = 0; m < kObsMoments; ++m) v[m] = 0.0;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
#pragma unroll
    for (int m = 0; m < kObsMoments; ++m) v[m] += __ldcg(&partials[(size_t)b * kObsMoments + m]);
  }
#pragma unroll
  for (int m = 0; m < kObsMoments; ++m) {
    const double w = warp_sum_d(v[m]);
    if (lane == 0) s_part[warp][m] = w;
  }
  __syncthreads();
  __shared__ double s_tot[kObsMoments];
  if (threadIdx.x < kObsMoments) {
    double t = 0.0;
    for (int w = 0; w < kObsThreads / 32; ++w) t += s_part[w][threadIdx.x];
    s_tot[threadIdx.x] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *ticket = 0;
    const long long n = (long long)L.ni * L.nj * L.nk;
    const float n3 = (float)n;  // float(ni*nj*nk)
    // etot = e/float(N), a default REAL function result (chll_mod.f90:453)
    row[kRowEtotRef] = (double)(float)(s_tot[1] / (double)n3);
    // e_excess = sum(float(s))/float(N) in FP32 (chll_mod.f90:97)
    row[kRowEta] = (double)((float)s_tot[2] / n3);
    row[kRowPaccept] = ctl ? (double)ctl->paccept : 0.0;
    row[kRowFaccept] = ctl ? (double)ctl->faccept : 0.0;
    row[kRowD] = ctl ? ctl->d : 0.0;
    row[kRowEnergy] = s_tot[0];
    row[kRowSumS] = s_tot[2];
    row[kRowQxx] = s_tot[3];
    row[kRowQyy] = s_tot[4];
    row[kRowQzz] = s_tot[5];
    row[kRowQxy] = s_tot[6];
    row[kRowQxz] = s_tot[7];
    row[kRowQyz] = s_tot[8];
    row[kRowEtotRefSum] = s_tot[1];
    row[kRowStep] = (double)(step == kStepOfControl ? ctl->step - 1 : step);
    row[kRowNsites] = (double)n;
  }
}

}  // namespace

int observables_max_blocks() { return kObsMaxBlocks; }

namespace {

using ObsKernel = void (*)(LatticeView, MomentGeom, ObsWalk, CouplingD, const Control*, double*,
                           unsigned int*, double*, long long);
// [periodic][padded rows]
const ObsKernel kObs[2][2] = {{observables_kernel<false, false>, observables_kernel<false, true>},
                              {observables_kernel<true, false>, observables_kernel<true, true>}};

int obs_ctas() {
  static std::atomic<int> cache[16];
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int>& slot = cache[dev & 15];
  int n = slot.load(std::memory_order_relaxed);
  if (n == 0) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    n = std::min(std::max(1, sms) * kObsCtasPerSm, kObsMaxBlocks);
    slot.store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace

void launch_observables(const LatticeView& L, const MomentGeom& M, const CouplingD& cp,
                        const Control* ctl, double* partials, unsigned int* ticket, double* row,
                        long long step, cudaStream_t stream) {
  ObsWalk W;
  W.Q = (uint32_t)(L.hx >> 1);
  W.ncols = W.Q * (uint32_t)L.nj;
  // Planes per task: the fewest steps on the busiest thread, a task's first
  // block counted as a third of a step.
  const uint32_t threads = (uint32_t)obs_ctas() * kObsThreads, nk = (uint32_t)L.nk;
  W.seg = cheapest_segment(W.ncols, nk, threads, 0.33);
  W.ntasks = W.ncols * ((nk + W.seg - 1) / W.seg);
  const uint32_t need = (W.ntasks + kObsThreads - 1) / kObsThreads;
  const uint32_t blocks = std::min(need, (uint32_t)obs_ctas());
  kObs[L.periodic ? 1 : 0][L.ni % 4 ? 1 : 0]<<<blocks, kObsThreads, 0, stream>>>(
      L, M, W, cp, ctl, partials, ticket, row, step);
}

void launch_observables(const LatticeView& L, const CouplingD& cp, const Control* ctl,
                        double* partials, unsigned int* ticket, double* row, long long step,
                        cudaStream_t stream) {
  launch_observables(L, make_moment_geom(L), cp, ctl, partials, ticket, row, step, stream);
}

}  // namespace chll
