// Analysis kernels on one lattice's state: shell correlations of the director
// and the chirality, and integer projections of the chirality along a lattice
// direction (the input of the structure factor).
//
// Shell correlations restate calc_n_corr / calc_s_corr of the reference's
// analysis notebook (notebooks/paper_plots2.ipynb, cell 0, lines 61-112): over
// every ordered pair of sites (x, x + d) with |d|^2 < R^2 and both sites
// inside the lattice (open boundaries; optionally periodic images), shell
// floor(|d|) collects (n_x . n_{x+d})^2 and s_x s_{x+d}.  The sum over all
// sites of a pair term is the same for d and -d, so the kernel walks d = 0
// and one half-space of offsets (the host doubles shells >= 1; shell 0 holds
// d = 0 only) and the pair counts come from the host in closed form.
//
// Work layout: natural-order float4 sites (unpacked once into scratch).  The
// offsets, sorted by shell, are cut into chunks of at most kCorrChunk of one
// shell; a thread holds a strip of eight sites (i, j .. j+7, k) in registers and
// runs every site's pairs with a chunk's offsets: FP32 dot products and one FP32
// running sum per site and chunk (the chirality term is exact: +-1 products),
// then FP64 sums per thread and shell in shared memory.  CTA partials are summed
// in a fixed order by a second kernel, so results are reproducible bit for bit.
//
// What bounds it: a pair loads its other site, four L1 wavefronts of a warp's
// 512 bytes (offsets of one shell lie on a thin sphere, so a strip's sites share
// few neighbours while it is walked).  With one thread per site, the offset's
// load, wrap and bounds tests, the shell test and the 64-bit address were paid
// per pair: 33 instructions, and 8 wavefronts (96^3, 10 shells: 2460 us, the
// sum of the partials by one thread per column another 59).  The strip shares
// them: 14 instructions and 5 wavefronts, 1310 and 3 us (64^3, 20 shells: 7.2 ->
// 4.3 ms; strips of four sites: 1.72 ms and 4.8).  A site past an open boundary reads as the zero site behind
// the lattice.  Small lattices give a strip several tasks, chunks in turn.
//
// The projection kernel bins s by m = p . (i+1, j+1, k+1) for an integer
// direction p into an integer histogram (exact, order-free), from which the
// structure factor of hero_stripe.py's get_sc (a sum of s exp(-i k.(x+1)) for
// k along p) is a short one-dimensional transform (structure_factor_kernel).
#include <algorithm>
#include <atomic>

#include "chll_common.cuh"
#include "moments.cuh"
#include "sweep.cuh"

namespace chll {

namespace {

constexpr int kCorrThreads = 128;
constexpr int kStrip = 8;

struct CorrGeom {
  uint32_t ni, nj, nk;
  uint32_t strips;  // ni * ceil(nj / kStrip) * nk, rounded up to whole warps
  uint32_t splits;  // tasks per strip, each every splits-th chunk
  int nchunks, nshells;
};

// offs[o] = {di, dj, dk, 0}, with WRAP reduced into [0, n); chunks[c] = {first
// offset, end, shell}.  site[ni * nj * nk] is zero.
template <bool WRAP>
__global__ void __launch_bounds__(kCorrThreads)
    shell_corr_kernel(const float4* __restrict__ site, CorrGeom G, const int4* __restrict__ offs,
                      const int4* __restrict__ chunks, double* __restrict__ partials) {
  extern __shared__ double s_acc[];  // [2 * nshells][thread]
  const int R = G.nshells, tid = threadIdx.x;
  double* const an64 = s_acc + tid;
  double* const as64 = s_acc + (size_t)R * kCorrThreads + tid;
  for (int r = 0; r < R; ++r) an64[r * kCorrThreads] = as64[r * kCorrThreads] = 0.0;
  const uint32_t njs = (G.nj + kStrip - 1) / kStrip;
  const uint32_t nothing = G.ni * G.nj * G.nk;  // the zero site
  const uint64_t tasks = (uint64_t)G.strips * G.splits;
  double ssum = 0.0;
  for (uint64_t t = (uint64_t)blockIdx.x * kCorrThreads + tid; t < tasks;
       t += (uint64_t)gridDim.x * kCorrThreads) {
    const uint32_t split = (uint32_t)(t / G.strips);  // the same in a whole warp
    const uint32_t x = (uint32_t)(t - (uint64_t)split * G.strips);
    const uint32_t row = x / G.ni, i = x - row * G.ni;
    const uint32_t k = row / njs, j0 = (row - k * njs) * kStrip;
    const bool has = k < G.nk;
    // the strip's sites; those past its row's end are zero and sit at j = 0
    float4 a[kStrip];
    uint32_t j[kStrip];
#pragma unroll
    for (int c = 0; c < kStrip; ++c) {
      const bool v = has && j0 + c < G.nj;
      j[c] = v ? j0 + c : 0u;
      a[c] = __ldg(site + (v ? i + G.ni * (j[c] + G.nj * k) : nothing));
      if (split == 0) ssum += (double)a[c].w;
    }
    for (int q = (int)split; q < G.nchunks; q += (int)G.splits) {
      const int4 chunk = __ldg(chunks + q);
      float an[kStrip], as[kStrip];
#pragma unroll
      for (int c = 0; c < kStrip; ++c) an[c] = as[c] = 0.f;
      int4 after = __ldg(offs + chunk.x);
      for (int o = chunk.x; o < chunk.y; ++o) {
        const int4 d = after;
        after = __ldg(offs + o + 1);  // the chunks follow the offsets
        uint32_t ii = i + (uint32_t)d.x, kk = k + (uint32_t)d.z;
        bool in = has;
        if (WRAP) {
          if (ii >= G.ni) ii -= G.ni;
          if (kk >= G.nk) kk -= G.nk;
        } else {
          in = in && ii < G.ni && kk < G.nk;
        }
        const uint32_t base = ii + G.ni * G.nj * kk;
#pragma unroll
        for (int c = 0; c < kStrip; ++c) {
          uint32_t jj = j[c] + (uint32_t)d.y;
          if (WRAP && jj >= G.nj) jj -= G.nj;
          const float4 b = __ldg(site + (in && (WRAP || jj < G.nj) ? base + G.ni * jj : nothing));
          const float dt = fmaf(a[c].z, b.z, fmaf(a[c].y, b.y, __fmul_rn(a[c].x, b.x)));
          an[c] = fmaf(dt, dt, an[c]);
          as[c] = fmaf(a[c].w, b.w, as[c]);
        }
      }
      double vn = 0.0, vs = 0.0;
#pragma unroll
      for (int c = 0; c < kStrip; ++c) {
        vn += (double)an[c];
        vs += (double)as[c];
      }
      an64[chunk.z * kCorrThreads] += vn;
      as64[chunk.z * kCorrThreads] += vs;
    }
  }
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5, width = 2 * R + 1;
  double* const out = partials + (size_t)blockIdx.x * width;
  for (int c = warp; c < 2 * R; c += kCorrThreads / 32) {
    double v = 0.0;
    for (int w = lane; w < kCorrThreads; w += 32) v += s_acc[(size_t)c * kCorrThreads + w];
    v = warp_sum_d(v);
    if (lane == 0) out[c] = v;
  }
  __shared__ double s_sum[kCorrThreads / 32];
  ssum = warp_sum_d(ssum);
  if (lane == 0) s_sum[warp] = ssum;
  __syncthreads();
  if (tid == 0) {
    double v = 0.0;
    for (int w = 0; w < kCorrThreads / 32; ++w) v += s_sum[w];
    out[2 * R] = v;
  }
}

// Column blockIdx.x of the CTA partials summed over the CTAs, one warp per
// column in a fixed order.
__global__ void __launch_bounds__(32)
    sum_partials_kernel(const double* __restrict__ partials, int rows, int width,
                        double* __restrict__ out) {
  double v = 0.0;
  for (int r = threadIdx.x; r < rows; r += 32) v += partials[(size_t)r * width + blockIdx.x];
  v = warp_sum_d(v);
  if (threadIdx.x == 0) out[blockIdx.x] = v;
}

// hist[m - m0] += s over the real sites, m = p . (i+1, j+1, k+1).  A thread
// takes one slot (h, j) of a colour over a run of planes, where m moves by pz per
// plane and by px between even and odd planes.  With pz = 0 the run has two
// bins, kept in registers; with px = 0 the lanes of a row share their bin, summed
// in the warp first (else 32 lanes add to one shared word in turn).  256^3 along
// (1, 1, 1): 46 us (73 with one site per thread and its index divisions, 41 for
// the read of the state alone).
__global__ void __launch_bounds__(256)
    projection_kernel(LatticeView L, uint32_t seg, uint32_t ntasks, int px, int py, int pz,
                      long long m0, int nbins, unsigned long long* __restrict__ hist) {
  extern __shared__ int s_hist[];
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) s_hist[b] = 0;
  __syncthreads();
  const uint32_t hx = (uint32_t)L.hx, nj = (uint32_t)L.nj, nk = (uint32_t)L.nk;
  const uint32_t plane = hx * nj;
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t first = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
  // whole warps go round together (px = 0 exchanges between lanes)
  for (uint64_t t0 = first; t0 < ntasks; t0 += stride) {
    const uint32_t t = (uint32_t)t0 + (threadIdx.x & 31);
    const bool has = t0 + (threadIdx.x & 31) < ntasks;
    const uint32_t sg = t / (2 * plane), r = t - sg * 2 * plane;
    const uint32_t c = r >= plane, col = r - (c ? plane : 0u);
    const uint32_t j = col / hx, h = col - j * hx;
    const uint32_t k0 = has ? sg * seg : nk, k1 = min(k0 + seg, nk);
    const float* w = &colour_array(L, (int)c)[(size_t)(has ? k0 : 0u) * plane + col].w;
    // bins in 32-bit wrapping arithmetic: exact for the real sites
    uint32_t par = (c + j + k0) & 1u;
    uint32_t m = (uint32_t)((long long)px * (2 * (long long)h + 1) + (long long)py * (j + 1) +
                            (long long)pz * ((long long)k0 + 1) - m0);
    int sum[2] = {0, 0};  // pz = 0: sites of parity 0, 1
    const uint32_t steps = seg < nk ? seg : nk;
    for (uint32_t n0 = 0; n0 < steps; n0 += 4) {
      int s[4];
#pragma unroll
      for (uint32_t n = 0; n < 4; ++n) {  // loads of four planes in flight
        const bool in = k0 + n0 + n < k1 && 2 * h + (par ^ (n & 1u)) < (uint32_t)L.ni;
        s[n] = in ? (int)__ldg(w + 4 * (size_t)plane * n) : 0;
      }
      w += 16 * (size_t)plane;
#pragma unroll
      for (uint32_t n = 0; n < 4; ++n, m += (uint32_t)pz) {
        const uint32_t odd = par ^ (n & 1u);
        const uint32_t bin = m + (odd ? (uint32_t)px : 0u);
        if (pz == 0) {
          sum[0] += odd ? 0 : s[n];
          sum[1] += odd ? s[n] : 0;
        } else if (px == 0) {
          const uint32_t peers = __match_any_sync(0xffffffffu, s[n] ? bin : 0xffffffffu);
          const int v = __reduce_add_sync(peers, s[n]);
          if (s[n] && (threadIdx.x & 31) == (uint32_t)(__ffs(peers) - 1))
            atomicAdd(&s_hist[bin], v);
        } else if (s[n]) {
          atomicAdd(&s_hist[bin], s[n]);
        }
      }
    }
    if (pz == 0) {
      if (sum[0]) atomicAdd(&s_hist[m], sum[0]);
      if (sum[1]) atomicAdd(&s_hist[m + (uint32_t)px], sum[1]);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nbins; b += blockDim.x)
    if (s_hist[b]) atomicAdd(&hist[b], (unsigned long long)(long long)s_hist[b]);
}

// sf[q] = |sum_b hist[b] exp(-i kvs[q] (m0 + b)) / N|^2, one CTA per wave number.
// The transform on the host took a few thousand exponentials per wave number,
// one numpy call each: 8 ms for 500 of them on 256^3; here 5 us.
constexpr int kSfThreads = 128;
__global__ void __launch_bounds__(kSfThreads)
    structure_factor_kernel(const unsigned long long* __restrict__ hist, long long m0, int nbins,
                            const double* __restrict__ kvs, double nsites,
                            double* __restrict__ sf) {
  const double kv = kvs[blockIdx.x];
  double re = 0.0, im = 0.0;
  for (int b = threadIdx.x; b < nbins; b += kSfThreads) {
    const long long h = (long long)hist[b];
    if (h == 0) continue;
    double sn, cs;
    sincos(kv * (double)(m0 + b), &sn, &cs);
    re += (double)h * cs;
    im -= (double)h * sn;
  }
  __shared__ double s_part[2][kSfThreads / 32];
  re = warp_sum_d(re);
  im = warp_sum_d(im);
  if ((threadIdx.x & 31) == 0) {
    s_part[0][threadIdx.x >> 5] = re;
    s_part[1][threadIdx.x >> 5] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    re = im = 0.0;
    for (int w = 0; w < kSfThreads / 32; ++w) {
      re += s_part[0][w];
      im += s_part[1][w];
    }
    re /= nsites;
    im /= nsites;
    sf[blockIdx.x] = re * re + im * im;
  }
}

int device_sms() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 148;
}

}  // namespace

namespace {

size_t corr_smem(int nshells) { return 2 * (size_t)nshells * kCorrThreads * sizeof(double); }

CorrGeom corr_geom(int ni, int nj, int nk, int nchunks, int nshells, int blocks) {
  CorrGeom G;
  G.ni = (uint32_t)ni;
  G.nj = (uint32_t)nj;
  G.nk = (uint32_t)nk;
  const uint64_t strips = (uint64_t)ni * ((nj + kStrip - 1) / kStrip) * nk;
  G.strips = (uint32_t)((strips + 31) / 32 * 32);
  // the least work on the busiest thread, a task's start counted as half a
  // percent of a strip
  const uint64_t threads = (uint64_t)blocks * kCorrThreads;
  double best = 1e300;
  for (uint32_t s = 1; s <= (uint32_t)nchunks; ++s) {
    const double cost =
        (double)((G.strips * (uint64_t)s + threads - 1) / threads) * (1.0 / s + 0.005);
    if (cost < best) {
      best = cost;
      G.splits = s;
    }
  }
  G.nchunks = nchunks;
  G.nshells = nshells;
  return G;
}

}  // namespace

// Resident CTAs of the kernel with these shells, queried once per device and
// number of shells.
int shell_corr_blocks(int nshells) {
  static std::atomic<int> cache[16][kMaxCorrShells + 1];
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int>& known = cache[dev & 15][nshells];
  if (const int n = known.load(std::memory_order_relaxed)) return n;
  const size_t smem = corr_smem(nshells);
  int per_sm = 1 << 30;
  for (auto kernel : {shell_corr_kernel<false>, shell_corr_kernel<true>}) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)corr_smem(kMaxCorrShells));
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kCorrThreads, smem);
    if (n < per_sm) per_sm = n;
  }
  const int blocks = device_sms() * (per_sm > 0 ? per_sm : 1);
  known.store(blocks, std::memory_order_relaxed);
  return blocks;
}

void launch_shell_corr(const float4* site, int ni, int nj, int nk, const int4* offs,
                       const int4* chunks, int nchunks, int nshells, bool wrap, double* partials,
                       int blocks, double* out, cudaStream_t stream) {
  const CorrGeom G = corr_geom(ni, nj, nk, nchunks, nshells, blocks);
  const uint64_t need = ((uint64_t)G.strips * G.splits + kCorrThreads - 1) / kCorrThreads;
  const int grid = (int)std::min<uint64_t>(need, (uint64_t)blocks);
  const size_t smem = corr_smem(nshells);
  if (wrap)
    shell_corr_kernel<true><<<grid, kCorrThreads, smem, stream>>>(site, G, offs, chunks, partials);
  else
    shell_corr_kernel<false><<<grid, kCorrThreads, smem, stream>>>(site, G, offs, chunks, partials);
  const int width = 2 * nshells + 1;
  sum_partials_kernel<<<width, 32, 0, stream>>>(partials, grid, width, out);
}

void launch_projection(const LatticeView& L, int px, int py, int pz, long long m0, int nbins,
                       unsigned long long* hist, cudaStream_t stream) {
  const uint32_t cols = 2 * (uint32_t)L.hx * (uint32_t)L.nj, nk = (uint32_t)L.nk;
  // Six CTAs per SM, or as many as the bins leave room for: the loads of four planes
  // are all a thread has in flight.  With four, a whole call for 100 wave numbers took
  // 155 us at 320^3 along (1, -1, 2) and 97 at 256^3 along (0, 0, 1), with six 124 and
  // 85; eight are no better (126 and 79 to 86), and 96^3 takes 40 us with any.
  const uint32_t room = (227u << 10) / ((uint32_t)nbins * (uint32_t)sizeof(int) + 1024);
  const uint32_t ctas = (uint32_t)device_sms() * std::max(1u, std::min(6u, room));
  const uint32_t threads = ctas * 256;
  // planes per task: enough tasks for the resident threads, runs as long as that
  // leaves them
  const uint32_t nseg = std::min(nk, std::max(1u, threads / cols));
  const uint32_t seg = (nk + nseg - 1) / nseg;
  const uint32_t ntasks = cols * ((nk + seg - 1) / seg);
  const uint32_t need = (uint32_t)(((uint64_t)ntasks + 255) / 256);  // ntasks < 2^32
  projection_kernel<<<std::min(need, ctas), 256, (size_t)nbins * sizeof(int), stream>>>(
      L, seg, ntasks, px, py, pz, m0, nbins, hist);
}

void launch_structure_factor(const unsigned long long* hist, long long m0, int nbins,
                             const double* kvs, int nkv, double nsites, double* sf,
                             cudaStream_t stream) {
  structure_factor_kernel<<<nkv, kSfThreads, 0, stream>>>(hist, m0, nbins, kvs, nsites, sf);
}

}  // namespace chll
