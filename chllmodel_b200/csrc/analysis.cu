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
// Work layout: natural-order float4 sites (unpacked once into scratch), one
// thread per site, grid-stride in whole warps so every lane walks the same
// offset list (sorted by shell) and the warp reduces a shell's sums together.
// Per pair: FP32 dot product and FP32 running sums over at most kChunk
// offsets (the chirality term is exact: +-1 products), then an FP64 warp sum
// into per-warp shared slots; CTA partials are summed in a fixed order by a
// second kernel, so results are reproducible bit for bit.
//
// The projection kernel bins s by m = p . (i+1, j+1, k+1) for an integer
// direction p into an integer histogram (exact, order-free), from which the
// structure factor of hero_stripe.py's get_sc (a sum of s exp(-i k.(x+1)) for
// k along p) is a short one-dimensional transform (structure_factor_kernel).
#include <algorithm>

#include "chll_common.cuh"
#include "moments.cuh"
#include "sweep.cuh"

namespace chll {

namespace {

constexpr int kCorrThreads = 256;
constexpr int kCorrWarps = kCorrThreads / 32;
constexpr int kChunk = 128;  // FP32 terms per running sum before the FP64 flush

__device__ __forceinline__ void flush_shell(double (*s_n)[kMaxCorrShells],
                                            double (*s_s)[kMaxCorrShells], int warp, int lane,
                                            int shell, float an, float as) {
  const double vn = warp_sum_d((double)an);
  const double vs = warp_sum_d((double)as);
  if (lane == 0) {
    s_n[warp][shell] += vn;
    s_s[warp][shell] += vs;
  }
}

// offs[o] = {di, dj, dk, shell}, sorted by shell.  With WRAP the host has
// reduced di, dj, dk into [0, n) so one conditional subtraction wraps.
template <bool WRAP>
__global__ void __launch_bounds__(kCorrThreads)
    shell_corr_kernel(const float4* __restrict__ site, int ni, int nj, int nk,
                      const int4* __restrict__ offs, int noffs, int nshells,
                      double* __restrict__ partials) {
  __shared__ double s_n[kCorrWarps][kMaxCorrShells];
  __shared__ double s_s[kCorrWarps][kMaxCorrShells];
  __shared__ double s_sum[kCorrWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = lane; r < nshells; r += 32) {
    s_n[warp][r] = 0.0;
    s_s[warp][r] = 0.0;
  }
  __syncwarp();
  const uint32_t uni = (uint32_t)ni, unj = (uint32_t)nj, unk = (uint32_t)nk;
  const uint64_t N = (uint64_t)uni * unj * unk;
  const uint64_t stride = (uint64_t)gridDim.x * kCorrThreads;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  double ssum = 0.0;
  for (uint64_t x0 = (uint64_t)blockIdx.x * kCorrThreads + (uint64_t)warp * 32; x0 < N;
       x0 += stride) {
    const uint64_t x = x0 + (uint64_t)lane;
    const bool valid = x < N;
    const uint32_t xi = valid ? (uint32_t)x : 0u;
    const uint32_t row = xi / uni;
    const int i = (int)(xi - row * uni);
    const int k = (int)(row / unj);
    const int j = (int)(row - (uint32_t)k * unj);
    const float4 a = valid ? site[xi] : zero;
    ssum += (double)a.w;
    int cur = -1, run = 0;
    float an = 0.f, as = 0.f;
    for (int o = 0; o < noffs; ++o) {
      const int4 d = __ldg(offs + o);
      if (d.w != cur || run == kChunk) {
        if (cur >= 0) flush_shell(s_n, s_s, warp, lane, cur, an, as);
        cur = d.w;
        run = 0;
        an = 0.f;
        as = 0.f;
      }
      ++run;
      uint32_t ii = (uint32_t)(i + d.x), jj = (uint32_t)(j + d.y), kk = (uint32_t)(k + d.z);
      bool in = valid;
      if (WRAP) {
        if (ii >= uni) ii -= uni;
        if (jj >= unj) jj -= unj;
        if (kk >= unk) kk -= unk;
      } else {
        in = in && ii < uni && jj < unj && kk < unk;
      }
      if (in) {
        const float4 b = site[ii + uni * (jj + unj * kk)];
        const float dt = fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x)));
        an = fmaf(dt, dt, an);
        as = fmaf(a.w, b.w, as);
      }
    }
    if (cur >= 0) flush_shell(s_n, s_s, warp, lane, cur, an, as);
  }
  ssum = warp_sum_d(ssum);
  if (lane == 0) s_sum[warp] = ssum;
  __syncthreads();
  const int width = 2 * nshells + 1;
  double* out = partials + (size_t)blockIdx.x * width;
  for (int t = threadIdx.x; t < width; t += kCorrThreads) {
    double v = 0.0;
    for (int w = 0; w < kCorrWarps; ++w)
      v += t < nshells ? s_n[w][t] : (t < 2 * nshells ? s_s[w][t - nshells] : s_sum[w]);
    out[t] = v;
  }
}

// Column t of the CTA partials summed over CTAs in index order.
__global__ void sum_partials_kernel(const double* __restrict__ partials, int rows, int width,
                                    double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= width) return;
  double v = 0.0;
  for (int r = 0; r < rows; ++r) v += partials[(size_t)r * width + t];
  out[t] = v;
}

// hist[m - m0] += s over the real sites, m = p . (i+1, j+1, k+1).  A thread
// takes one slot (h, j) of a colour over a run of planes, where m moves by pz per
// plane and by px between even and odd planes.  With pz = 0 the run has two
// bins, kept in registers; with px = 0 the lanes of a row share their bin, summed
// in the warp first (else 32 lanes add to one shared word in turn).  256^3 along
// (1, 1, 1): 54 us (73 with one site per thread and its index divisions, 41 for
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

int shell_corr_blocks(uint64_t nsites) {
  const uint64_t need = (nsites + kCorrThreads - 1) / kCorrThreads;
  const uint64_t cap = (uint64_t)device_sms() * 8;
  return (int)(need < cap ? (need ? need : 1) : cap);
}

void launch_shell_corr(const float4* site, int ni, int nj, int nk, const int4* offs, int noffs,
                       int nshells, bool wrap, double* partials, int blocks, double* out,
                       cudaStream_t stream) {
  if (wrap)
    shell_corr_kernel<true><<<blocks, kCorrThreads, 0, stream>>>(site, ni, nj, nk, offs, noffs,
                                                                  nshells, partials);
  else
    shell_corr_kernel<false><<<blocks, kCorrThreads, 0, stream>>>(site, ni, nj, nk, offs,
                                                                   noffs, nshells, partials);
  const int width = 2 * nshells + 1;
  sum_partials_kernel<<<(width + 127) / 128, 128, 0, stream>>>(partials, blocks, width, out);
}

void launch_projection(const LatticeView& L, int px, int py, int pz, long long m0, int nbins,
                       unsigned long long* hist, cudaStream_t stream) {
  const uint32_t cols = 2 * (uint32_t)L.hx * (uint32_t)L.nj, nk = (uint32_t)L.nk;
  const uint32_t ctas = (uint32_t)device_sms() * 4, threads = ctas * 256;
  // planes per task: enough tasks for the resident threads, runs as long as that
  // leaves them
  const uint32_t nseg = std::min(nk, std::max(1u, threads / cols));
  const uint32_t seg = (nk + nseg - 1) / nseg;
  const uint32_t ntasks = cols * ((nk + seg - 1) / seg);
  const uint32_t need = (ntasks + 255) / 256;
  projection_kernel<<<std::min(need, ctas), 256, (size_t)nbins * sizeof(int), stream>>>(
      L, seg, ntasks, px, py, pz, m0, nbins, hist);
}

void launch_structure_factor(const unsigned long long* hist, long long m0, int nbins,
                             const double* kvs, int nkv, double nsites, double* sf,
                             cudaStream_t stream) {
  structure_factor_kernel<<<nkv, kSfThreads, 0, stream>>>(hist, m0, nbins, kvs, nsites, sf);
}

}  // namespace chll
