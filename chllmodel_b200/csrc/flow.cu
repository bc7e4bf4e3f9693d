// Resident sweeps without a barrier: a chunk of sweeps of a small lattice in one
// cooperative launch whose threads wait for their neighbours' sites instead of
// for the grid.
//
// The barrier form (resident.cu) spends more than half of a small lattice's pass
// in the barrier: the CTA's stores have to reach L2 before its arrival may be
// counted, the count has to reach L2, and a poll has to come back (about 1.1 of
// 2.0 us per pass at 32^3).  Here a thread holds one site of each colour
// (OwnSite) and publishes an updated site as one 128-bit word: the director, and
// the chirality's sign beside the number of the sweep.  A relaxed 128-bit access
// of device scope is one atomic access, so a reader that finds the sweep's number
// has the whole site, with no fence and no flag.  What a pass needs are its five
// neighbours in other threads' hands, which its loads poll for.
//
//   - The chirality's magnitude does not change in a sweep: every thread keeps
//     its neighbours' magnitudes and takes only the sign from the word.
//   - A word is overwritten only after its readers have read it: a site's next
//     value needs its neighbours' values of the pass between, which they publish
//     after reading this one.
//   - The first pass reads its neighbours from the lattice, and every thread
//     writes its two sites there at the end.
//   - Sweep numbers run on from launch to launch (the epoch word), so that a word
//     of an earlier launch is never taken for this one's.
//
// Only the step size needs the whole grid: while it is adapted, a sweep's first
// pass takes d from the count of the sweep before.  A warp of its own in each CTA
// brings the count out (one relaxed reduction) and d back (one polling lane), and
// the site warps meet it at named barriers, so that none of them waits for the
// CTA: their first trials are made with the d that comes out if the rule steps the
// same way again, which it mostly does, and are made anew where it does not.  The
// counts run on within a launch (three words in turn, told apart by how often each
// has been used), so nothing is cleared on the way.
//
// us per sweep on one B200 (kT 0.5, K 0.5, d adapted): the barrier form, this one
// with the count in the site warps and no guess, and its three further steps:
//
//   periodic         16^3   32^3   40^3   48^3    open  30x18x10  33x31x17  48^3
//   barrier          3.92   4.03   4.49   4.59          4.06      4.20      4.84
//   neighbours       3.30   3.29   3.59   3.88          3.35      3.49      3.93
//   control warp     2.86   2.84   3.18   3.42          3.03      3.30      3.48
//   proposal first   2.64   2.74   2.91   3.27          2.75      2.96      3.39
//   aligned          2.61   2.60   2.86   3.17          2.69      2.87      3.34
//
// (30^3, which had a launch per pass before: 7.0 and 2.9.)  Proposal first: what a
// trial does not need its neighbours for is done while they are on their way, and
// its acceptance is worked out for both outcomes of the trial before it.  What is
// left of a pass, 1.2 us with d fixed and 1.3 while it is adapted, is a store's way to
// L2 and a load's back, and more than that the dependent instructions of one site's
// trials, 470 per warp and pass on one warp per scheduler (issue active 18%, waits on
// fixed latencies twice those on loads).  Several polls in flight do not shorten it
// (32^3 with d fixed 2.43 against 2.36 us; the count's polls 2.73 against 2.70), and
// exchanging a CTA's own sites through shared memory, as the quench does, takes as
// long (2.67 against 2.60 us).
//
// Units, counters, arithmetic and control block are the fused form's bit for bit.
// Every wait is bounded; one that runs out sets the status word.
#include <cuda_runtime.h>

#include "resident.cuh"
#include "sweep.cuh"
#include "sweep_unit.cuh"

namespace chll {
namespace {

struct FlowArgs {
  LatticeView L;
  SweepGeom G;
  Coupling cp;
  PhiloxKeys keys;
  uint32_t replica;
  Control* ctl;
  unsigned long long* words;  // three count words, zero between launches
  uint32_t* epoch;
  uint4* xch;                 // a word per slot of both colours
  uint32_t per_colour;
  int nsweeps;
  uint32_t first_poll;
};

struct FlowShared {
  unsigned int cnt[2][kResThreads / 32];
  float d, guess;  // this sweep's step size, and the next one's by the same rule
  volatile int lost;
  // the control warp's values, here so that no register holds them
  double d64;
  unsigned long long open_acc, open_flip;  // left open by single passes
  unsigned long long before[3];            // each word's count up to its last use
};

// Named barriers between the site warps and the control warp: the sites' counts
// are in shared memory, the next step size is, and the last counts are.  Aligned:
// every warp is together there (the other form cost 0.1 us per sweep at 32^3).
enum FlowBarrier : int { kBarCounts = 1, kBarStep = 2, kBarEnd = 3 };

__device__ __forceinline__ void bar_arrive(int id) {
  __syncwarp();
  asm volatile("barrier.cta.arrive.aligned %0, %1;" ::"r"(id), "r"(blockDim.x) : "memory");
}
__device__ __forceinline__ void bar_wait(int id) {
  __syncwarp();
  asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(id), "r"(blockDim.x) : "memory");
}

constexpr int kUseShift = 52;  // count words: director accepts or flips below, arrivals above
constexpr unsigned long long kSumMask = (1ull << kUseShift) - 1;

template <bool P, bool LIMITED>
struct FlowSite {
  const FlowArgs& A;
  OwnSite<P> B;
  float mag[2][5];  // [colour]: |s| of that colour's site's neighbours +y, -y, +z, -z and x
  float ang, acc, flip;  // the next trials' random numbers (UnitRandoms)
  float mx, my, mz;      // the proposed director

  __device__ __forceinline__ explicit FlowSite(const FlowArgs& a)
      : A(a), B(a.L, a.G, blockIdx.x * (blockDim.x - 32) + threadIdx.x) {}

  // What colour C's next trials do not need the neighbours for.
  template <int C>
  __device__ __forceinline__ void draw(uint32_t step, float d) {
    const UnitRandoms u =
        unit_randoms(philox4x32_10({{B.g, step, A.replica, (uint32_t)C}}, A.keys));
    const bool second = (B.h & 1u) != 0;
    ang = second ? u.ang[1] : u.ang[0];
    acc = second ? u.acc[1] : u.acc[0];
    flip = second ? u.flip[1] : u.flip[0];
    propose<C>(d);
    asm volatile("" : "+f"(ang), "+f"(acc), "+f"(flip), "+f"(mx), "+f"(my), "+f"(mz));
  }
  template <int C>
  __device__ __forceinline__ void propose(float d) {
    propose_director(B.n[C].x, B.n[C].y, B.n[C].z, d, ang, mx, my, mz);
  }

  // The neighbours of colour C's site from the lattice, their magnitudes kept.
  template <int C>
  __device__ __forceinline__ void first(Nbrs& nb) {
    if (!B.has) return;
    B.template neighbours<C>(A.L, nb);
#pragma unroll
    for (int i = 0; i < 4; ++i) mag[C][i] = fabsf(nb.b[2 + i].w);
    mag[C][4] = fabsf(B.template odd<C>() ? nb.b[0].w : nb.b[1].w);
  }

  // The neighbours of colour C's site as published with `tag`.
  template <int C>
  __device__ __forceinline__ void wait(uint32_t tag, FlowShared& S, Nbrs& nb) {
    if (!B.has) return;
    const uint4* const oth = A.xch + (C ? 0u : A.per_colour);
    const bool o = B.template odd<C>();
    const uint32_t at[5] = {B.yp, B.ym, B.zp, B.zm, o ? B.xp : B.xm};
    bool open[5] = {B.hyp, B.hym, B.hzp, B.hzm, o ? B.hxp : B.hxm};
    float4 v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t polls = LIMITED ? A.first_poll : 0u;
    bool again;
    do {
      uint4 w[5];
#pragma unroll
      for (int i = 0; i < 5; ++i)
        if (open[i]) w[i] = ld_word(oth + at[i]);
      again = false;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        if (!open[i]) continue;
        if ((w[i].w & kTagMask) == (tag & kTagMask)) {
          v[i] = make_float4(__uint_as_float(w[i].x), __uint_as_float(w[i].y),
                             __uint_as_float(w[i].z),
                             __uint_as_float(__float_as_uint(mag[C][i]) | (w[i].w & ~kTagMask)));
          open[i] = false;
        } else {
          again = true;
        }
      }
      if (again && ++polls % 1024 == 0) {
        if (polls >= kWaitPolls || *(volatile unsigned int*)&A.ctl->status) S.lost = 1;
        again = !S.lost;  // a lost launch runs to its end without waiting
      }
    } while (again);
#pragma unroll
    for (int i = 0; i < 4; ++i) nb.b[2 + i] = v[i];
    nb.b[0] = o ? v[4] : B.n[C ^ 1];
    nb.b[1] = o ? B.n[C ^ 1] : v[4];
  }

  // unit_trials_drawn of one site, its operations; a trial's acceptance is worked
  // out for both outcomes of the trial before it.
  template <int C, bool FLIP_BEFORE, bool DIR, bool FLIP_AFTER>
  __device__ __forceinline__ void trial(const Nbrs& nb, unsigned int& nacc, unsigned int& nflip) {
    if (!B.has) return;
    float4& n = B.n[C];
    const Coupling& cp = A.cp;
    const bool v = B.template valid<C>();
    BondSums o, m;
    if (DIR)
      bond_sums2(n.x, n.y, n.z, mx, my, mz, nb, o, m);
    else
      o = bond_sums(n.x, n.y, n.z, nb);
    bool moved = false;
    if (DIR) moved = metropolis(director_dE(o, m, n.w, cp), acc, cp.inv_kT);
    if (FLIP_BEFORE) {
      const bool f = v && metropolis(flip_dE(o.c, n.w, cp), flip, cp.inv_kT);
      if (DIR) {
        const bool other = metropolis(director_dE(o, m, -n.w, cp), acc, cp.inv_kT);
        moved = f ? other : moved;
      }
      if (f) n.w = -n.w;
      nflip += (unsigned int)f;
    }
    if (DIR) {
      moved = v && moved;
      if (moved) {
        n.x = mx;
        n.y = my;
        n.z = mz;
      }
      nacc += (unsigned int)moved;
    }
    if (FLIP_AFTER) {
      const bool stay = metropolis(flip_dE(o.c, n.w, cp), flip, cp.inv_kT);
      const bool f =
          v && (DIR && moved ? metropolis(flip_dE(m.c, n.w, cp), flip, cp.inv_kT) : stay);
      if (f) n.w = -n.w;
      nflip += (unsigned int)f;
    }
  }

  template <int C>
  __device__ __forceinline__ void publish(uint32_t tag) const {
    if (B.has) st_word(A.xch + (C ? A.per_colour : 0u) + B.h, B.n[C], tag);
    __syncwarp();  // no lane waits before all have published
  }
};

// A warp's sum of one count into shared memory, for the control warp.
__device__ __forceinline__ void put_count(unsigned int (&part)[kResThreads / 32], unsigned int n) {
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = n;
}

// The last warp of a CTA: counts out, step sizes back.  One lane of it works.
template <bool LIMITED>
__device__ __forceinline__ void control_warp(const FlowArgs& A, FlowShared& S, int nadapt,
                                             uint32_t base) {
  Control* const ctl = A.ctl;
  const bool lead = (threadIdx.x & 31) == 0;
  const uint32_t nct = gridDim.x;
  const int site_warps = (int)(blockDim.x >> 5) - 1;
  int uses = 0;
  auto sum = [&](const unsigned int* part) {
    unsigned int t = 0;
    for (int w = 0; w < site_warps; ++w) t += part[w];
    return t;
  };
  // what the latest use of its word counted, once all CTAs have arrived there
  auto closed = [&](unsigned long long v) {
    const int w = (uses - 1) % 3;
    const unsigned long long t = v & kSumMask, n = t - S.before[w];
    S.before[w] = t;
    return n;
  };
  auto complete = [&](unsigned long long v) {
    return (uint32_t)(v >> kUseShift) == ((nct * (uint32_t)((uses + 2) / 3)) & 0xfffu);
  };
  auto accepted = [&](unsigned long long n) { return (float)n / (float)ctl->nsites; };
  for (int s = 0; s < A.nsweeps; ++s) {
    const bool last = s == A.nsweeps - 1;
    if (s >= nadapt && !last) continue;
    bar_wait(kBarCounts);
    if (lead) {
      unsigned long long* const word = A.words + (uses % 3) * kWordStride;
      const unsigned long long add = sum(S.cnt[s & 1]) + (1ull << kUseShift);
      asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(add) : "memory");
      ++uses;
      if (!last) {
        unsigned long long v;
        uint32_t polls = LIMITED ? A.first_poll : 0u;
        for (;;) {
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
          if (complete(v)) break;
          if (++polls % 1024 == 0) {
            if (polls >= kWaitPolls || *(volatile unsigned int*)&ctl->status) S.lost = 1;
            if (S.lost) break;
          }
        }
        // fused_close of pass B (chll_mod.f90:83-90)
        const float pa = accepted(closed(v) + (s == 0 ? S.open_acc : 0ull));
        S.d64 = adapt_d(S.d64, pa);
        S.d = (float)S.d64;
        S.guess = (float)adapt_d(S.d64, pa);
      }
    }
    if (!last) bar_arrive(kBarStep);
  }
  bar_wait(kBarEnd);
  if (!lead) return;
  if (S.lost) {
    set_status(ctl, 4u);
    atomicAdd(A.epoch, (uint32_t)A.nsweeps + 2u);  // what was published is never read again
    return;
  }
  // the CTA that completes the last word has both counts and writes the control
  // block; nobody waits for this word
  unsigned long long v, acc;
  const unsigned long long add = sum(S.cnt[A.nsweeps & 1]) + (1ull << kUseShift);
  asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;"
               : "=l"(v)
               : "l"(A.words + (uses % 3) * kWordStride), "l"(add)
               : "memory");
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
               : "=l"(acc)
               : "l"(A.words + ((uses - 1) % 3) * kWordStride)
               : "memory");
  const unsigned long long n = closed(acc) + (A.nsweeps == 1 ? S.open_acc : 0ull);
  ++uses;
  if (!complete(v + add)) return;
  const unsigned long long nfl = closed(v + add) + (A.nsweeps == 1 ? S.open_flip : 0ull);
  const float pa = accepted(n);
  ctl->d = A.nsweeps <= nadapt ? adapt_d(S.d64, pa) : S.d64;
  ctl->step = ctl->step + A.nsweeps;
  ctl->paccept = pa;
  ctl->nacc_last = (long long)n;
  ctl->nacc = 0;
  ctl->faccept = accepted(nfl);  // chll_mod.f90:93
  ctl->nflip_last = (long long)nfl;
  ctl->nflip = 0;
  *A.epoch = base + (uint32_t)A.nsweeps;
  clear_words(A.words);
}

// The other warps.  A sweep's first trials are made with the step size that the
// last change's rule gives again, while the count is on its way; where it turns
// out otherwise they are made anew.
template <bool P, bool LIMITED>
__device__ __forceinline__ void site_warps(const FlowArgs& A, FlowShared& S, int nadapt,
                                           uint32_t base, uint32_t step) {
  FlowSite<P, LIMITED> F(A);
  Nbrs nb;
  F.template first<1>(nb);
  F.template first<0>(nb);
  float d = S.d, guess = d;
  F.template draw<0>(step, d);
  unsigned int na, nf = 0, none = 0;
  for (int s = 0; s < A.nsweeps; ++s) {
    const bool last = s == A.nsweeps - 1;
    na = nf = 0;
    if (s) {
      F.template wait<0>(base + (uint32_t)s, S, nb);
      const float4 n = F.B.n[0];
      F.template trial<0, true, true, false>(nb, na, none);
      if (s <= nadapt) {
        bar_wait(kBarStep);
        d = S.d;
        if (d != guess) {
          F.B.n[0] = n;
          na = 0;
          F.template propose<0>(d);
          F.template trial<0, true, true, false>(nb, na, none);
        }
        guess = s < nadapt ? S.guess : d;
      }
    } else {
      F.template trial<0, false, true, false>(nb, na, none);
    }
    F.template publish<0>(base + (uint32_t)s + 1u);
    F.template draw<1>(step, d);
    F.template wait<1>(base + (uint32_t)s + 1u, S, nb);
    F.template trial<1, false, true, true>(nb, na, nf);
    F.template publish<1>(base + (uint32_t)s + 1u);
    if (s < nadapt || last) {
      put_count(S.cnt[s & 1], na);
      bar_arrive(kBarCounts);
    }
    ++step;
    F.template draw<0>(step, guess);
  }
  F.template wait<0>(base + (uint32_t)A.nsweeps, S, nb);
  F.template trial<0, true, false, false>(nb, none, nf);  // with B's flips: the sweep's
  if (F.B.has && !S.lost) {
    F.B.template store<0>(A.L);
    F.B.template store<1>(A.L);
  }
  put_count(S.cnt[A.nsweeps & 1], nf);
  bar_arrive(kBarEnd);
}

template <bool P, bool LIMITED>
__global__ void __launch_bounds__(kResThreads, 1)
    flow_sweeps_kernel(const __grid_constant__ FlowArgs A) {
  __shared__ FlowShared S;
  Control* const ctl = A.ctl;
  const uint32_t base = *(volatile uint32_t*)A.epoch;
  const uint32_t step = (uint32_t)ctl->step;
  const long long left = ctl->adapt_until - ctl->step;
  const int nadapt = left <= 0 ? 0 : (left < A.nsweeps ? (int)left : A.nsweeps);
  if (threadIdx.x == 0) {
    S.d64 = ctl->d;
    S.d = S.guess = (float)S.d64;
    S.open_acc = ctl->nacc;
    S.open_flip = ctl->nflip;
    S.before[0] = S.before[1] = S.before[2] = 0;
    S.lost = *(volatile unsigned int*)&ctl->status ? 1 : 0;
  }
  __syncthreads();
  const bool stale = S.lost;  // an earlier wait ran out: the words are not to be trusted
  __syncthreads();
  if (stale) return;
  if ((threadIdx.x >> 5) + 1 == blockDim.x >> 5)
    control_warp<LIMITED>(A, S, nadapt, base);
  else
    site_warps<P, LIMITED>(A, S, nadapt, base, step);
}

constexpr uint32_t kFlowSites = kResThreads - 32;  // site threads per SM beside the control warp

}  // namespace

// More than one CTA of threads with a site of each colour: up to 256 sites of a
// colour the barrier is the CTA's own (8^3: 1.9 us per sweep), and beyond 148 x 480
// the sites do not fit beside the control warps (52^3 3.8 us here, 53 x 52 x 52
// 5.0 with the barrier).
bool flow_pays(const LatticeView& L) {
  const uint32_t units = make_geom(L).units;
  return one_site_each(units, kFlowSites) && 2 * units > 256;
}

cudaError_t launch_flow_sweeps(const LatticeView& L, const Coupling& cp, uint32_t key0,
                               uint32_t key1, uint32_t replica, Control* ctl,
                               unsigned long long* words, void* xch, int nsweeps,
                               uint32_t wait_limit, cudaStream_t stream) {
  FlowArgs A;
  A.L = L;
  A.G = make_geom(L);
  A.cp = cp;
  A.keys = philox_keys(key0, key1);
  A.replica = replica;
  A.ctl = ctl;
  A.words = words;
  A.epoch = reinterpret_cast<uint32_t*>(words + 3 * kWordStride);
  A.xch = static_cast<uint4*>(xch);
  A.per_colour = 2 * A.G.units;
  A.nsweeps = nsweeps;
  A.first_poll = first_poll(wait_limit);
  uint32_t block, ctas;
  resident_shape(2 * A.G.units, block, ctas, kFlowSites);
  using Kernel = void (*)(const FlowArgs);
  static const Kernel kernels[2][2] = {
      {flow_sweeps_kernel<false, false>, flow_sweeps_kernel<false, true>},
      {flow_sweeps_kernel<true, false>, flow_sweeps_kernel<true, true>}};
  return launch_cooperative(kernels[L.periodic ? 1 : 0][A.first_poll ? 1 : 0], ctas, block + 32,
                            stream, A);
}

}  // namespace chll
