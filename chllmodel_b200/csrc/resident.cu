// Resident sweeps: a whole chunk of fused sweeps of one lattice in ONE
// cooperative launch whose CTAs stay on the SMs and meet at a grid barrier
// between passes.
//
// What bounds a small lattice's sweep is latency: at 32^3 a pass holds 8,192
// units, and as a launch of its own it takes 3.3 us, most of it the grid's
// start and drain, the read of the control block and the count epilogue.
// Here a pass is its loads (L2: the lattice was written by other SMs a pass
// earlier), one site's or unit's serial trial arithmetic, and the barrier, about
// 0.8 us of 128 CTAs.  So the sites are spread over all SMs, as few warps on each
// as there can be: a thread holds one site of each colour while that fits (37 k
// units), then one unit, then several, and the threads per CTA come from their
// number per SM.  Lattices of a site per thread and more than one CTA leave the
// barrier out (flow.cu, which sweeps take there).  us per sweep on one B200
// (periodic, kT 0.5, K 0.5; one cluster: a form of 16 CTAs with the hardware
// cluster barrier, whose 16 SMs had to issue every instruction of the pass):
//
//   edge                    8     16    24    32    48    64    96    128   200
//   passes launched each   5.8   5.8   6.4   6.6   6.9   7.9   14.2  25.6  84.8
//   one cluster            3.5   5.4   5.5   5.6  14.5
//   this form              1.9   3.9   4.0   4.0   4.6   6.1   12.4  23.2  78.6
//   flow.cu                      2.6   2.6   2.6   3.2
//
// The barrier and the counts are one 64-bit word per pass: a CTA adds its
// accept counts and its arrival with one release reduction and polls the
// word (acquire) until every CTA has arrived, so the wait already holds the
// pass's total; every CTA then derives the next d and step from it with the
// control update's arithmetic (fused_close), and the chain -- units, counters,
// arithmetic, control block -- is the fused form's bit for bit.  Every wait is
// bounded; one that runs out sets the control block's status word, and
// launches do nothing until set_control clears it.
#include <cuda_runtime.h>

#include "resident.cuh"
#include "sweep.cuh"
#include "sweep_unit.cuh"

namespace chll {
namespace {

struct ResidentArgs {
  LatticeView L;
  SweepGeom G;
  WalkGeom W;
  Coupling cp;
  PhiloxKeys keys;
  uint32_t replica;
  Control* ctl;
  unsigned long long* words;
  int nsweeps;
  uint32_t first_poll;
};

struct ResidentShared {
  unsigned int cnt[2][kResThreads / 32];
  double d;
  long long step;
  unsigned long long nacc, nflip;
  float paccept;
  int ok;
};

// Which trials a phase runs, of which colour (sweep.cuh FusedPhase).
template <int PHASE>
struct PhaseOf {
  static constexpr int C = PHASE == kFusedB ? 1 : 0;
  static constexpr bool flip_before = PHASE == kFusedA || PHASE == kFusedF;
  static constexpr bool dir = PHASE != kFusedF;
  static constexpr bool flip_after = PHASE == kFusedB;
};

// Lattices of more units than threads: the plain kernels' column walk or
// unit loop, with coherent loads that the compiler keeps between the barriers
// around a pass.
template <bool P, int FORM>
struct SharedUnits {
  const ResidentArgs& A;
  __device__ __forceinline__ explicit SharedUnits(const ResidentArgs& a) : A(a) {}

  template <int C>
  __device__ __forceinline__ void draw(uint32_t) {}

  template <int PHASE>
  __device__ __forceinline__ void pass(uint32_t step, float d, unsigned int& nacc,
                                       unsigned int& nflip) {
    using T = PhaseOf<PHASE>;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned int na = 0, nf = 0;
    if (FORM == 2) {
      for (uint32_t t = first; t < A.W.ntasks; t += stride)
        walk_task<T::C, P, P, T::flip_before, T::dir, T::flip_after, kLoadCoherentOrdered>(
            A.L, A.W, t, step, d, A.cp, A.keys, A.replica, na, nf);
    } else {
      const uint32_t plane = (uint32_t)A.L.hx * (uint32_t)A.L.nj;
      const uint32_t per_colour = plane * (uint32_t)A.L.nk;
      for (uint32_t g = first; g < A.G.units; g += stride) {
        if (g + stride < A.G.units) prefetch_unit<T::C>(A.L, g + stride, plane, per_colour);
        unit_step<T::C, P, P, T::flip_before, T::dir, T::flip_after, FORM != 0,
                  kLoadCoherentOrdered>(A.L, A.G, g, step, d, A.cp, A.keys, A.replica, na, nf);
      }
    }
    nacc = na;
    nflip = nf;
  }
};

// Lattices of at most one unit per thread (48^3 5.1 against 5.4 us per sweep
// with the unit loop, 64^3 6.5 against 7.1): the block in registers
// (resident.cuh), and the pass's random words drawn while the barrier before it
// is waited for.
template <bool P>
struct OwnUnit {
  const ResidentArgs& A;
  OwnBlock<P> B;
  Ctr4 words;

  __device__ __forceinline__ explicit OwnUnit(const ResidentArgs& a) : A(a), B(a.L, a.G) {}

  // The random words of the next pass (colour C, step): independent of the
  // lattice, so they are drawn before the wait.
  template <int C>
  __device__ __forceinline__ void draw(uint32_t step) {
    words = philox4x32_10({{B.g, step, A.replica, (uint32_t)C}}, A.keys);
    asm volatile("" : "+r"(words.v[0]), "+r"(words.v[1]), "+r"(words.v[2]), "+r"(words.v[3]));
  }

  template <int PHASE>
  __device__ __forceinline__ void pass(uint32_t, float d, unsigned int& nacc,
                                       unsigned int& nflip) {
    using T = PhaseOf<PHASE>;
    constexpr int C = T::C;
    nacc = nflip = 0;
    if (!B.has) return;
    Nbrs nb0, nb1;
    B.template neighbours<C>(A.L, nb0, nb1);
    const bool odd = B.template odd<C>();
    unit_trials_drawn<T::flip_before, T::dir, T::flip_after>(
        B.n[C][0], B.n[C][1], nb0, nb1, odd ? B.v[1] : B.v[0], odd ? B.v[3] : B.v[2],
        unit_randoms(words), d, A.cp, nacc, nflip);
    st_unit(A.L.col[C] + B.u, B.n[C][0], B.n[C][1]);
  }
};

// The same with a site of each colour per thread.
template <bool P>
struct OwnSiteUnit {
  const ResidentArgs& A;
  OwnSite<P> B;
  Ctr4 words;

  __device__ __forceinline__ explicit OwnSiteUnit(const ResidentArgs& a) : A(a), B(a.L, a.G) {}

  template <int C>
  __device__ __forceinline__ void draw(uint32_t step) {
    words = philox4x32_10({{B.g, step, A.replica, (uint32_t)C}}, A.keys);
    asm volatile("" : "+r"(words.v[0]), "+r"(words.v[1]), "+r"(words.v[2]), "+r"(words.v[3]));
  }

  template <int PHASE>
  __device__ __forceinline__ void pass(uint32_t, float d, unsigned int& nacc,
                                       unsigned int& nflip) {
    using T = PhaseOf<PHASE>;
    constexpr int C = T::C;
    nacc = nflip = 0;
    if (!B.has) return;
    Nbrs nb;
    B.template neighbours<C>(A.L, nb);
    // this site's numbers of the unit's call first; the second site is not there
    UnitRandoms u = unit_randoms(words);
    const bool second = (B.h & 1u) != 0;
    u.acc[0] = second ? u.acc[1] : u.acc[0];
    u.ang[0] = second ? u.ang[1] : u.ang[0];
    u.flip[0] = second ? u.flip[1] : u.flip[0];
    float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    unit_trials_drawn<T::flip_before, T::dir, T::flip_after>(B.n[C], none, nb, nb,
                                                             B.template valid<C>(), false, u, d,
                                                             A.cp, nacc, nflip);
    B.template store<C>(A.L);
  }
};

// The CTA's counts of a pass (thread 0): director accepts, and flips where
// they are wanted.  Ends with the CTA's stores ordered before thread 0's
// release.
__device__ __forceinline__ unsigned long long cta_counts(ResidentShared& S, unsigned int na,
                                                         unsigned int nf, bool flips) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  na = __reduce_add_sync(0xffffffffu, na);
  if (flips) nf = __reduce_add_sync(0xffffffffu, nf);
  if (lane == 0) {
    S.cnt[0][warp] = na;
    if (flips) S.cnt[1][warp] = nf;
  }
  __syncthreads();
  unsigned long long v = 0;
  if (threadIdx.x == 0) {
    unsigned int a = 0, f = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a += S.cnt[0][w];
      if (flips) f += S.cnt[1][w];
    }
    v = (unsigned long long)a | ((unsigned long long)f << kCountBits);
  }
  return v;
}

// The chunk: A0 B (A B)... F with the grid barrier after every pass but the
// last.  The control values live in shared memory, thread 0's to change: kept in
// registers across the passes they cost the unit loops theirs.
template <class UNITS, bool LIMITED>
__device__ __forceinline__ void resident_sweeps(const ResidentArgs& A, ResidentShared& S) {
  Control* ctl = A.ctl;
  if (ctl->status) return;  // an earlier wait ran out: the words are not to be trusted
  if (threadIdx.x == 0) {
    S.d = ctl->d;
    S.step = ctl->step;
    S.nacc = ctl->nacc;  // left open by single passes
    S.nflip = ctl->nflip;
    S.ok = 1;
  }
  uint32_t step = (uint32_t)ctl->step;
  uint32_t slot = 0;  // word of the pass
  unsigned int na, nf;
  UNITS units(A);
  units.template draw<0>(step);
  __syncthreads();
  // thread 0: this pass's word, complete; the word before it cleared
  auto wait = [&](unsigned long long v) {
    bool ok = true;
    v = grid_wait(A.words + slot * kWordStride, v, gridDim.x, LIMITED ? A.first_poll : 0u, ok);
    if (blockIdx.x == 0) A.words[(slot == 0 ? 2 : slot - 1) * kWordStride] = 0;
    S.nacc += v & kCountMask;
    S.ok = ok;
    return v;
  };
  for (int s = 0; s < A.nsweeps; ++s) {
    const bool last = s == A.nsweeps - 1;
    if (s)
      units.template pass<kFusedA>(step, (float)S.d, na, nf);
    else
      units.template pass<kFusedA0>(step, (float)S.d, na, nf);
    unsigned long long v = cta_counts(S, na, nf, false);
    if (threadIdx.x == 0) grid_arrive(A.words + slot * kWordStride, v, gridDim.x);
    units.template draw<1>(step);
    if (threadIdx.x == 0) wait(v);
    slot = slot == 2 ? 0 : slot + 1;
    __syncthreads();
    if (!S.ok) break;
    units.template pass<kFusedB>(step, (float)S.d, na, nf);
    v = cta_counts(S, na, nf, last);
    if (threadIdx.x == 0) grid_arrive(A.words + slot * kWordStride, v, gridDim.x);
    units.template draw<0>(step + 1u);
    if (threadIdx.x == 0) {
      // both outcomes of adapt_d ahead of the wait
      double dn = adapt_d(S.d, 0.f), up = adapt_d(S.d, 1.f);
      asm volatile("" : "+d"(dn), "+d"(up));
      v = wait(v);
      // the control update that closes the director count (fused_close)
      const float pa = (float)S.nacc / (float)ctl->nsites;  // chll_mod.f90:83
      S.paccept = pa;
      if (S.step < ctl->adapt_until) {
        if ((double)pa < 0.4) S.d = dn;
        else if ((double)pa > 0.6) S.d = up;
      }
      ++S.step;
      if (last) {
        // earlier flips were closed by this sweep's pass A
        S.nflip = (s ? 0ull : S.nflip) + (v >> kCountBits & kCountMask);
      } else {
        S.nacc = 0;
      }
    }
    slot = slot == 2 ? 0 : slot + 1;
    ++step;
    __syncthreads();
    if (!S.ok) break;
  }
  if (!S.ok) {
    if (threadIdx.x == 0) set_status(ctl, 4u);
    return;
  }
  units.template pass<kFusedF>(step, (float)S.d, na, nf);
  unsigned long long v = cta_counts(S, 0, nf, true);
  if (threadIdx.x != 0) return;
  // the CTA that completes the closing pass's word has the flip count and
  // writes the control block
  if (gridDim.x > 1) {
    const unsigned long long old =
        atomicAdd(A.words + slot * kWordStride, v + (1ull << kArriveShift));
    if ((uint32_t)(old >> kArriveShift) != gridDim.x - 1) return;
    v += old;
    clear_words(A.words);
  }
  const unsigned long long nflip = S.nflip + (v >> kCountBits & kCountMask);
  ctl->d = S.d;
  ctl->step = S.step;
  ctl->paccept = S.paccept;
  ctl->nacc_last = (long long)S.nacc;
  ctl->nacc = 0;
  ctl->faccept = (float)nflip / (float)ctl->nsites;  // chll_mod.f90:93
  ctl->nflip_last = (long long)nflip;
  ctl->nflip = 0;
}

template <bool P, int FORM, bool LIMITED>
__global__ void __launch_bounds__(kResThreads, 1)
    resident_sweeps_kernel(const __grid_constant__ ResidentArgs A) {
  __shared__ ResidentShared S;
  if (FORM == 4)
    resident_sweeps<OwnSiteUnit<P>, LIMITED>(A, S);
  else if (FORM == 3)
    resident_sweeps<OwnUnit<P>, LIMITED>(A, S);
  else
    resident_sweeps<SharedUnits<P, FORM>, LIMITED>(A, S);
}

using ResidentKernel = void (*)(const ResidentArgs);
template <bool LIMITED>
ResidentKernel resident_kernel(int periodic, int form) {
  // [periodic][form]: 0 unit loop with padding checks, 1 unit loop, 2 column
  // walk, 3 one unit per thread, 4 one site of each colour per thread
  static const ResidentKernel kernels[2][5] = {
      {resident_sweeps_kernel<false, 0, LIMITED>, resident_sweeps_kernel<false, 1, LIMITED>,
       resident_sweeps_kernel<false, 2, LIMITED>, resident_sweeps_kernel<false, 3, LIMITED>,
       resident_sweeps_kernel<false, 4, LIMITED>},
      {resident_sweeps_kernel<true, 0, LIMITED>, resident_sweeps_kernel<true, 1, LIMITED>,
       resident_sweeps_kernel<true, 2, LIMITED>, resident_sweeps_kernel<true, 3, LIMITED>,
       resident_sweeps_kernel<true, 4, LIMITED>}};
  return kernels[periodic][form];
}

}  // namespace

// A pass's counts fit 26 bits (fewer than 2^27 sites).
bool resident_fits(const LatticeView& L) {
  return 2 * (uint64_t)make_geom(L).units < (1ull << kCountBits);
}

// Against a launch per pass: always where a thread holds one site of each colour
// or one unit (50^3 periodic 3.7 against 7.5 us, 64^3 6.1 against 7.9).  Beyond
// that the barrier still saves about 1 us per pass, but the loops' coherent
// loads cost the units more than the read-only ones do.  With unpadded rows it
// pays up to 256^3 (4 M units) periodic (128^3 23.2 against 25.6 us, 200^3 78.6
// against 84.8, 256^3 167 against 175) and 200^3 (2 M units) open (128^3 24.6
// against 26.0, 176^3 56.4 against 60.1, 200^3 81.3 against 84.9, 256^3 180 against
// 178; 192^3 alone loses, 82.6 against 81.1); with padded rows
// it does not (130^3 open 31.1 against 29.7, 150 x 125 x 101 28.1 against 27.2).
bool resident_pays(const LatticeView& L) {
  const uint32_t units = make_geom(L).units;
  return one_site_each(units) || one_unit_each(L, units) ||
         (L.ni % 4 == 0 && units <= (L.periodic ? 1u << 22 : 1u << 21));
}

cudaError_t launch_resident_sweeps(const LatticeView& L, const Coupling& cp, uint32_t key0,
                                   uint32_t key1, uint32_t replica, Control* ctl,
                                   unsigned long long* words, int nsweeps, uint32_t wait_limit,
                                   cudaStream_t stream) {
  ResidentArgs A;
  A.L = L;
  A.G = make_geom(L);
  const bool full = L.ni % 4 == 0;
  const bool own = one_unit_each(L, A.G.units);
  const bool site = one_site_each(A.G.units);
  uint32_t block, ctas;
  resident_shape(site ? 2 * A.G.units : A.G.units, block, ctas);
  const uint32_t ncols = A.G.Q * (uint32_t)L.nj;
  uint32_t seg = 0;
  if (full && !own && !site)
    walk_pass_cost(A.G.units, ncols, (uint32_t)L.nk, true, ctas * block, -1, &seg);
  A.W = make_walk(A.G, L, seg ? seg : 1);
  const int form = site ? 4 : (own ? 3 : (seg ? 2 : (full ? 1 : 0)));
  A.cp = cp;
  A.keys = philox_keys(key0, key1);
  A.replica = replica;
  A.ctl = ctl;
  A.words = words;
  A.nsweeps = nsweeps;
  A.first_poll = first_poll(wait_limit);
  const int periodic = L.periodic ? 1 : 0;
  return launch_cooperative(A.first_poll ? resident_kernel<true>(periodic, form)
                                         : resident_kernel<false>(periodic, form),
                            ctas, block, stream, A);
}

}  // namespace chll
