// Host-side launchers of the device kernels (one translation unit each).
#pragma once
#include <cuda_runtime.h>

#include "chll_common.cuh"

namespace chll {

// sweep.cu: per-device launch shapes (call once per device, outside any
// stream capture) and one half-sweep (pass = kPassDir0..kPassSpin1).
void sweep_prepare();
// Sweep form: the two-pass fused sweep, the fused passes of a chunk in one
// cooperative launch (flow.cu or resident.cu; auto picks it where resident_pays,
// else the fused sweep), or the reference's four half-sweeps with the direct
// kernel or the staged kernel (shared-memory tiles by bulk copies).  All give the
// same chain.  Single half-sweeps (chll_lattice_pass) use the direct kernel unless
// staged is chosen.
enum SweepKernel : int {
  kSweepAuto = 0,
  kSweepDirect = 1,
  kSweepStaged = 2,
  kSweepFused = 3,
  kSweepResident = 4
};
void launch_sweep_pass(const LatticeView& L, const Coupling& cp, uint32_t key0, uint32_t key1,
                       uint32_t replica, Control* ctl, int pass, cudaStream_t stream,
                       int kernel = kSweepAuto);
bool staged_fits(const LatticeView& L);
// Fused sweep passes (sweep.cu): A0 = director trials of colour 0 (first
// sweep), A = previous sweep's colour-0 flips + colour-0 director trials,
// B = colour-1 director trials + colour-1 flips (ends the sweep),
// F = previous sweep's colour-0 flips (after the last sweep).
enum FusedPhase : int { kFusedA0 = 0, kFusedA = 1, kFusedB = 2, kFusedF = 3 };
void launch_fused_pass(const LatticeView& L, const Coupling& cp, uint32_t key0, uint32_t key1,
                       uint32_t replica, Control* ctl, int phase, cudaStream_t stream);
// The same on an explicit unit range and boundary mode (sweep_unit.cuh:
// make_slab_geom, BoundaryMode), for a z-slab with halo planes.  peer_lo /
// peer_hi: where the range's first / last plane is also written (the halo
// planes of the neighbouring slabs, 32-byte aligned), or null.
struct SweepGeom;
void launch_fused_pass(const LatticeView& L, const SweepGeom& G, int bmode, const Coupling& cp,
                       uint32_t key0, uint32_t key1, uint32_t replica, Control* ctl, int phase,
                       cudaStream_t stream, float4* peer_lo = nullptr,
                       float4* peer_hi = nullptr);
// The control update of a fused pass when the control block defers it.
void launch_control_update(Control* ctl, int phase, cudaStream_t stream);

// resident.cu: nsweeps fused sweeps of a whole lattice (A0 B (A B)... F, the
// same chain and control block as the fused passes) in one cooperative launch
// whose CTAs meet at a grid barrier between passes.  words: kResidentWordBytes
// of device memory, zero before the first launch (a launch leaves them zero).
// resident_fits: the lattice's counts fit the words; resident_pays: the form
// is faster than the fused passes' launches.
// The words' memory is kResidentAllocBytes: behind them flow.cu's sweep number.
// wait_limit, here and below: polls that a wait makes before it gives up and sets
// the control block's status word; at most kWaitPolls.
constexpr uint32_t kWaitPolls = 1u << 22;
constexpr size_t kResidentWordBytes = 3 * 128, kResidentAllocBytes = 4 * 128;
bool resident_fits(const LatticeView& L);
bool resident_pays(const LatticeView& L);
cudaError_t launch_resident_sweeps(const LatticeView& L, const Coupling& cp, uint32_t key0,
                                   uint32_t key1, uint32_t replica, Control* ctl,
                                   unsigned long long* words, int nsweeps, uint32_t wait_limit,
                                   cudaStream_t stream);

// flow.cu: the same for small lattices, threads waiting for their neighbours'
// sites instead of the grid.  xch: flow_bytes of device memory, zero before the
// first launch; it and the words' sweep number are left alone between launches.
bool flow_pays(const LatticeView& L);
inline size_t flow_bytes(const LatticeView& L) {
  return 2 * (size_t)L.hx * L.nj * L.nk * sizeof(float4);
}
cudaError_t launch_flow_sweeps(const LatticeView& L, const Coupling& cp, uint32_t key0,
                               uint32_t key1, uint32_t replica, Control* ctl,
                               unsigned long long* words, void* xch, int nsweeps,
                               uint32_t wait_limit, cudaStream_t stream);

// layout.cu: natural-order (F-order, i fastest) <-> red/black float4.
void launch_pack_f64(const LatticeView& L, const double* nx, const double* ny, const double* nz,
                     const int* s, cudaStream_t stream);
void launch_unpack_f64(const LatticeView& L, double* nx, double* ny, double* nz, int* s,
                       cudaStream_t stream);
void launch_pack_f4(const LatticeView& L, const float4* xyzs, cudaStream_t stream);
void launch_unpack_f4(const LatticeView& L, float4* xyzs, cudaStream_t stream);
void launch_init_random(const LatticeView& L, uint32_t key0, uint32_t key1, uint32_t replica,
                        cudaStream_t stream, uint64_t site0 = 0);

// observables.cu: FP64 moments and the measurement row.  step: the row's step
// column, or kStepOfControl for the control block's last completed step.
constexpr long long kStepOfControl = -0x7fffffffffffffffll;
int observables_max_blocks();
void launch_observables(const LatticeView& L, const CouplingD& cp, const Control* ctl,
                        double* partials, unsigned int* ticket, double* row, long long step,
                        cudaStream_t stream);
struct MomentGeom;
void launch_observables(const LatticeView& L, const MomentGeom& M, const CouplingD& cp,
                        const Control* ctl, double* partials, unsigned int* ticket, double* row,
                        long long step, cudaStream_t stream);

// adjoint.cu: energy gradient.
void launch_energy_grad(const LatticeView& L, const CouplingD& cp, float4* grad_rb, int project,
                        double* partials, unsigned int* ticket, double* out4,
                        cudaStream_t stream);
// The same of natural-order arrays n (3 per site), s: the gradient (3 per site,
// or null) and the sums E and dE/d(eps, K, h); partials: kGradMaxBlocks * 4.
cudaError_t launch_natural_grad(int ni, int nj, int nk, int periodic, const float* n,
                                const float* s, const CouplingD& cd, float* grad, int project,
                                double* partials, double* energy, double* derivs,
                                cudaStream_t stream);
// The adjoint kernels run at most kGradMaxBlocks CTAs (grid-stride beyond
// that), each leaving four FP64 partial sums: the partial-sum buffers of the
// adjoint hold kGradMaxBlocks * 4 doubles on any GPU.
constexpr int kGradMaxBlocks = 148 * 4;
int energy_grad_max_blocks();
// adjoint.cu: one colour of the zero-temperature gradient quench.
void launch_quench_pass(const LatticeView& L, const CouplingD& cd, float eta, int colour,
                        cudaStream_t stream);

// adjoint.cu: nsteps quench steps (a pass of colour 0, then 1) in one
// cooperative launch; words as launch_resident_sweeps, xch as launch_flow_sweeps.
// quench_resident_pays: faster than the passes' launches.
bool quench_resident_pays(const LatticeView& L);
int quench_flow_sites(const LatticeView& L);  // nonzero: launch_quench_resident uses xch
cudaError_t launch_quench_resident(const LatticeView& L, const CouplingD& cd, float eta,
                                   Control* ctl, unsigned long long* words, void* xch, int nsteps,
                                   uint32_t wait_limit, cudaStream_t stream);

// analysis.cu: shell correlations over natural-order float4 sites and a zero
// site behind them (offsets {di, dj, dk}, chunks {first, end, shell} of at most
// kCorrChunk offsets of one shell; out = [sum (n.n')^2 per shell, sum s s' per
// shell, sum s]; partials: blocks * (2 nshells + 1) doubles for blocks =
// shell_corr_blocks), the chirality histogram along an integer direction p of
// m = p . (i+1, j+1, k+1) - m0, and its transform.
constexpr int kCorrChunk = 128;  // FP32 terms per running sum
constexpr int kMaxCorrShells = 64;
constexpr int kMaxProjectionBins = 12288;  // 48 KB of shared int bins
int shell_corr_blocks(int nshells);
void launch_shell_corr(const float4* site, int ni, int nj, int nk, const int4* offs,
                       const int4* chunks, int nchunks, int nshells, bool wrap, double* partials,
                       int blocks, double* out, cudaStream_t stream);
void launch_projection(const LatticeView& L, int px, int py, int pz, long long m0, int nbins,
                       unsigned long long* hist, cudaStream_t stream);
void launch_structure_factor(const unsigned long long* hist, long long m0, int nbins,
                             const double* kvs, int nkv, double nsites, double* sf,
                             cudaStream_t stream);

}  // namespace chll
