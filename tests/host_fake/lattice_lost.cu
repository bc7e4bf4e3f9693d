// A wait that gave up (a launch that sets the control block's status word) is
// reported by every call that waits for the lattice's stream, and by run(), until
// set_control; run() leaves the caller's arrays alone.  With an argument: copies of a
// run that fail.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/chll_mod.h"
#include "fake_cuda.h"
#include "../../chllmodel_b200/csrc/moments.cuh"
#include "stubs.h"

static int bad = 0;
static bool lose = false;
static int sweeps = 0;

static void expect(bool ok, const char* what) {
  if (!ok) {
    std::printf("wrong: %s (%s)\n", what, chll_last_error());
    ++bad;
  }
}

static void launch(chll::Control* ctl, int n) {
  if (ctl->status) return;
  if (lose) {
    ctl->status = 4;
    *ctl->host_status = 4;
  } else {
    ctl->step += n;
  }
}

namespace chll {
bool resident_fits(const LatticeView&) { return true; }
bool resident_pays(const LatticeView&) { return true; }
bool flow_pays(const LatticeView& L) { return L.ni > 8; }
bool quench_resident_pays(const LatticeView&) { return true; }
int quench_flow_sites(const LatticeView&) { return 1; }
bool staged_fits(const LatticeView&) { return true; }
int energy_grad_max_blocks() { return 8; }
int observables_max_blocks() { return 8; }
int shell_corr_blocks(int) { return 8; }
cudaError_t launch_flow_sweeps(const LatticeView&, const Coupling&, uint32_t, uint32_t, uint32_t,
                               Control* ctl, unsigned long long*, void*, int n, uint32_t, cudaStream_t) {
  launch(ctl, n);
  return cudaSuccess;
}
cudaError_t launch_resident_sweeps(const LatticeView&, const Coupling&, uint32_t, uint32_t, uint32_t,
                                   Control* ctl, unsigned long long*, int n, uint32_t, cudaStream_t) {
  launch(ctl, n);
  return cudaSuccess;
}
cudaError_t launch_quench_resident(const LatticeView&, const CouplingD&, float, Control* ctl,
                                   unsigned long long*, void*, int, uint32_t, cudaStream_t) {
  launch(ctl, 0);
  return cudaSuccess;
}
void launch_sweep_pass(const LatticeView&, const Coupling&, uint32_t, uint32_t, uint32_t, Control* ctl,
                       int, cudaStream_t, int) {
  launch(ctl, 1);
}
void launch_pack_f64(const LatticeView&, const double*, const double*, const double*, const int*,
                     cudaStream_t) {}
void launch_unpack_f64(const LatticeView&, double*, double*, double*, int*, cudaStream_t) {}
void launch_unpack_f4(const LatticeView&, float4*, cudaStream_t) {}
void launch_init_random(const LatticeView&, uint32_t, uint32_t, uint32_t, cudaStream_t, uint64_t) {}
void launch_observables(const LatticeView&, const MomentGeom&, const CouplingD&, const Control*,
                        double*, unsigned int*, double* row, long long, cudaStream_t) {
  for (int c = 0; c < kRowLen; ++c) row[c] = c + 0.5;
}
void launch_energy_grad(const LatticeView&, const CouplingD&, float4*, int, double*, unsigned int*,
                        double* out4, cudaStream_t) {
  for (int c = 0; c < 4; ++c) out4[c] = c + 0.25;
}
void launch_shell_corr(const float4*, int, int, int, const int4*, const int4*, int, int, bool, double*,
                       int, double*, cudaStream_t) {}
void launch_projection(const LatticeView&, int, int, int, long long, int, unsigned long long*,
                       cudaStream_t) {}
void launch_structure_factor(const unsigned long long*, long long, int, const double*, int, double,
                             double*, cudaStream_t) {}
}  // namespace chll

// Every call that waits for the stream, each on its own first.
static void calls(chll_lattice* L, const chll_coupling* c, int sites, int want, const char* after) {
  std::vector<float> f4(4 * sites);
  std::vector<double> x(sites), y(sites), z(sites);
  std::vector<int> s(sites);
  double row[16] = {}, measured[16] = {}, out4[4] = {}, d = 0, gn[2], gs[2], cnt[2], kv = 0.1, sf;
  long long m0, hist[64];
  int nb = 0;
  const int plane[3] = {1, 0, 0};
  int64_t step;
  auto is = [&](int rc, const char* what) {
    if (rc != want) {
      std::printf("wrong: %s after %s gives %d (%s)\n", what, after, rc, chll_last_error());
      ++bad;
    }
  };
  is(chll_lattice_sync(L), "sync");
  is(chll_lattice_observe(L, c, row), "observe");
  is(chll_lattice_read_rows(L, measured, 0, 1), "read_rows");
  is(chll_lattice_energy_grad(L, c, nullptr, 0, out4), "energy_grad");
  is(chll_lattice_energy_grad(L, c, f4.data(), 0, nullptr), "energy_grad without sums");
  is(chll_lattice_download_f4(L, f4.data()), "download_f4");
  is(chll_lattice_download_f64(L, x.data(), y.data(), z.data(), s.data()), "download_f64");
  is(chll_lattice_shell_corr(L, 2, 0, gn, gs, cnt), "shell_corr");
  is(chll_lattice_projection(L, plane, hist, &m0, &nb), "projection");
  is(chll_lattice_structure_factor(L, plane, &kv, 1, &sf), "structure_factor");
  is(chll_lattice_get_control(L, &d, &step, nullptr, nullptr), "get_control");
  if (want == CHLL_OK) {
    expect(row[14] == 14.5 && out4[3] == 3.25, "results");
  }
}

// Every copy of a run that fails is reported.
static void run_copies() {
  const int edge = 12, sites = edge * edge * edge;
  chll_run_config cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.kT = cfg.K = cfg.eps = 1.0;
  cfg.d = 0.1;
  std::vector<double> x(sites), y(sites), z(sites), m(5 * 2), rows(2 * 16);
  std::vector<int> s(sites), steps(2);
  double d;
  for (int verbose : {0, 1}) {
    cfg.verbose = verbose;
    int nth = 0;
    do {
      fake::fail_copy = ++nth;
      const int rc = chll_run_ex(&cfg, 1, 20, 10, x.data(), y.data(), z.data(), s.data(), edge, edge,
                                 edge, steps.data(), m.data(), rows.data(), &d);
      const int want = fake::fail_copy ? CHLL_OK : CHLL_ECUDA;
      if (rc != want) {
        std::printf("wrong: run gives %d where copy %d of it fails\n", rc, nth);
        ++bad;
      }
    } while (!fake::fail_copy);
    fake::fail_copy = 0;
    expect(nth > 10, "copies of a run");
  }
}

int main(int argc, char**) {
  if (argc > 1) {
    run_copies();
    std::printf("%d wrong\n", bad);
    return bad != 0;
  }
  const chll_coupling c = {0.5, 1.0, 0.0, 1.0};
  for (int edge : {8, 12}) {
    const int sites = edge * edge * edge;
    for (const char* form : {"sweep", "quench", "staged", "staged pass"}) {
      // the first call after the lost launch is another one each time
      for (int first = 0; first < 2; ++first) {
        chll_lattice* L = nullptr;
        expect(chll_lattice_create(edge, edge, edge, CHLL_PERIODIC, &L) == CHLL_OK, "create");
        expect(chll_lattice_reserve_rows(L, 4) == CHLL_OK, "rows");
        if (std::strncmp(form, "staged", 6) == 0) chll_lattice_set_kernel(L, 2);
        auto go = [&] {
          if (std::strcmp(form, "quench") == 0)
            expect(chll_lattice_quench(L, &c, 0.05, 3) == CHLL_OK, "quench");
          else if (std::strcmp(form, "staged pass") == 0)
            expect(chll_lattice_pass(L, &c, 1, 0, 0) == CHLL_OK, "pass");
          else  // another number of sweeps each time: a new graph of the staged passes
            expect(chll_lattice_sweep(L, &c, 1, 0, ++sweeps) == CHLL_OK, "sweep");
        };
        lose = false;
        go();
        calls(L, &c, sites, CHLL_OK, form);
        lose = true;
        go();
        lose = false;
        if (first) {
          double d;
          int64_t step;
          expect(chll_lattice_get_control(L, &d, &step, nullptr, nullptr) == CHLL_EDEVICE, "control");
        }
        calls(L, &c, sites, CHLL_EDEVICE, form);
        go();
        calls(L, &c, sites, CHLL_EDEVICE, form);
        expect(chll_lattice_set_control(L, 0.1, 1, 100) == CHLL_OK, "set_control");
        go();
        calls(L, &c, sites, CHLL_OK, form);
        chll_lattice_destroy(L);
      }
    }
    // run(): chll_run_ex, then the reference's entry point
    chll_run_config cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.kT = cfg.K = cfg.eps = 1.0;
    cfg.d = 0.1;
    cfg.adapt_until = 10000;
    std::vector<double> x(sites, 2.0), y(sites, 3.0), z(sites, 4.0), m(5 * 2), rows(2 * 16);
    std::vector<int> s(sites, 7), steps(2, -1);
    double d = -1.0;
    for (int verbose : {0, 1}) {
      cfg.verbose = verbose;
      lose = true;
      expect(chll_run_ex(&cfg, 1, 20, 10, x.data(), y.data(), z.data(), s.data(), edge, edge, edge,
                         steps.data(), m.data(), rows.data(), &d) == CHLL_EDEVICE,
             "run that lost a wait");
      expect(d == -1.0 && steps[0] == -1, "its results are not handed out");
      for (int i = 0; i < sites; ++i) bad += x[i] != 2.0 || y[i] != 3.0 || z[i] != 4.0 || s[i] != 7;
      lose = false;
    }
    lose = true;
    int one = 1, twenty = 20, ten = 10, nsub = 0, e = edge;
    double g = 0, K = 1, dd = 0.1, kbt = 1;
    run(&one, &twenty, &ten, x.data(), y.data(), z.data(), s.data(), nullptr, nullptr, nullptr, &g, &K,
        &dd, &kbt, &e, &e, &e, &nsub, steps.data(), m.data());
    expect(chll_last_status() == CHLL_EDEVICE && dd == 0.1, "run()");
    lose = false;
    expect(chll_run_ex(&cfg, 1, 20, 10, x.data(), y.data(), z.data(), s.data(), edge, edge, edge,
                       steps.data(), m.data(), rows.data(), &d) == CHLL_OK,
           "run after it");
    expect(d == 0.1 && steps[1] == 20 && rows[16 + 14] == 14.5, "its results");
  }
  std::printf("%d wrong\n", bad);
  return bad != 0;
}
