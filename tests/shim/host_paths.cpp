// Host paths of the library on a CUDA runtime without a GPU (fake_cudart).
// One case per run: its name is the argument, the exit status says whether it
// holds.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

#include "fake_cudart.hpp"
#include "pisces_gb300.h"

namespace {

#define REQUIRE(cond)                                                                    \
  do {                                                                                   \
    if (!(cond)) {                                                                       \
      fprintf(stderr, "%s:%d: %s (%s)\n", __FILE__, __LINE__, #cond, pg_last_error());   \
      return 1;                                                                          \
    }                                                                                    \
  } while (0)

bool is(const std::string& kernel, const char* name) { return kernel.find(name) != std::string::npos; }

pg_grid* grid(int nx, int ny, int nz) {
  const int n[3] = {nx, ny, nz};
  const double L[3] = {0.6 * (nx + 1), 0.6 * (ny + 1), 0.6 * (nz + 1)};
  pg_grid* g = nullptr;
  if (pg_grid_create(n, L, &g) != PG_OK) fprintf(stderr, "grid: %s\n", pg_last_error());
  return g;
}

// A polarisation model on the first npp sites.
struct Model {
  std::vector<double> sites, inva, epc;
  std::vector<int> pol;
  pg_sites t{};
  pg_scpol_model m{};
  explicit Model(int npp) {
    for (int i = 0; i < 3 * npp; ++i) sites.push_back(0.25 * i - 3.0), epc.push_back(0.01 * i);
    inva.assign((size_t)9 * npp * npp, 0.125);
    for (int i = 0; i < npp; ++i) pol.push_back(i);
    t.nsites = npp;
    t.sites = sites.data();
    m.npp = npp;
    m.pol_site = pol.data();
    m.inva = inva.data();
    m.epc = epc.data();
    m.damp_type = 2;
    m.damp = 2.0;
  }
};

// The positions that the field kernel is given are the sites', also where the
// runtime reads pageable host memory only when the stream gets to the copy.
int scpol_upload() {
  pg_grid* g = grid(6, 5, 4);
  Model a(7);
  std::vector<double> v(g ? pg_grid_npoints(g) : 1), psi(v.size());
  const double* pos = nullptr;
  std::vector<double> seen;
  fake::state().on_launch = [&](const std::string& k, void** args) {
    if (is(k, "k_scpol_field")) pos = *static_cast<const double**>(args[9]);
  };
  fake::state().on_wait = [&] {
    if (pos && seen.empty()) seen.assign(pos, pos + 21);
  };
  fake::state().defer_copies = true;
  REQUIRE(pg_potential_scpol_add(g, &a.t, &a.m, v.data(), nullptr, nullptr) == PG_OK);
  REQUIRE(seen == a.sites);
  pos = nullptr;
  seen.clear();
  std::vector<double> grad(21), tmu(21), mcm(441);
  REQUIRE(pg_hf_gradient_grid(g, &a.t, &a.m, psi.data(), grad.data(), tmu.data(), mcm.data(), nullptr) == PG_OK);
  REQUIRE(seen == a.sites);
  pg_grid_destroy(g);
  return 0;
}

// The FP64 calls queue, and depend on no status word: the kernels finish their
// outputs whatever their waits do, so a word that an earlier product of the
// mixed form has set is neither reported nor cleared by them.
int hx_status() {
  pg_grid* g = grid(32, 32, 32);
  const long N = g ? pg_grid_npoints(g) : 1;
  std::vector<double> buf(16 * N + 2);
  double* v = buf.data() + ((size_t)buf.data() % 16 ? 1 : 0);
  double *x = v + N, *y = x + N;
  bool fail = true;
  REQUIRE(pg_grid_set_hx_kernel(g, 1) == PG_OK);  // the axis passes: k_hx_tc, whose last argument is the word
  fake::state().on_launch = [&](const std::string& k, void** args) {
    if (fail && is(k, "k_hx_tcILi")) **static_cast<int**>(args[14]) = 1;
  };
  const int waits = fake::state().waits;
  REQUIRE(pg_hx(g, v, x, y, 1, PG_FP64, nullptr) == PG_OK && fake::state().waits == waits);
  REQUIRE(pg_hx(g, v, x, y, 1, PG_MIXED, nullptr) == PG_DEVICE_TIMEOUT);
  fail = false;
  REQUIRE(pg_hx(g, v, x, y, 1, PG_FP64, nullptr) == PG_OK);
  const double sigma = -0.1;
  REQUIRE(pg_kinetic_precondition(g, x, 1, &sigma, PG_FP64, nullptr) == PG_OK);
  Model a(7);
  REQUIRE(pg_potential_scpol_add(g, &a.t, &a.m, v, nullptr, nullptr) == PG_OK);
  REQUIRE(pg_grid_check(g, nullptr) == PG_DEVICE_TIMEOUT);
  REQUIRE(pg_grid_check(g, nullptr) == PG_OK);
  REQUIRE(pg_hx(g, v, x, y, 1, PG_MIXED, nullptr) == PG_OK);
  pg_grid_destroy(g);
  return 0;
}

// On a stream that is being captured the FP64 form only queues.
int hx_captured() {
  pg_grid* g = grid(66, 20, 20);
  const long N = g ? pg_grid_npoints(g) : 1;
  std::vector<double> v(N), x(N), y(N);
  fake::state().capturing = true;
  REQUIRE(pg_hx(g, v.data(), x.data(), y.data(), 1, PG_FP64, nullptr) == PG_OK);
  fake::state().capturing = false;
  pg_grid_destroy(g);
  return 0;
}

// Kernels that need more shared memory than the default get it on every device
// they run on.
int second_device() {
  for (int dev = 0; dev < 3; ++dev) {
    REQUIRE(cudaSetDevice(dev) == cudaSuccess);
    pg_grid* g = grid(66, 20, 20);
    const long N = g ? pg_grid_npoints(g) : 1;
    std::vector<double> v(N), x(N * 44), y(N * 44), out(40 * 4);
    const double sigma = -0.1;
    REQUIRE(pg_hx(g, v.data(), x.data(), y.data(), 1, PG_FP64, nullptr) == PG_OK);
    REQUIRE(pg_kinetic_precondition(g, x.data(), 1, &sigma, PG_FP64, nullptr) == PG_OK);
    for (int precision : {PG_FP64, PG_MIXED})
      REQUIRE(pg_block_gram(N, x.data(), 40, y.data(), 4, out.data(), precision, nullptr) == PG_OK);
    REQUIRE(fake::state().refused.empty());
    pg_grid_destroy(g);
  }
  return 0;
}

// The tables of a V(r) call lie on the device that the call runs on, and what
// a thread keeps of them between calls is bounded.
int potential_tables() {
  std::vector<double> sites(3 * 60000, 0.5), q(60000, -0.1);
  std::vector<int> at(60000);
  for (int i = 0; i < 60000; ++i) at[i] = i;
  std::vector<const void*> seen;
  fake::state().on_launch = [&](const std::string& k, void** args) {
    if (is(k, "k_potential_dpp")) seen = {*static_cast<void**>(args[3]), *static_cast<void**>(args[5])};
    if (is(k, "k_potential_ions")) seen = {*static_cast<void**>(args[6])};
  };
  for (int dev : {0, 1, 0}) {
    REQUIRE(cudaSetDevice(dev) == cudaSuccess);
    pg_grid* g = grid(20, 12, 10);
    std::vector<double> v(g ? pg_grid_npoints(g) : 1);
    pg_sites t{};
    t.sites = sites.data();
    t.charges = q.data();
    t.charge_site = at.data();
    t.charge_damp = 1.7;
    for (int ns : {5, 60000, 7}) {
      t.nsites = t.ncharges = ns;
      const size_t before = fake::kept_on(dev);
      REQUIRE(pg_potential_eval(g, &t, v.data(), nullptr, nullptr) == PG_OK);
      for (const void* p : seen) REQUIRE(fake::device_of(p) == dev || ns == 60000);
      REQUIRE(seen.size() == 2 && fake::kept_on(dev) <= before + (32u << 20));
    }
    REQUIRE(pg_potential_ions_add(g, 3, sites.data(), q.data(), 1.0, 1.0, v.data(), nullptr) == PG_OK);
    for (const void* p : seen) REQUIRE(fake::device_of(p) == dev);
    pg_grid_destroy(g);
  }
  return 0;
}

// The tiles of an axis are spread over the SMs that the device has.
int slice_grids() {
  std::pair<unsigned, unsigned> want[2] = {{13, 2}, {4, 1}};  // 400 lines of 66 points, two column chunks
  for (int dev : {0, 1}) {
    REQUIRE(cudaSetDevice(dev) == cudaSuccess);
    fake::state().sms = dev == 0 ? 152 : 6;
    pg_grid* g = grid(66, 20, 20);
    std::vector<double> v(g ? pg_grid_npoints(g) : 1), x(v), y(v);
    REQUIRE(pg_hx(g, v.data(), x.data(), y.data(), 1, PG_FP64, nullptr) == PG_OK);
    bool seen = false;
    for (auto& k : fake::state().grids)
      if (is(k.first, "k_slice_axisILi2ELb1E")) seen = k.second == want[dev];
    REQUIRE(seen);
    pg_grid_destroy(g);
  }
  return 0;
}

// What grids keep between calls is given back: on request, with the grid, and
// before an allocation is given up.
int kept_buffers() {
  pg_grid *a = grid(30, 20, 20), *b = grid(66, 20, 20);
  const long N = pg_grid_npoints(b);
  std::vector<double> r(8 * N), v(N), vec(2 * N), ev(2);
  const std::vector<double> sigma(8, -0.1);
  auto precondition = [&](pg_grid* g, int k) {
    return pg_kinetic_precondition(g, r.data(), k, sigma.data(), PG_FP64, nullptr);
  };
  REQUIRE(pg_release_buffers() == 0);
  const size_t bare = fake::kept_on(0);
  REQUIRE(precondition(b, 4) == PG_OK);
  const size_t kept = fake::kept_on(0) - bare;
  REQUIRE(kept >= 8u * 8u * (size_t)N);
  REQUIRE(precondition(b, 2) == PG_OK && fake::kept_on(0) - bare == kept);
  REQUIRE(pg_release_buffers() == (long)kept && fake::kept_on(0) == bare);
  // no room for a's scratch but b's
  REQUIRE(precondition(b, 4) == PG_OK);
  fake::state().memory = fake::state().in_use + 1000;
  REQUIRE(precondition(a, 4) == PG_OK);
  REQUIRE(precondition(b, 4) == PG_OK);
  // nothing to give back: refused, and the grid is as it was
  fake::state().memory = bare + 1000;
  pg_release_buffers();
  REQUIRE(precondition(a, 4) == PG_OOM);
  fake::state().memory = (size_t)-1;
  REQUIRE(precondition(a, 4) == PG_OK);
  pg_release_buffers();
  // the buffers of a solve
  pg_solve_params p{};
  p.nroots = 2;
  p.maxsub = 8;
  p.maxiter = 1;
  p.ptol = 5;
  p.corrflag = 1;
  p.startvec = 1;
  pg_solve(b, v.data(), &p, ev.data(), vec.data(), nullptr, nullptr);
  const size_t solve = fake::kept_on(0);
  REQUIRE(solve >= bare + 2u * 8u * 8u * (size_t)N);
  fake::state().memory = fake::state().in_use + 1000;
  REQUIRE(precondition(a, 4) == PG_OK);
  REQUIRE(fake::kept_on(0) < solve);
  fake::state().memory = (size_t)-1;
  pg_solve(b, v.data(), &p, ev.data(), vec.data(), nullptr, nullptr);
  pg_grid_destroy(b);
  REQUIRE(precondition(a, 4) == PG_OK);
  pg_grid_destroy(a);
  REQUIRE(pg_release_buffers() == 0);
  return 0;
}

// Work counters of a stream whose first use is captured: zero when the call
// returns, not once the graph has run (the stream may be used before).
int captured_counters() {
  pg_grid* g = grid(32, 32, 32);
  const long N = g ? pg_grid_npoints(g) : 1;
  std::vector<double> buf(4 * N + 2);
  double* x = buf.data() + ((size_t)buf.data() % 16 ? 1 : 0);
  for (int kind : {3, 2}) {  // FP16 split, TF32 split
    REQUIRE(pg_grid_set_hx_kernel(g, kind) == PG_OK);
    fake::state().capturing = true;
    REQUIRE(pg_hx_async(g, x + 2 * N, x, x + N, 1, PG_MIXED, nullptr) == PG_OK);
    REQUIRE(fake::state().recorded == 0);
    fake::state().capturing = false;
  }
  pg_grid_destroy(g);
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  const std::map<std::string, std::function<int()>> cases = {
      {"scpol_upload", scpol_upload},
      {"hx_status", hx_status},
      {"hx_captured", hx_captured},
      {"second_device", second_device},
      {"potential_tables", potential_tables},
      {"slice_grids", slice_grids},
      {"kept_buffers", kept_buffers},
      {"captured_counters", captured_counters},
  };
  const auto it = cases.find(argc > 1 ? argv[1] : "");
  return it == cases.end() ? 2 : it->second();
}
