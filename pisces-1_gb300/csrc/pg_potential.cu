// V(r) on the grid: electron-water DPP model, Bloomfield ions, harmonic well.
//
// Compiled with -fmad=false: every product and sum is rounded separately, in
// the reference's evaluation order.  The differences from the CPU code are
// last-place ones: exp/erf, and the undamped inverse powers of R taken from
// one reciprocal square root per site instead of a square root and divisions;
// and a Slater core term c exp(-z R) with z R > 50 (below 2e-22 c) is not
// added.
//
// Layout: the reference's per-term lists (charges, dipoles, Slater cores,
// polarisable sites, each with a site index) are packed on the host into one
// 128-byte record per site, staged in shared memory in tiles.  Walking sites
// in site order keeps each term's sum in the reference's list order for the
// default model (its lists are all in site order), and the four sums are
// combined as Vpc + Vind + Vrep + Vpol (src/Potential.cpp:928).
//
// The kernel is bound by the FP64 pipe, which issues a warp-wide instruction
// about every 74 cycles per SM sub-partition here (the integer pipes one or
// two a cycle).  What need not be there is kept off it: the squares of the
// coordinate differences and the dipole products along each axis come from
// tables (k_site_axes; the same values, rounded the same way), a thread owns R
// points of one (x, y) column and forms their x and y part once, and flags
// and comparisons of non-negative values are integer operations.  That leaves
// about 90 of 145 FP64 instructions per water and point, mostly the
// reciprocal square roots and exponentials: (H2O)24 on 64^3 2.15 -> 1.45 ms,
// (H2O)128 on 160^3 136 -> 81 ms, the same bits.  (A 64-bit fixed-point
// evaluation takes 0.48 and 21 ms and is as exact, but V's last bits change
// with it, and a mixed solve carries those into the seventh digit and the
// sign of its states.)
#include <algorithm>
#include <cstdint>
#include <cmath>
#include <cstring>
#include <vector>

#include "pg_common.cuh"

namespace {

constexpr int kRec = 16;        // doubles per site record
constexpr int kTile = 64;       // records per shared-memory tile
constexpr int kPT = 64;         // threads per block: small blocks spread evenly over the SMs

// record fields
enum { R_X, R_Y, R_Z, R_Q, R_MX, R_MY, R_MZ, R_ALPHA, R_Z0, R_C0, R_Z1, R_C1, R_FLAGS };
enum { F_CHARGE = 1, F_DIPOLE = 2, F_POL = 4, F_ZPOS = 32 };  // bits 3..4: number of Slater terms; Slater exponents without a sign

constexpr double kStoCut = 50.0;  // z R beyond which a Slater core term is dropped
constexpr uint64_t kStoCutBits = 0x4049000000000000ull;  // its FP64 bits

__device__ __forceinline__ double reff(double r, double r0) {
  // Effective-distance damping (DampType 2), src/Potential.cpp:1192-1196.
  if (r < r0) {
    const double q = r / r0;
    return r0 * (0.5 + q * q * q * (1.0 - 0.5 * q));
  }
  return r;
}

// Tables of a site along one axis: d^2 and the dipole component times d, d =
// coordinate - site.
struct alignas(16) AxisEntry {
  double d2, m;
};

__global__ void k_site_axes(int nx, int ny, int nz, const double* __restrict__ xs, const double* __restrict__ ys,
                            const double* __restrict__ zs, const double* __restrict__ rec, int nrec,
                            AxisEntry* __restrict__ tab) {
  const int per = nx + ny + nz;
  const long total = (long)nrec * per;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const int s = (int)(e / per), c = (int)(e - (long)s * per);
    const int a = c < nx ? 0 : (c < nx + ny ? 1 : 2);
    const int i = a == 0 ? c : (a == 1 ? c - nx : c - nx - ny);
    const double* R = rec + (long)s * kRec;
    const double d = (a == 0 ? xs : (a == 1 ? ys : zs))[i] - R[R_X + a];
    tab[e] = AxisEntry{d * d, d * R[R_MX + a]};
  }
}

// Damping radii with the bits of their FP64 values: non-negative values
// compare as integers (a radius that is not positive matches nothing).
struct Damping {
  double q, d, p;
  uint64_t qb, db, pb;
};

__device__ __forceinline__ uint64_t bits_of(double x) { return (uint64_t)__double_as_longlong(x); }

// The terms of one site in FP64, added to the sums: r2 = R^2, mr = mu . R
// (distance table entry, src/Potential.cpp:136-146).  One reciprocal square
// root serves every undamped term (1/R, 1/R^3, 1/R^4); R = R^2 / R.  The
// damped branches (R < r0, including R = 0 on a site) keep the reference's
// divisions.
__device__ __forceinline__ void site_terms(const double* R, int flags, double r2, double mr, const Damping& D,
                                           double& pc, double& ind, double& rep, double& pol) {
  const double ir = rsqrt(r2);
  const double r = bits_of(r2) - 1 < 0x7ff0000000000000ull ? r2 * ir : 0.0;  // r2 > 0
  const uint64_t rb = bits_of(r);
  if (flags & F_CHARGE) pc += rb < D.qb ? -R[R_Q] / reff(r, D.q) : -R[R_Q] * ir;  // :1188-1204
  if (flags & F_DIPOLE) {                                                          // :1246-1262
    double m3;
    if (rb < D.db) {
      const double re = reff(r, D.d);
      m3 = 1.0 / (re * re * re);
    } else {
      m3 = ir * ir * ir;
    }
    ind += -mr * m3;
  }
  // repulsive Slater cores c exp(-z R) (:1301-1308); a term with z R >
  // kStoCut is below c e^-50 (< 1e-20 Eh for the water model's c <= 43) and
  // is not evaluated
  const int nsto = (flags >> 3) & 3;
  const bool zpos = flags & F_ZPOS;  // z R compares as an integer
  if (nsto > 0) {
    const double zr = R[R_Z0] * r;
    if (zpos ? bits_of(zr) < kStoCutBits : zr < kStoCut) rep += R[R_C0] * exp(-zr);
  }
  if (nsto > 1) {
    const double zr = R[R_Z1] * r;
    if (zpos ? bits_of(zr) < kStoCutBits : zr < kStoCut) rep += R[R_C1] * exp(-zr);
  }
  if (flags & F_POL) {  // :1350-1366
    if (rb < D.pb) {
      const double re = reff(r, D.p);
      const double re2 = re * re;
      pol += R[R_ALPHA] * r2 / (re2 * re2 * re2);
    } else {
      const double ir2 = ir * ir;
      pol += R[R_ALPHA] * (ir2 * ir2);
    }
  }
}

template <int R>
__global__ void __launch_bounds__(kPT) k_potential_dpp(int nx, int ny, int nz, const double* __restrict__ rec,
                                                       int nrec, const AxisEntry* __restrict__ axes,
                                                       const Damping D, double* __restrict__ v,
                                                       double* __restrict__ parts) {
  __shared__ __align__(16) double s_rec[kTile * kRec];
  __shared__ int s_flags[kTile];
  __shared__ AxisEntry s_z[kTile][R];
  const int tid = threadIdx.x;
  const long nxny = (long)nx * ny, N = nxny * nz;
  const int per = nx + ny + nz;  // table entries of a site
  const long p = blockIdx.x * (long)kPT + tid;
  const bool in = p < nxny;
  const int i = in ? (int)(p % nx) : 0, j = in ? (int)(p / nx) : 0;
  const int k0 = blockIdx.y * R;
  double vpc[R], vind[R], vrep[R], spol[R];
#pragma unroll
  for (int r = 0; r < R; ++r) vpc[r] = vind[r] = vrep[r] = spol[r] = 0.0;
  for (int s0 = 0; s0 < nrec; s0 += kTile) {
    const int cnt = nrec - s0 < kTile ? nrec - s0 : kTile;
    __syncthreads();
    for (int e = tid; e < cnt * kRec / 2; e += kPT)
      reinterpret_cast<double2*>(s_rec)[e] = reinterpret_cast<const double2*>(rec + (long)s0 * kRec)[e];
    for (int e = tid; e < cnt; e += kPT) s_flags[e] = (int)rec[(long)(s0 + e) * kRec + R_FLAGS];
    for (int e = tid; e < cnt * R; e += kPT) {
      const int s = e / R, r = e - s * R;
      s_z[s][r] = axes[(long)(s0 + s) * per + nx + ny + (k0 + r < nz ? k0 + r : nz - 1)];
    }
    __syncthreads();
    const AxisEntry* ap = axes + (long)s0 * per;
    AxisEntry tx = ap[i], ty = ap[nx + j];
    for (int s = 0; s < cnt; ++s) {
      const double xy2 = tx.d2 + ty.d2, xym = tx.m + ty.m;
      if (s + 1 < cnt) {
        ap += per;
        tx = ap[i];
        ty = ap[nx + j];
      }
      const int flags = s_flags[s];
#pragma unroll
      for (int r = 0; r < R; ++r)
        site_terms(s_rec + s * kRec, flags, xy2 + s_z[s][r].d2, xym + s_z[s][r].m, D, vpc[r], vind[r], vrep[r],
                   spol[r]);
    }
  }
  if (!in) return;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (k0 + r >= nz) break;
    const double vpol = spol[r] * -0.5;  // first-order polarisation, :884
    const long g = p + nxny * (k0 + r);
    v[g] = vpc[r] + vind[r] + vrep[r] + vpol;
    if (parts) {
      parts[g] = vpc[r];
      parts[N + g] = vind[r];
      parts[2 * N + g] = vrep[r];
      parts[3 * N + g] = vpol;
    }
  }
}

__global__ void k_potential_ions(int nx, int ny, int nz, const double* __restrict__ xs, const double* __restrict__ ys,
                                 const double* __restrict__ zs, const double* __restrict__ ion, int nions,
                                 double dcat, double dan, double* __restrict__ v) {
  const long N = (long)nx * ny * nz;
  for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < N; g += (long)gridDim.x * blockDim.x) {
    const int i = (int)(g % nx);
    const long r0 = g / nx;
    const double px = xs[i], py = ys[(int)(r0 % ny)], pz = zs[(int)(r0 / ny)];
    double acc = 0;
    for (int s = 0; s < nions; ++s) {  // src/NaCl.cpp:300-307
      const double rx = px - ion[4 * s], ry = py - ion[4 * s + 1], rz = pz - ion[4 * s + 2];
      const double r = sqrt(rx * rx + ry * ry + rz * rz);
      const double q = ion[4 * s + 3];
      const double damp = q > 0 ? dcat : dan;
      acc += -q * erf(damp * r) / r;
    }
    v[g] = v[g] + acc;
  }
}

__global__ void k_potential_spherical(int nx, int ny, int nz, const double* __restrict__ xs,
                                      const double* __restrict__ ys, const double* __restrict__ zs, double k,
                                      double* __restrict__ v) {
  const long N = (long)nx * ny * nz;
  for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < N; g += (long)gridDim.x * blockDim.x) {
    const int i = (int)(g % nx);
    const long r0 = g / nx;
    const double px = xs[i], py = ys[(int)(r0 % ny)], pz = zs[(int)(r0 / ny)];
    const double d = sqrt(px * px + py * py + pz * pz);  // src/Model_pot.cpp:147-149
    v[g] = 0.5 * k * d * d;
  }
}

// Device memory for the tables of one call, which waits for its stream before
// it returns: kept with the thread for the next call on the same device, up to
// kTablesMost; a larger buffer lasts for the call.
constexpr size_t kTablesMost = 32u << 20;
class CallTables {
 public:
  pg_status get(size_t bytes, unsigned char** p) {
    static thread_local struct {
      int device = -1;
      pg::DevBuf<unsigned char> buf;
    } kept;
    pg::DevBuf<unsigned char>* b = &own_;
    if (bytes <= kTablesMost) {
      int dev = 0;
      PG_CUDA_TRY(cudaGetDevice(&dev));
      if (dev != kept.device) kept.buf.release();
      kept.device = dev;
      b = &kept.buf;
    }
    PG_TRY(b->ensure(bytes));
    *p = b->p;
    return PG_OK;
  }

 private:
  pg::DevBuf<unsigned char> own_;
};

int grid_stride_blocks(long N) {
  long b = (N + 255) / 256;
  return (int)(b < 152L * 16 ? (b > 0 ? b : 1) : 152L * 16);
}

}  // namespace

extern "C" pg_status pg_potential_eval(const pg_grid* g, const pg_sites* t, double* v, double* parts, void* stream) {
  PG_ARG(g && t && v, "pg_potential_eval: null argument");
  PG_ARG(t->nsites >= 0 && (t->nsites == 0 || t->sites), "pg_potential_eval: bad site list");
  const int ns = t->nsites;
  std::vector<double> rec((size_t)(ns > 0 ? ns : 1) * kRec, 0.0);
  std::vector<int> nsto(ns, 0);
  for (int s = 0; s < ns; ++s)
    for (int c = 0; c < 3; ++c) rec[(size_t)s * kRec + c] = t->sites[3 * s + c];
  auto site_of = [&](const int* idx, int e, const char* what) -> long {
    const int s = idx[e];
    if (s < 0 || s >= ns) {
      pg::set_error("pg_potential_eval: %s %d refers to site %d of %d", what, e, s, ns);
      return -1;
    }
    return (long)s * kRec;
  };
  int flags_err = 0;
  std::vector<int> flags(ns, 0);
  for (int e = 0; e < t->ncharges; ++e) {
    const long o = site_of(t->charge_site, e, "charge");
    if (o < 0) return PG_BAD_ARG;
    if (flags[o / kRec] & F_CHARGE) flags_err = 1;
    flags[o / kRec] |= F_CHARGE;
    rec[o + R_Q] = t->charges[e];
  }
  for (int e = 0; e < t->ndipoles; ++e) {
    const long o = site_of(t->dipole_site, e, "dipole");
    if (o < 0) return PG_BAD_ARG;
    if (flags[o / kRec] & F_DIPOLE) flags_err = 1;
    flags[o / kRec] |= F_DIPOLE;
    for (int c = 0; c < 3; ++c) rec[o + R_MX + c] = t->dipoles[3 * e + c];
  }
  for (int e = 0; e < t->nsto; ++e) {
    const long o = site_of(t->sto_site, e, "Slater term");
    if (o < 0) return PG_BAD_ARG;
    const int k = nsto[o / kRec]++;
    if (k > 1) { flags_err = 1; continue; }
    rec[o + R_Z0 + 2 * k] = t->sto[2 * e];
    rec[o + R_C0 + 2 * k] = t->sto[2 * e + 1];
  }
  for (int e = 0; e < t->npol; ++e) {
    const long o = site_of(t->pol_site, e, "polarisable site");
    if (o < 0) return PG_BAD_ARG;
    if (flags[o / kRec] & F_POL) flags_err = 1;
    flags[o / kRec] |= F_POL;
    rec[o + R_ALPHA] = t->pol_alpha[e];
  }
  if (flags_err) {
    pg::set_error("pg_potential_eval: more than one charge, dipole or polarisable site, or more than two "
                  "Slater terms, on one site");
    return PG_UNSUPPORTED;
  }
  // The reference sums each term over its own list; walking records in site
  // order reproduces that order only if every list is sorted by site.
  for (int s = 0; s < ns; ++s) {
    double* R = &rec[(size_t)s * kRec];
    const bool zpos = !std::signbit(R[R_Z0]) && !std::signbit(R[R_Z1]);  // -0 R is not above 0 as an integer
    R[R_FLAGS] = (double)(flags[s] | ((nsto[s] > 2 ? 2 : nsto[s]) << 3) | (zpos ? F_ZPOS : 0));
  }

  if (ns == 0) {
    cudaStream_t st = pg::as_stream(stream);
    PG_CUDA_TRY(cudaMemsetAsync(v, 0, g->N * sizeof(double), st));
    if (parts) PG_CUDA_TRY(cudaMemsetAsync(parts, 0, 4 * g->N * sizeof(double), st));
    PG_CUDA_TRY(cudaStreamSynchronize(st));
    return PG_OK;
  }
  auto bits = [](double r) {
    uint64_t b = 0;
    if (r > 0) memcpy(&b, &r, 8);
    return b;
  };
  const Damping D{t->charge_damp,       t->dipole_damp,       t->pol_damp,
                  bits(t->charge_damp), bits(t->dipole_damp), bits(t->pol_damp)};
  cudaStream_t st = pg::as_stream(stream);
  const int per = g->n[0] + g->n[1] + g->n[2];
  // points per thread: four where that leaves every SM several blocks, fewer
  // on small grids (blocks of 64 threads spread evenly over the SMs: 64^3 in
  // 1.45 ms, with 128 threads 1.65)
  const long cols = (long)g->n[0] * g->n[1];
  const int R = g->N >= 200000 ? 4 : (g->N >= 80000 ? 2 : 1);
  const dim3 grid((unsigned)((cols + kPT - 1) / kPT), (unsigned)((g->n[2] + R - 1) / R));
  CallTables tables;
  unsigned char* tab = nullptr;
  const size_t rec_bytes = rec.size() * sizeof(double);  // a multiple of 128
  PG_TRY(tables.get(rec_bytes + (size_t)ns * per * sizeof(AxisEntry), &tab));
  double* drec = reinterpret_cast<double*>(tab);
  AxisEntry* daxes = reinterpret_cast<AxisEntry*>(tab + rec_bytes);
  PG_CUDA_TRY(cudaMemcpyAsync(drec, rec.data(), rec_bytes, cudaMemcpyHostToDevice, st));
  const long entries = (long)ns * per;
  k_site_axes<<<(unsigned)std::min<long>((entries + 255) / 256, 152L * 16), 256, 0, st>>>(
      g->n[0], g->n[1], g->n[2], g->x_dev[0].p, g->x_dev[1].p, g->x_dev[2].p, drec, ns, daxes);
  PG_TRY(pg::check_launch("k_site_axes"));
  const auto k = R == 4 ? k_potential_dpp<4> : (R == 2 ? k_potential_dpp<2> : k_potential_dpp<1>);
  k<<<grid, kPT, 0, st>>>(g->n[0], g->n[1], g->n[2], drec, ns, daxes, D, v, parts);
  PG_TRY(pg::check_launch("k_potential_dpp"));
  PG_CUDA_TRY(cudaStreamSynchronize(st));
  return PG_OK;
}

extern "C" pg_status pg_potential_ions_add(const pg_grid* g, int nions, const double* pos, const double* q,
                                           double r_cation, double r_anion, double* v, void* stream) {
  PG_ARG(g && v && nions >= 0 && (nions == 0 || (pos && q)), "pg_potential_ions_add: bad arguments");
  PG_ARG(r_cation > 0 && r_anion > 0, "pg_potential_ions_add: damping radii must be positive");
  if (nions == 0) return PG_OK;
  std::vector<double> ion(4 * (size_t)nions);
  for (int s = 0; s < nions; ++s) {
    for (int c = 0; c < 3; ++c) ion[4 * s + c] = pos[3 * s + c];
    ion[4 * s + 3] = q[s];
  }
  CallTables tables;
  unsigned char* tab = nullptr;
  PG_TRY(tables.get(ion.size() * sizeof(double), &tab));
  double* d = reinterpret_cast<double*>(tab);
  cudaStream_t st = pg::as_stream(stream);
  PG_CUDA_TRY(cudaMemcpyAsync(d, ion.data(), ion.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  k_potential_ions<<<grid_stride_blocks(g->N), 256, 0, st>>>(g->n[0], g->n[1], g->n[2], g->x_dev[0].p,
                                                             g->x_dev[1].p, g->x_dev[2].p, d, nions,
                                                             1.0 / r_cation, 1.0 / r_anion, v);
  PG_TRY(pg::check_launch("k_potential_ions"));
  PG_CUDA_TRY(cudaStreamSynchronize(st));
  return PG_OK;
}

extern "C" pg_status pg_potential_spherical(const pg_grid* g, double k, double* v, void* stream) {
  PG_ARG(g && v, "pg_potential_spherical: null argument");
  k_potential_spherical<<<grid_stride_blocks(g->N), 256, 0, pg::as_stream(stream)>>>(
      g->n[0], g->n[1], g->n[2], g->x_dev[0].p, g->x_dev[1].p, g->x_dev[2].p, k, v);
  return pg::check_launch("k_potential_spherical");
}
