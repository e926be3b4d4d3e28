// Y = H X on the 3-D sine-DVR grid, FP64 form.
//
// H = diag(V) + Tx (+) Ty (+) Tz: for every grid point and vector,
//   y = v x + sum_b Tx[i,b] x[b,j,k] + sum_b Ty[j,b] x[i,b,k] + sum_b Tz[k,b] x[i,j,b]
// (src/mtx.cpp:35-104 applies the same operator line by line with dspmv).
// Three axis contractions from slices of both operands on the tensor cores
// (pg_slice.cu): z with V X, then y and x added to Y.
//
// k_hx_fp64 and k_axis_fp64 are the same contractions as chains of FP64
// multiply-adds in a fixed order, bound by that pipe (344 us against 63 at
// 64^3 x 4, the pipe 98 % active).  They serve the FP64 solver of several
// roots, whose states come out of a restart with signs that the rounding noise
// of the products decides: with another product the states are the same to
// 1e-14, but a third of them change sign, and a solve keeps the states it has
// always returned; and they serve grids that are very small, or whose T the
// slices do not hold (chain_is_shorter, t_sliced).
#include <algorithm>
#include <type_traits>

#include "pg_slice.cuh"

namespace {

// One thread owns one grid point for four vectors (four independent
// accumulators), in the last group of blocks for the REST that are left over;
// operand loads are coalesced or warp-wide broadcasts.  Every vector of a body
// exists: one left out by a predicate would take the FP64 pipe as long as any
// other, and the predicates keep the loads from running ahead.  All groups are
// one launch: on small grids the ones left over cost as much time as a group
// of four, beside which they now run.
template <int NV>
__device__ __forceinline__ void hx_point(int nx, int ny, int nz, const double* __restrict__ tx,
                                         const double* __restrict__ ty, const double* __restrict__ tz,
                                         const double* __restrict__ v, const double* __restrict__ Xv,
                                         double* __restrict__ Yv, long N, long g) {
  const int i = (int)(g % nx);
  const long r = g / nx;
  const int j = (int)(r % ny);
  const int k = (int)(r / ny);
  double acc[NV];
  const double vg = v[g];
#pragma unroll
  for (int q = 0; q < NV; ++q) acc[q] = vg * Xv[(long)q * N + g];
  // x sweep: T[b][i] (coalesced over i), x[b,j,k] broadcast
  {
    const long base = (long)nx * (j + (long)ny * k);
#pragma unroll 4
    for (int b = 0; b < nx; ++b) {
      const double t = tx[(long)b * nx + i];
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q] += t * Xv[(long)q * N + base + b];
    }
  }
  // y sweep: Ty[j][b] broadcast, x[i,b,k] coalesced
  {
    const long base = i + (long)nx * ny * k;
    const double* trow = ty + (long)j * ny;
#pragma unroll 4
    for (int b = 0; b < ny; ++b) {
      const double t = trow[b];
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q] += t * Xv[(long)q * N + base + (long)nx * b];
    }
  }
  // z sweep: Tz[k][b] broadcast, x[i,j,b] coalesced
  {
    const long base = i + (long)nx * j;
    const long sz = (long)nx * ny;
    const double* trow = tz + (long)k * nz;
#pragma unroll 4
    for (int b = 0; b < nz; ++b) {
      const double t = trow[b];
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q] += t * Xv[(long)q * N + base + sz * b];
    }
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) Yv[(long)q * N + g] = acc[q];
}

// Groups blockIdx.y < four take four vectors each, the next one the REST.
template <int REST>
__global__ void __launch_bounds__(256) k_hx_fp64(int nx, int ny, int nz, const double* __restrict__ tx,
                                                 const double* __restrict__ ty, const double* __restrict__ tz,
                                                 const double* __restrict__ v, const double* __restrict__ X,
                                                 double* __restrict__ Y, int four) {
  const long N = (long)nx * ny * nz;
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= N) return;
  const long off = 4l * blockIdx.y * N;
  if (REST == 0 || (int)blockIdx.y < four) hx_point<4>(nx, ny, nz, tx, ty, tz, v, X + off, Y + off, N, g);
  else hx_point<REST == 0 ? 4 : REST>(nx, ny, nz, tx, ty, tz, v, X + off, Y + off, N, g);
}

// Y (mode) A x_axis X: one axis contraction in FP64, mode 0 write, 1 add, for
// vectors v0 .. v0 + nv - 1.  The bodies as above; the groups of four keep
// their predicates (nv is not a constant there): without them the compiler runs
// more loads ahead and the pass is slower (six passes, 96^3 x 8: 6.84 ms, 8.13).
template <int NV>
__device__ __forceinline__ void axis_point(int na, int idx, long stride, const double* __restrict__ A,
                                           const double* __restrict__ X, double* __restrict__ Y, long N, long g,
                                           int mode, int v0, int nv) {
  const long base = g - (long)idx * stride;
  double acc[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) acc[q] = (q < nv && mode == 1) ? Y[(long)(v0 + q) * N + g] : 0.0;
  const double* arow = A + (long)idx * na;
  for (int b = 0; b < na; ++b) {
    const double t = arow[b];
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (q < nv) acc[q] += t * X[(long)(v0 + q) * N + base + (long)b * stride];
  }
#pragma unroll
  for (int q = 0; q < NV; ++q)
    if (q < nv) Y[(long)(v0 + q) * N + g] = acc[q];
}

template <int REST>
__global__ void __launch_bounds__(256) k_axis_fp64(int nx, int ny, int nz, int axis, const double* __restrict__ A,
                                                   const double* __restrict__ X, double* __restrict__ Y, int four,
                                                   int mode) {
  const long N = (long)nx * ny * nz;
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= N) return;
  const int i = (int)(g % nx);
  const long r = g / nx;
  const int j = (int)(r % ny);
  const int k = (int)(r / ny);
  const int na = axis == 0 ? nx : (axis == 1 ? ny : nz);
  const int idx = axis == 0 ? i : (axis == 1 ? j : k);
  const long stride = axis == 0 ? 1 : (axis == 1 ? nx : (long)nx * ny);
  const int v0 = 4 * blockIdx.y, nv = 4 * four + REST - v0;
  if (REST == 0 || (int)blockIdx.y < four) axis_point<4>(na, idx, stride, A, X, Y, N, g, mode, v0, nv < 4 ? nv : 4);
  else axis_point<REST == 0 ? 4 : REST>(na, idx, stride, A, X, Y, N, g, mode, v0, REST);
}

}  // namespace

namespace pg {

pg_status tc_axis(const pg_grid* g, int a, const float* Ahi, const float* Alo, const double* v, const double* x,
                  double* y, int nvec, int mode, cudaStream_t st);

// Launches an in-order kernel over nvec vectors: launch(REST, blocks, four).
// A launch for the groups of four and one for the rest took, for 5 vectors on
// 12^3 / 28^3 / 64^3, 25.1 / 51.8 / 474 us, one launch of predicated groups 16.7 /
// 50.6 / 716, and one launch with a body for the rest 16.6 / 31.3 / 417.
template <typename F>
static void by_vectors(long N, int nvec, const F& launch) {
  const int four = nvec / 4, rest = nvec % 4;
  const dim3 blocks((unsigned)((N + 255) / 256), (unsigned)(four + (rest ? 1 : 0)));
  if (rest == 0) launch(std::integral_constant<int, 0>(), blocks, four);
  if (rest == 1) launch(std::integral_constant<int, 1>(), blocks, four);
  if (rest == 2) launch(std::integral_constant<int, 2>(), blocks, four);
  if (rest == 3) launch(std::integral_constant<int, 3>(), blocks, four);
}

pg_status axis_apply(const pg_grid* g, int axis, const SliceMat& S, const double* A64, const float* Ahi,
                     const float* Alo, const double* x, double* y, int nvec, int mode, int precision,
                     cudaStream_t st, bool in_order) {
  PG_ARG(g && x && y && x != y && axis >= 0 && axis < 3 && (mode == 0 || mode == 1), "axis_apply: bad arguments");
  if (precision == PG_MIXED) return tc_axis(g, axis, Ahi, Alo, nullptr, x, y, nvec, mode, st);
  if (!in_order) return slice_axis(g, axis, S, A64, nullptr, x, y, nvec, mode, st);
  by_vectors(g->N, nvec, [&](auto rest, dim3 blocks, int four) {
    k_axis_fp64<rest.value><<<blocks, 256, 0, st>>>(g->n[0], g->n[1], g->n[2], axis, A64, x, y, four, mode);
  });
  return check_launch("k_axis_fp64");
}

// Whether the chain of multiply-adds is as fast as the slices, for this grid and
// block.  Its one launch lasts as long as the FP64 pipe needs for a block of
// 256 points on an SM, 78 ns for each multiply-add of a point, times the turns
// its blocks take; the slices' three launches take 21 to 27 us on grids that
// small, whatever their size (back to back, us, chain / slices: 8^3 x 1 9 / 21,
// 12^3 x 8 17 / 21, 16^3 x 40 30 / 26).  Up to 36 multiply-adds a value, whose
// roundings stay near the slices' few; longer chains round more (on 15x17x16
// beyond four roundings of a value's terms) and are not taken for speed.
static bool chain_is_shorter(const pg_grid* g, int nvec) {
  const long blocks = (g->N + 255) / 256 * ((nvec + 3) / 4);
  const long sms = sm_count(g->device);
  const int terms = g->n[0] + g->n[1] + g->n[2];
  return terms <= 36 && (long)terms * std::min(nvec, 4) * ((blocks + sms - 1) / sms) <= 250;
}

pg_status hx_mixed(const pg_grid* g, const double* v, const double* x, double* y, int nvec, cudaStream_t st,
                   bool check, bool unit);

pg_status hx(const pg_grid* g, const double* v, const double* x, double* y, int nvec, int precision,
             cudaStream_t st, bool unit, bool in_order) {
  PG_ARG(g && v && nvec >= 0, "pg_hx: bad arguments");
  if (nvec == 0) return PG_OK;  // an empty block may come with null X and Y
  PG_ARG(x && y, "pg_hx: null X or Y");
  PG_ARG(x != y, "pg_hx: X and Y must not alias");
  if (precision == PG_MIXED) return hx_mixed(g, v, x, y, nvec, st, false, unit);
  PG_ARG(precision == PG_FP64, "pg_hx: unknown precision %d", precision);
  // !t_sliced: the slices would round T's small entries further than the chain
  // rounds (a sine-DVR axis above about 750 points)
  if (in_order || !g->t_sliced || chain_is_shorter(g, nvec)) {
    by_vectors(g->N, nvec, [&](auto rest, dim3 blocks, int four) {
      k_hx_fp64<rest.value><<<blocks, 256, 0, st>>>(g->n[0], g->n[1], g->n[2], g->t_dev[0].p, g->t_dev[1].p,
                                                    g->t_dev[2].p, v, x, y, four);
    });
    return check_launch("k_hx_fp64");
  }
  PG_TRY(slice_axis(g, 2, g->t_sl[2], g->t_dev[2].p, v, x, y, nvec, 2, st));
  PG_TRY(slice_axis(g, 1, g->t_sl[1], g->t_dev[1].p, nullptr, x, y, nvec, 1, st));
  return slice_axis(g, 0, g->t_sl[0], g->t_dev[0].p, nullptr, x, y, nvec, 1, st);
}

}  // namespace pg

extern "C" pg_status pg_hx(const pg_grid* g, const double* v, const double* x, double* y, int nvec, int precision,
                           void* stream) {
  cudaStream_t st = pg::as_stream(stream);
  PG_TRY(pg::hx(g, v, x, y, nvec, precision, st));
  // the FP64 kernels finish their outputs whatever their waits do
  return precision == PG_MIXED ? pg::check_tc_error(g, st) : PG_OK;
}

extern "C" pg_status pg_hx_async(const pg_grid* g, const double* v, const double* x, double* y, int nvec,
                                 int precision, void* stream) {
  return pg::hx(g, v, x, y, nvec, precision, pg::as_stream(stream));
}

extern "C" pg_status pg_grid_check(const pg_grid* g, void* stream) {
  PG_ARG(g, "pg_grid_check: null grid");
  cudaStream_t st = pg::as_stream(stream);
  const pg_status s = pg::check_tc_error(g, st);
  if (s == PG_DEVICE_TIMEOUT) *g->tc_err.h = 0;
  return s;
}
