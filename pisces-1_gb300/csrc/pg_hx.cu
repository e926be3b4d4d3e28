// Y = H X on the 3-D sine-DVR grid, FP64 form.
//
// H = diag(V) + Tx (+) Ty (+) Tz: for every grid point and vector,
//   y = v x + sum_b Tx[i,b] x[b,j,k] + sum_b Ty[j,b] x[i,b,k] + sum_b Tz[k,b] x[i,j,b]
// (src/mtx.cpp:35-104 applies the same operator line by line with dspmv).
// Three axis contractions from exact slices on the tensor cores
// (pg_slice.cu): z with V X, then y and x added to Y.
#include "pg_slice.cuh"

namespace pg {

pg_status tc_axis(const pg_grid* g, int a, const float* Ahi, const float* Alo, const double* v, const double* x,
                  double* y, int nvec, int mode, cudaStream_t st);

pg_status axis_apply(const pg_grid* g, int axis, const SliceMat& S, const double* A64, const float* Ahi,
                     const float* Alo, const double* x, double* y, int nvec, int mode, int precision,
                     cudaStream_t st) {
  PG_ARG(g && x && y && x != y && axis >= 0 && axis < 3 && (mode == 0 || mode == 1), "axis_apply: bad arguments");
  if (precision == PG_MIXED) return tc_axis(g, axis, Ahi, Alo, nullptr, x, y, nvec, mode, st);
  return slice_axis(g, axis, S, A64, nullptr, x, y, nvec, mode, st);
}

pg_status hx_mixed(const pg_grid* g, const double* v, const double* x, double* y, int nvec, cudaStream_t st,
                   bool check, bool unit);

pg_status hx(const pg_grid* g, const double* v, const double* x, double* y, int nvec, int precision,
             cudaStream_t st, bool unit) {
  PG_ARG(g && v && nvec >= 0, "pg_hx: bad arguments");
  if (nvec == 0) return PG_OK;  // an empty block may come with null X and Y
  PG_ARG(x && y, "pg_hx: null X or Y");
  PG_ARG(x != y, "pg_hx: X and Y must not alias");
  if (precision == PG_MIXED) return hx_mixed(g, v, x, y, nvec, st, false, unit);
  PG_ARG(precision == PG_FP64, "pg_hx: unknown precision %d", precision);
  PG_TRY(slice_axis(g, 2, g->t_sl[2], g->t_dev[2].p, v, x, y, nvec, 2, st));
  PG_TRY(slice_axis(g, 1, g->t_sl[1], g->t_dev[1].p, nullptr, x, y, nvec, 1, st));
  return slice_axis(g, 0, g->t_sl[0], g->t_dev[0].p, nullptr, x, y, nvec, 1, st);
}

}  // namespace pg

extern "C" pg_status pg_hx(const pg_grid* g, const double* v, const double* x, double* y, int nvec, int precision,
                           void* stream) {
  cudaStream_t st = pg::as_stream(stream);
  PG_TRY(pg::hx(g, v, x, y, nvec, precision, st));
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
  if (s == PG_DEVICE_TIMEOUT) PG_CUDA_TRY(cudaMemsetAsync(g->tc_err.p, 0, sizeof(int), st));
  return s;
}
