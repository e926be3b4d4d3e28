// Deterministic skinny FP64 kernels for the Davidson subspace (see pg_linalg.cuh).
//
// Blocks write partial sums (one per output); the partials of each output are
// reduced by one warp in a fixed order, by a second launch (Gram products) or
// by the block that an arrival counter finds to be the last (norms, k_ritz_df,
// and the coefficients of a Gram-Schmidt pass after its second launch).  Which
// block that is does not change the sums: no dependence on scheduling.
#include <algorithm>
#include <cstdint>
#include <mutex>

#include "pg_linalg.cuh"

namespace pg {

namespace {

constexpr int kT = 256;
constexpr int kTP = 32;     // points per shared-memory tile in k_gram
constexpr int kBatch = 8;   // global loads a thread keeps in flight
constexpr int kStreamBlocks = 4 * kRedBlocks;  // blocks of the streaming kernels (about one point per thread)

long chunk_for(long N, int blocks, int align) {
  long c = (N + blocks - 1) / blocks;
  c = (c + align - 1) / align * align;
  return c > 0 ? c : align;
}

// out[o] = sum_b partial[b*no + o] over nb partial rows; one warp per output,
// lanes stride over the rows, then a fixed shuffle tree.  inv_sqrt_out: also
// store 1/sqrt(out[o]) at out[no + o] (used to normalise vectors on device).
__device__ __forceinline__ void reduce_rows(const double* __restrict__ partial, int nb, int no, double* out,
                                            int sqrt_mode) {
  const int warp = (blockIdx.x * kT + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= no) return;
  double s = 0;
  for (int b0 = 0; b0 < nb; b0 += 8 * 32) {  // eight independent loads in flight per lane
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int b = b0 + u * 32 + lane;
      v[u] = b < nb ? partial[(long)b * no + warp] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b0 + u * 32 < nb) s += v[u];  // zero rows left out: the same sum
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) {
    out[warp] = s;
    if (sqrt_mode) out[no + warp] = 1.0 / sqrt(s);
  }
}
__global__ void __launch_bounds__(kT) k_reduce_partials(const double* __restrict__ partial, int nb, int no,
                                                        double* __restrict__ out, int sqrt_mode,
                                                        const int* __restrict__ skip) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  reduce_rows(partial, nb, no, out, sqrt_mode);
}

// Coefficients of one block Gram-Schmidt pass with the Pythagorean Gram (the
// BCGS-PIP form): the corrections R (k vectors) sit right after the nb basis
// vectors of B, and G holds the Gram products of [B R] against R,
// G[a*k + j] = [B R]_a . R_j, so the first nb rows are C = B^T R and the last
// k rows are R^T R.  With B orthonormal, (R - B C)^T (R - B C) = R^T R - C^T C,
// whose Cholesky factor L gives U = L^-T; the pass is then one combine over
// [B R] with coef[a*k + j] = -(C U)[a][j] for a < nb and U[a-nb][j] below.
// A pivot is floored at 1e-24 of that vector's R^T R diagonal: where the
// subtraction cancels (R almost inside span(B)) the pass yields scaled
// rounding noise, mostly orthogonal to B, which the second pass (no
// cancellation left) projects and normalises.  k <= 16, nb <= 128.
//
// skip_out (first pass): 1 when every squared pivot L_jj^2 keeps at least
// kPipKeep of that correction's squared norm R_j^T R_j, else 0.  Pivot j is
// what remains of R_j after removing span(B) and the corrections before it;
// with ratios that large the pass's rounding leaves the block orthonormal to
// about u / kPipKeep (u: the unit roundoff of the products, 2^-53 in FP64,
// about 2^-48 in double-float), and the second pass, which would change the
// vectors only by that much, is skipped.
constexpr double kPipKeep = 1e-3;
__device__ __forceinline__ void pip_coef(const double* G, int nb, int k, double* __restrict__ coef,
                                         int* __restrict__ skip_out) {
  __shared__ double Cs[128][kMaxCombine];
  __shared__ double L[kMaxCombine][kMaxCombine + 1];
  __shared__ double U[kMaxCombine][kMaxCombine + 1];
  __shared__ int Keep[kMaxCombine];
  __shared__ double Rd[kMaxCombine];  // R_j^T R_j
  const int tid = threadIdx.x;
  for (int e = tid; e < nb * k; e += blockDim.x) Cs[e / k][e % k] = __ldcg(G + e);
  __syncthreads();
  if (tid < k * k) {  // R^T R - C^T C, each entry summed in basis order
    const int i = tid / k, j = tid % k;
    double s = __ldcg(G + (long)(nb + i) * k + j);
    if (i == j) Rd[j] = s;
    for (int a = 0; a < nb; ++a) s -= Cs[a][i] * Cs[a][j];
    L[i][j] = s;
  }
  __syncthreads();
  if (tid < 32) {
    const int lane = tid;
    for (int j = 0; j < k; ++j) {
      if (lane == 0) {
        double s = L[j][j];
        for (int p = 0; p < j; ++p) s -= L[j][p] * L[j][p];
        const double floor = 1e-24 * Rd[j];
        const double piv = s > floor ? s : (floor > 1e-300 ? floor : 1e-300);
        L[j][j] = sqrt(piv);
        Keep[j] = piv >= kPipKeep * Rd[j];
      }
      __syncwarp();
      if (lane > j && lane < k) {
        double t = L[lane][j];
        for (int p = 0; p < j; ++p) t -= L[lane][p] * L[j][p];
        L[lane][j] = t / L[j][j];
      }
      __syncwarp();
    }
    if (skip_out && lane == 0) {
      int all = 1;
      for (int j = 0; j < k; ++j) all &= Keep[j];
      *skip_out = all;
    }
    if (lane < k) {  // U = L^-T, column c on lane c (upper triangular)
      const int c = lane;
      for (int i = k - 1; i >= 0; --i) {
        double s = i == c ? 1.0 : 0.0;
        for (int p = i + 1; p < k; ++p) s -= L[p][i] * U[p][c];
        U[i][c] = i > c ? 0.0 : s / L[i][i];
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < (nb + k) * k; e += blockDim.x) {
    const int a = e / k, j = e % k;
    double s;
    if (a < nb) {
      s = 0.0;
      for (int i = 0; i <= j; ++i) s -= Cs[a][i] * U[i][j];
    } else {
      s = U[a - nb][j];
    }
    coef[e] = s;
  }
}

// k_reduce_partials followed by pip_coef in the block that finishes last: one
// launch between a pass's Gram product and its combine.
__global__ void __launch_bounds__(kT) k_reduce_pip(const double* __restrict__ partial, int nb, int no, double* out,
                                                   const int* __restrict__ skip, const PipPass pass,
                                                   unsigned* counter) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  reduce_rows(partial, nb, no, out, 0);
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x == 0) *counter = 0u;
  pip_coef(out, pass.nb, pass.k, pass.coef, pass.skip_out);
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

// Gram partials in FP64.  Bound by the FP64 pipe: 36 operations per output and
// kTP points (4 chains of 8 multiply-adds, which are the order of the sums),
// 64 to 76 cycles each per warp and scheduler.  T tiles of kTP points are
// resident at a time, and the warps take units of (32 outputs, tile) in turn,
// so that all four schedulers have the same work: with a thread per output
// and one tile at a time, 40 x 4 outputs kept 5 warps of 8 busy (two of them
// on one scheduler) and 20 x 1 only one.  The tiles' sums meet in shared
// memory and are added in the tiles' order.  The next T tiles are copied
// meanwhile.
// Over 262144 points, us: 8 x 1 71 -> 29, 20 x 1 72 -> 32, 40 x 4 120 -> 100,
// 56 x 8 276 -> 254, 120 x 16 1064 -> 1017.
__global__ void __launch_bounds__(kT, 2) k_gram(long N, long chunk, const double* __restrict__ P, int na,
                                                const double* __restrict__ Q, int nb, int logT,
                                                double* __restrict__ partial, const int* __restrict__ skip) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  extern __shared__ double sm[];
  const int rows = na + nb, no = na * nb;
  const int W = kTP << logT, pitch = W + 1;
  double* sums = sm + (size_t)2 * rows * pitch;  // [tile][output]
  double acc[kMaxGramOut / kT];
#pragma unroll
  for (int s = 0; s < kMaxGramOut / kT; ++s) acc[s] = 0;
  const long g_begin = blockIdx.x * chunk;
  const long g_end = g_begin + chunk < N ? g_begin + chunk : N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (no + 31) >> 5;
  auto issue = [&](long g0, int buf) {  // rows 0 .. na-1 of P, then those of Q
    double* dst = sm + (size_t)buf * rows * pitch;
    const int cnt = g_end - g0 < W ? (int)(g_end - g0) : W;
    for (int e = threadIdx.x; e < rows * W; e += kT) {
      const int row = e >> (5 + logT), p = e & (W - 1);
      const double* src = (row < na ? P + (long)row * N : Q + (long)(row - na) * N) + g0;
      const unsigned sa = (unsigned)__cvta_generic_to_shared(dst + row * pitch + p);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(src + (p < cnt ? p : 0)),
                   "r"(p < cnt ? 8 : 0)
                   : "memory");
    }
  };
  if (g_begin < g_end) issue(g_begin, 0);
  cp_async_commit();
  int buf = 0;
  for (long g0 = g_begin; g0 < g_end; g0 += W, buf ^= 1) {
    if (g0 + W < g_end) issue(g0 + W, buf ^ 1);
    cp_async_commit();
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // these tiles have landed; the sums before have been read
    const int nt = g_end - g0 < W ? (int)((g_end - g0 + kTP - 1) / kTP) : 1 << logT;
    const double* Ps = sm + (size_t)buf * rows * pitch;
    const double* Qs = Ps + na * pitch;
    for (int u = warp; u < groups * nt; u += kT / 32) {
      const int tile = u / groups, o = (u - tile * groups) * 32 + lane;
      if (o < no) {
        const double* pa = Ps + (o / nb) * pitch + tile * kTP;
        const double* qb = Qs + (o % nb) * pitch + tile * kTP;
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0;  // four chains hide the DFMA latency
#pragma unroll
        for (int p = 0; p < kTP; p += 4) {
          a0 += pa[p] * qb[p];
          a1 += pa[p + 1] * qb[p + 1];
          a2 += pa[p + 2] * qb[p + 2];
          a3 += pa[p + 3] * qb[p + 3];
        }
        sums[tile * no + o] = (a0 + a1) + (a2 + a3);
      }
    }
    __syncthreads();  // the sums are complete, these tiles free
#pragma unroll
    for (int s = 0; s < kMaxGramOut / kT; ++s) {
      const int o = threadIdx.x + s * kT;
      if (o < no)
        for (int tile = 0; tile < nt; ++tile) acc[s] += sums[tile * no + o];
    }
  }
#pragma unroll
  for (int s = 0; s < kMaxGramOut / kT; ++s) {
    const int o = threadIdx.x + s * kT;
    if (o < no) partial[(long)blockIdx.x * no + o] = acc[s];
  }
}

// Blocks per SM asked of the compiler: left to itself it gave 7 and 8 outputs
// 99 registers (two blocks) and 15 outputs 170 (one), and one or two outputs,
// bound by loads in flight, three blocks.  884736 points, us, before / so: 40 x 1
// 84.5 / 69.2, 64 x 1 129 / 107, 120 x 1 232 / 194; 262144 points: 40 x 2
// 44.6 / 39.9, 40 x 7 151 / 131, 40 x 8 171 / 149, 120 x 2 127 / 113.
template <int NR>
__global__ void __launch_bounds__(kT, NR <= 2 ? 4 : (NR <= 8 ? 3 : 2)) k_combine(long N, long chunk, const double* P, const double* P2, int na,
                                                const double* __restrict__ C, int ca, int cr, double cscale,
                                                const double* X,
                                                const double* __restrict__ alpha, int inv_sqrt, double* Y, double* Y2,
                                                int nr, double* __restrict__ partial, double* sq_out, unsigned* counter,
                                                const int* __restrict__ skip) {
  // no early release: blocks of the next kernel that take the free places of
  // some SMs would leave it uneven (back to back 96 x 4 over 110592 points,
  // on the FP64 pipe: 79 us, 100 with a release here)
  pdl_wait();
  if (skip && *skip) return;
  if (blockIdx.y) {  // the second product of combine_pair
    P = P2;
    Y = Y2;
    partial = nullptr;
  }
  extern __shared__ double sm[];
  double* Cs = sm;                 // na x nr
  __shared__ double al[NR];
  __shared__ double red[kT / 32][NR];
  for (int e = threadIdx.x; e < na * nr; e += kT) Cs[e] = cscale * C[(long)(e / nr) * ca + (long)(e % nr) * cr];
  if (threadIdx.x < nr) {
    double a = 0;
    if (alpha) a = inv_sqrt ? 1.0 / sqrt(alpha[threadIdx.x]) : alpha[threadIdx.x];
    al[threadIdx.x] = a;
  }
  __syncthreads();
  double sacc[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) sacc[r] = 0;
  const long g_begin = blockIdx.x * chunk;
  const long g_end = g_begin + chunk < N ? g_begin + chunk : N;
  for (long g = g_begin + threadIdx.x; g < g_end; g += kT) {
    double acc[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = (r < nr && X && alpha) ? al[r] * X[(long)r * N + g] : 0.0;
    // eight independent loads in flight before they are consumed
    for (int a0 = 0; a0 < na; a0 += kBatch) {
      double pv[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) pv[u] = a0 + u < na ? P[(long)(a0 + u) * N + g] : 0.0;
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (a0 + u >= na) break;
        const double* c = Cs + (a0 + u) * nr;
#pragma unroll
        for (int r = 0; r < NR; ++r)
          if (r < nr) acc[r] += pv[u] * c[r];
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < nr) {
        Y[(long)r * N + g] = acc[r];
        sacc[r] += acc[r] * acc[r];
      }
  }
  if (!partial) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    double v = sacc[r];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp][r] = v;
  }
  __syncthreads();
  if (threadIdx.x < nr) {
    double s = 0;
    for (int w = 0; w < kT / 32; ++w) s += red[w][threadIdx.x];
    partial[(long)blockIdx.x * nr + threadIdx.x] = s;
  }
  reduce_in_last_block(partial, nr, sq_out, 1, counter);
}

// ------------------------------------------------------------------------
// Double-float (two FP32 numbers, hi + lo) arithmetic for the mixed form's
// subspace products.  The FP32 pipe of this part retires ~67 TFLOP/s against
// ~1 TFLOP/s for FP64; a double-float multiply-accumulate costs ~11 FP32
// operations and keeps ~48 significant bits (Dekker 1971, Knuth TwoSum).

// x = hi + lo to about 2^-48 |x| (hi takes the top 24 mantissa bits; the
// remaining 29 are rounded to the 24 of lo), with integer operations only
// (the FP64 pipe is not touched).  |x| < 2^-126 flushes to zero.  |x| >=
// 2^128 and Inf give hi = +-Inf, NaN gives hi = NaN (lo = 0), so a
// non-finite input reaches the products and norms built from the pair.
__device__ __forceinline__ void df_split(double x, float& hi, float& lo) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const uint32_t h = (uint32_t)(b >> 32);
  const int e = (int)((h >> 20) & 0x7ff);
  const int ef = e - 1023 + 127;
  if (ef <= 0) {
    hi = 0.f;
    lo = 0.f;
    return;
  }
  const uint32_t sign = h & 0x80000000u;
  if (ef >= 255) {
    const bool nan = e == 0x7ff && (b & 0xfffffffffffffull) != 0;
    hi = __uint_as_float(nan ? 0x7fc00000u : (sign | 0x7f800000u));
    lo = 0.f;
    return;
  }
  hi = __uint_as_float(sign | ((uint32_t)ef << 23) | (uint32_t)((b >> 29) & 0x7fffffu));
  const uint32_t rem = (uint32_t)(b & 0x1fffffffu);  // the 29 mantissa bits below hi
  const int el = e - 1075 + 127;                      // exponent of one unit of rem
  float scale = el > 0 ? __uint_as_float((uint32_t)el << 23) : 0.f;
  const float l = __uint2float_rn(rem) * scale;
  lo = sign ? -l : l;
}

// df_split of N values.  Where all of them lie in [2^-74, 2^128) the bits of
// hi only move by three places, and the scale of lo follows from them: about
// 12 instructions a value, half of the general form's (884736 points: Gram
// 56x8 293 -> 273 us, combine 234 -> 216); same results.
template <int N>
__device__ __forceinline__ void df_split_n(const double (&x)[N], float (&hi)[N], float (&lo)[N]) {
  bool fast = true;
#pragma unroll
  for (int i = 0; i < N; ++i)
    fast &= ((uint32_t)__double2hiint(x[i]) & 0x7fffffffu) - (949u << 20) < (202u << 20);
  if (fast) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint32_t h = (uint32_t)__double2hiint(x[i]), l = (uint32_t)__double2loint(x[i]);
      const uint32_t f = __funnelshift_l(l, h, 3) - (896u << 23), sign = h & 0x80000000u;
      hi[i] = __uint_as_float(f | sign);
      lo[i] = __uint2float_rn(l & 0x1fffffffu) * __uint_as_float(((f & 0x7f800000u) - (52u << 23)) | sign);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) df_split(x[i], hi[i], lo[i]);
  }
}

// (sh, sl) += a * b with a = (ah, al), b = (bh, bl)
__device__ __forceinline__ void df_fma(float& sh, float& sl, float ah, float al, float bh, float bl) {
  const float p = ah * bh;
  float e = fmaf(ah, bh, -p);
  e = fmaf(ah, bl, e);
  e = fmaf(al, bh, e);
  const float t = sh + p;
  const float bp = t - sh;
  const float err = (sh - (t - bp)) + (p - bp);
  sl += err + e;
  sh = t;
}

// Two FP32 numbers in one register pair, for the packed FP32 instructions: the
// same roundings at the same rate, but half the issue slots, which leaves
// slots for the integer work beside them.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void f2_unpack(f32x2 d, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(d));
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// a - b (b times -1 is exact, so one rounding)
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) { return f2_fma(b, 0xbf800000bf800000ull, a); }

// df_fma for two sums at once: the one value a = (ah, al), given as the pairs
// (ah, ah), (-ah, -ah) and (-al, -al), times two coefficients.  The error of
// the product is kept negated; the roundings are df_fma's.
__device__ __forceinline__ void df_fma2(f32x2& sh, f32x2& sl, f32x2 ah, f32x2 nah, f32x2 nal, f32x2 bh, f32x2 bl) {
  const f32x2 p = f2_mul(ah, bh);
  f32x2 e = f2_fma(nah, bh, p);
  e = f2_fma(nah, bl, e);
  e = f2_fma(nal, bh, e);
  const f32x2 t = f2_add(sh, p);
  const f32x2 bp = f2_sub(t, sh);
  const f32x2 err = f2_add(f2_sub(sh, f2_sub(t, bp)), f2_sub(p, bp));
  sl = f2_add(sl, f2_sub(err, e));
  sh = t;
}

// FP32 -> FP64 with integer operations (exact for normal numbers and zero;
// FP32 subnormals flush to a signed zero; Inf and NaN are kept): keeps the
// conversion off the FP64 pipe, which retires about two operations per SM
// per clock on this part.
__device__ __forceinline__ double f32_to_f64_int(float v) {
  const uint32_t u = __float_as_uint(v);
  const uint32_t sign = u & 0x80000000u, e = (u >> 23) & 0xffu, mt = u & 0x7fffffu;
  uint32_t hi = sign | ((e + 896u) << 20) | (mt >> 3);
  uint32_t lo = mt << 29;
  hi = e == 0 ? sign : hi;
  lo = e == 0 ? 0u : lo;
  hi = e == 255 ? (sign | 0x7ff00000u | (mt >> 3) | (mt ? 0x80000u : 0u)) : hi;
  lo = e == 255 ? 0u : lo;
  return __hiloint2double((int)hi, (int)lo);
}

// (double)h + (double)l rounded to nearest, with FP32 and integer operations:
// an FP64 conversion or addition costs 64 to 76 cycles a warp and scheduler
// here.  s = h + l in FP32 and its error e (two-sum, exact); then e, in units
// of the result's last place, is rounded to an integer and added to s's bits.
// Not for sums outside [2^-75, 2^127], or where the addition crosses below a
// power of two (its last place is then half as large): by FP64, as the caller
// asks for FP32 subnormals (kFlush: zero, as f32_to_f64_int).
template <bool kFlush>
__device__ __noinline__ double df_join_slow(float h, float l) {
  if (kFlush) return f32_to_f64_int(h) + f32_to_f64_int(l);
  return (double)h + (double)l;
}
template <bool kFlush>
__device__ __forceinline__ double df_join(float h, float l) {
  const float s = h + l;
  const float bp = s - h;
  const float e = (h - (s - bp)) + (l - bp);
  const uint32_t u = __float_as_uint(s);
  const uint32_t ex = u & 0x7f800000u;
  // e / 2^(exponent of s - 52), with the sign of s: at most 2^28 in magnitude
  const float v = e * __uint_as_float((0x99000000u - ex) ^ (u & 0x80000000u));
  if (ex - (52u << 23) > (202u << 23) || ((u & 0x7fffffu) == 0 && v < 0.f)) return df_join_slow<kFlush>(h, l);
  const long long r = (long long)(((unsigned long long)((u & 0x7fffffffu) >> 3) + (896ull << 20)) << 32 | (u << 29)) +
                      __float2int_rn(v);
  return __longlong_as_double(r | (long long)((unsigned long long)(u & 0x80000000u) << 32));
}

// Sums K values (a power of two) over the lanes as steps of 16, 8, .. to kLast
// of v[lane] + v[lane + step] would, several values to a register as lanes
// become free: value k ends in lane k (32 / K) for K <= 32 / kLast, else value
// k in v[k % (K kLast / 32)] of lane kLast (k / (K kLast / 32)).
template <int K, int kLast, typename T>
__device__ __forceinline__ void packed_sums(T (&v)[K], int lane) {
  int n = K;
#pragma unroll
  for (int o = 16; o >= kLast; o >>= 1) {
    if (n > 1) {
#pragma unroll
      for (int i = 0; i < K / 2; ++i) {
        if (i < n / 2) {
          const bool up = lane & o;
          const T keep = up ? v[i + n / 2] : v[i], send = up ? v[i] : v[i + n / 2];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      n >>= 1;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
}

// Gram partials in double-float, written as double (hi + lo): same contract
// as k_gram.  A thread owns a kGA x kGB block of outputs (kGA rows of P
// against kGB rows of Q) for one slice of the points of each tile, so every
// point value it reads from shared memory feeds kGB or kGA products.  Tiles of
// tp points of all na + nb rows stream through kGStages shared-memory stages
// with cp.async (each thread converts the doubles it copied to (hi, lo) pairs
// in place once they land), keeping two tiles in flight behind the one being
// multiplied.  At the end the slices of each output block are summed in a
// fixed order.
// Bound by the FP32 pipe in the multiply loop (12 operations per output and
// point) and by the issue slots of copies and conversions beside it.  Those
// had a warp to a row (36 point pairs: two rounds for 36 of 64 lanes), and the
// ends 48 FP64 operations a thread; without them, us over 884736 points: 16 x 4
// 83 -> 67, 40 x 4 188 -> 131, 56 x 8 404 -> 273, 96 x 4 563 -> 306.
constexpr int kGA = 4, kGB = 4, kGStages = 3;
constexpr int kGramSmemMax = 112 * 1024;

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_stages() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kGStages - 2) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Tile geometry of k_gram_df: S slices per output block, tiles of tp = 2 S m
// points so that every slice takes exactly m point pairs of every tile (no
// lanes idle in the multiply loop), as many pairs as kGStages stages of
// (na + nb) rows allow in kGramSmemMax.
struct GramGeom {
  int ablk, nblk, S, m, tp;
  size_t smem;
};

inline GramGeom gram_geometry(int na, int nb) {
  GramGeom g;
  g.ablk = (na + kGA - 1) / kGA;
  g.nblk = g.ablk * ((nb + kGB - 1) / kGB);
  g.S = g.nblk <= kT ? kT / g.nblk : 1;
  const size_t per_pair_set = (size_t)kGStages * (na + nb) * 2 * g.S * 8;  // stage bytes per unit of m
  g.m = (int)std::max<size_t>(1, std::min<size_t>(8, kGramSmemMax / per_pair_set));
  g.tp = 2 * g.S * g.m;
  g.smem = std::max((size_t)g.m * per_pair_set, (size_t)g.S * g.nblk * kGA * kGB * 8);
  return g;
}

// kPair: N even and P, Q 16-byte aligned, so that consecutive point pairs
// are copied with 16-byte cp.async and converted two at a time.
// split_p / split_q: the rows of P / Q are already double-float "twins" (a
// float2 (hi, lo) per point, the layout the staging converts to), copied as
// they are and not converted again.
template <bool kPair>
__global__ void __launch_bounds__(kT, 2) k_gram_df(long N, long chunk, const double* __restrict__ P, int na,
                                                   const double* __restrict__ Q, int nb, int tp, int m, int S,
                                                   int ablk, int nblk, int split_p, int split_q,
                                                   double* __restrict__ partial, const int* __restrict__ skip) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char gsm[];
  const int rows = na + nb;
  const int hp = tp >> 1;  // point pairs per tile row
  const int stage_elems = rows * tp;
  double* stage0 = reinterpret_cast<double*>(gsm);
  const long g_begin = blockIdx.x * chunk;
  const long g_end = g_begin + chunk < N ? g_begin + chunk : N;
  const int ntiles = g_end > g_begin ? (int)((g_end - g_begin + tp - 1) / tp) : 0;
  const int tid = threadIdx.x;
  const int blk = tid / S, slice = tid - blk * S;
  const bool active = blk < nblk;
  const int a0 = (blk % ablk) * kGA, b0 = (blk / ablk) * kGB;
  int ra[kGA], rb[kGB];  // stage rows of this thread's outputs (clamped; extra outputs are discarded)
#pragma unroll
  for (int i = 0; i < kGA; ++i) ra[i] = (a0 + i < na ? a0 + i : na - 1) * hp;
#pragma unroll
  for (int j = 0; j < kGB; ++j) rb[j] = (na + (b0 + j < nb ? b0 + j : nb - 1)) * hp;
  float sh[kGA][kGB], sl[kGA][kGB];
#pragma unroll
  for (int i = 0; i < kGA; ++i)
#pragma unroll
    for (int j = 0; j < kGB; ++j) sh[i][j] = sl[i][j] = 0.f;

  // staging: the threads take the tile's point pairs (points) row by row, kT
  // at a time, so that no lane idles where a row's are not a multiple of 32;
  // addresses count up
  const int per = kPair ? hp : tp, total = rows * per;
  constexpr int kStep = kPair ? 2 : 1;
  const int row0 = tid / per, q0 = tid - row0 * per, drow = kT / per, dq = kT - drow * per;
  const long jump = (long)drow * N + kStep * dq, wrap = N - (long)kStep * per;
  const double* first = (row0 < na ? P + (long)row0 * N : Q + (long)(row0 - na) * N) + g_begin + kStep * q0;
  const long to_q = Q - (P + (long)na * N);  // from where row na of P would be to row 0 of Q
  auto issue = [&](int tile) {
    double* d = stage0 + (size_t)(tile % kGStages) * stage_elems + kStep * tid;
    const long g0 = (long)tile * tp;
    const int cnt = g_end - g_begin - g0 < tp ? (int)(g_end - g_begin - g0) : tp;
    const double* src = first + g0;
    int row = row0, p = kStep * q0;
    for (int e = tid; e < total; e += kT, d += kStep * kT) {
      if (kPair) {
        if (p + 1 < cnt) {
          cp_async16(d, src);
        } else if (p < cnt) {
          cp_async8(d, src);
          d[1] = 0.0;
        } else {
          d[0] = 0.0;
          d[1] = 0.0;
        }
      } else {
        if (p < cnt) cp_async8(d, src);
        else d[0] = 0.0;
      }
      const bool in_p = row < na;
      row += drow;
      p += kStep * dq;
      src += jump;
      if (p >= kStep * per) p -= kStep * per, src += wrap, ++row;
      if (in_p && row >= na) src += to_q;
    }
  };
  for (int t = 0; t < kGStages - 1; ++t) {
    if (t < ntiles) issue(t);
    cp_async_commit();
  }
  for (int it = 0; it < ntiles; ++it) {
    cp_async_wait_stages();  // this thread's copies of tile `it` have landed
    double* cur = stage0 + (size_t)(it % kGStages) * stage_elems;
    // convert the points this thread copied, in place, to (hi, lo) pairs
    // (a twin's rows already are)
    const int conv0 = split_p ? na * per : 0, conv1 = split_q ? na * per : total;
    for (int e = tid; e < conv1; e += kT) {
      if (e < conv0) continue;
      double* d = cur + (size_t)kStep * e;
      if (kPair) {
        const double2 d2 = *reinterpret_cast<const double2*>(d);
        const double x[2] = {d2.x, d2.y};
        float h[2], l[2];
        df_split_n(x, h, l);
        *reinterpret_cast<float4*>(d) = make_float4(h[0], l[0], h[1], l[1]);
      } else {
        float h, l;
        df_split(d[0], h, l);
        *reinterpret_cast<float2*>(d) = make_float2(h, l);
      }
    }
    __syncthreads();  // tile `it` converted; everyone is done with tile it-1
    if (it + kGStages - 1 < ntiles) issue(it + kGStages - 1);
    cp_async_commit();
    if (active) {
      // m point pairs per slice (one 16-byte load per row each; zero points
      // past the tile's end add nothing)
      const float4* cur4 = reinterpret_cast<const float4*>(cur);
      for (int u = 0; u < m; ++u) {
        const int q = slice + u * S;
        float4 y[kGB];
#pragma unroll
        for (int j = 0; j < kGB; ++j) y[j] = cur4[rb[j] + q];
#pragma unroll
        for (int i = 0; i < kGA; ++i) {
          const float4 x = cur4[ra[i] + q];
#pragma unroll
          for (int j = 0; j < kGB; ++j) {
            df_fma(sh[i][j], sl[i][j], x.x, x.y, y[j].x, y[j].y);
            df_fma(sh[i][j], sl[i][j], x.z, x.w, y[j].z, y[j].w);
          }
        }
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();
  // slices -> one partial per output, summed in slice order
  double* red = reinterpret_cast<double*>(gsm);
  if (active) {
#pragma unroll
    for (int i = 0; i < kGA; ++i)
#pragma unroll
      for (int j = 0; j < kGB; ++j)
        red[((size_t)slice * nblk + blk) * (kGA * kGB) + i * kGB + j] = df_join<false>(sh[i][j], sl[i][j]);
  }
  __syncthreads();
  const int no = na * nb;
  for (int o = tid; o < no; o += kT) {
    const int a = o / nb, b = o - (o / nb) * nb;
    const int bo = a / kGA + (b / kGB) * ablk;
    const int k = (a % kGA) * kGB + (b % kGB);
    double acc = 0;
    for (int q = 0; q < S; ++q) acc += red[((size_t)q * nblk + bo) * (kGA * kGB) + k];
    partial[(long)blockIdx.x * no + o] = acc;
  }
}

// The coefficients of up to NR outputs as double-float: [row][pair of outputs]
// (hi, hi, lo, lo), zero past nr; for one output [row] (hi, lo).
template <int NR, typename Get>
__device__ __forceinline__ void load_coefs(float* Cs, int na, int nr, const Get& get) {
  for (int e = threadIdx.x; e < na * NR; e += kT) {
    const int a = e / NR, r = e % NR;
    float h = 0.f, l = 0.f;
    if (r < nr) df_split(get(a, r), h, l);
    float* c = NR == 1 ? Cs + 2 * a : Cs + 4 * (a * (NR / 2) + r / 2) + r % 2;
    c[0] = h;
    c[NR == 1 ? 1 : 2] = l;
  }
}
template <int NR>
constexpr size_t coef_bytes(int na) { return sizeof(float) * 2 * (size_t)(na > 0 ? na : 1) * NR; }

// NR double-float sums of one point, two to a register pair.
template <int NR>
struct DfSums {
  f32x2 h[NR / 2], l[NR / 2];
  __device__ __forceinline__ DfSums(const float (&sh)[NR], const float (&sl)[NR]) {
#pragma unroll
    for (int j = 0; j < NR / 2; ++j) h[j] = f2_pack(sh[2 * j], sh[2 * j + 1]), l[j] = f2_pack(sl[2 * j], sl[2 * j + 1]);
  }
  // += (ph, pl) times row a of the coefficients
  __device__ __forceinline__ void add(float ph, float pl, const float* Cs, int a) {
    const f32x2 ah = f2_pack(ph, ph), nah = f2_pack(-ph, -ph), nal = f2_pack(-pl, -pl);
    const ulonglong2* c = reinterpret_cast<const ulonglong2*>(Cs) + a * (NR / 2);
#pragma unroll
    for (int j = 0; j < NR / 2; ++j) {
      const ulonglong2 b = c[j];
      df_fma2(h[j], l[j], ah, nah, nal, b.x, b.y);
    }
  }
  __device__ __forceinline__ void get(float (&sh)[NR], float (&sl)[NR]) const {
#pragma unroll
    for (int j = 0; j < NR / 2; ++j) {
      f2_unpack(h[j], sh[2 * j], sh[2 * j + 1]);
      f2_unpack(l[j], sl[2 * j], sl[2 * j + 1]);
    }
  }
};
template <>
struct DfSums<1> {
  float h, l;
  __device__ __forceinline__ DfSums(const float (&sh)[1], const float (&sl)[1]) : h(sh[0]), l(sl[0]) {}
  __device__ __forceinline__ void add(float ph, float pl, const float* Cs, int a) {
    const float2 c = reinterpret_cast<const float2*>(Cs)[a];
    df_fma(h, l, ph, pl, c.x, c.y);
  }
  __device__ __forceinline__ void get(float (&sh)[1], float (&sl)[1]) const { sh[0] = h, sl[0] = l; }
};

// Combine in double-float: same contract as k_combine (coefficients and
// alpha are FP64 and split once per block; Y is written as double).
// kTwinIn: the rows of P are double-float twins (float2 (hi, lo) per point)
// and are read without converting; kTwinOut: each output is also written as
// its twin to Yt.  Compile-time flags: a runtime choice inside the unrolled
// loop doubles the registers of the kernel and halves its occupancy.
// Bound by the FP32 pipe: 12 operations per output and row, two outputs to an
// instruction, whose coefficients are one 16-byte read; the pairs become FP64
// without the FP64 pipe, and the norms' FP64 sums over the lanes share
// instructions.  With a read and a branch per coefficient, and conversions
// and every sum in FP64, us over 884736 points: 40 x 4 132 -> 100, 56 x 8
// 371 -> 216, 12 x 12 173 -> 107, 120 x 16 1370 -> 766; 40 x 1 74 -> 56 (rows
// read ahead).
template <int NR, bool kTwinIn, bool kTwinOut>
__global__ void __launch_bounds__(kT, NR <= 4 ? 4 : 2) k_combine_df(long N, long chunk, const double* P, int na,
                                                   const double* __restrict__ C, int ca, int cr, double cscale,
                                                   const double* X, const double* __restrict__ alpha, int inv_sqrt,
                                                   double* Y, int nr, float2* Yt, double* __restrict__ partial,
                                                   double* sq_out, unsigned* counter, const int* __restrict__ skip) {
  // the next kBatch rows are on their way while these are multiplied; not with
  // 4 outputs, where four blocks per SM (64 registers) are worth more (16 x 4
  // over 884736 points: 48 us, 56 with three blocks and the rows ahead)
  constexpr bool kAhead = NR != 4;
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  extern __shared__ __align__(16) float smf[];
  float* Cs = smf;  // [row][pair]: (hi, hi, lo, lo); NR 1: [row] (hi, lo)
  constexpr int NS = NR == 6 ? 8 : (NR > 8 ? 16 : NR);  // norms: a power of two
  __shared__ float alh[NR], all[NR];
  __shared__ double red[kT / 32][NS];
  load_coefs<NR>(Cs, na, nr, [&](int a, int r) { return cscale * C[(long)a * ca + (long)r * cr]; });
  if (threadIdx.x < nr) {
    double a = 0;
    if (alpha) a = inv_sqrt ? 1.0 / sqrt(alpha[threadIdx.x]) : alpha[threadIdx.x];
    float h, l;
    df_split(a, h, l);
    alh[threadIdx.x] = h;
    all[threadIdx.x] = l;
  }
  __syncthreads();
  double sacc[NS];
#pragma unroll
  for (int r = 0; r < NS; ++r) sacc[r] = 0;
  const bool keep = X && alpha;
  const long g_begin = blockIdx.x * chunk;
  const long g_end = g_begin + chunk < N ? g_begin + chunk : N;
  for (long g = g_begin + threadIdx.x; g < g_end; g += kT) {
    float sh[NR], sl[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      sh[r] = 0.f;
      sl[r] = 0.f;
      if (r < nr && keep) {
        float xh, xl;
        df_split(X[(long)r * N + g], xh, xl);
        df_fma(sh[r], sl[r], alh[r], all[r], xh, xl);
      }
    }
    DfSums<NR> sum(sh, sl);
    const double* row = P + g;
    double pv[kBatch], nv[kBatch];
    auto rows = [&](double (&w)[kBatch], int a0) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u) w[u] = a0 + u < na ? row[(long)(a0 + u) * N] : 1.0;  // 1: not used, but splits as the rest
    };
    rows(pv, 0);
    for (int a0 = 0; a0 < na; a0 += kBatch) {
      if (kAhead) rows(nv, a0 + kBatch);
      float ph[kBatch], pl[kBatch];
      if (kTwinIn) {  // the 8 bytes are a float2 (hi, lo): hi in the low word
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          ph[u] = __int_as_float(__double2loint(pv[u]));
          pl[u] = __int_as_float(__double2hiint(pv[u]));
        }
      } else {
        df_split_n(pv, ph, pl);
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (a0 + u >= na) break;
        sum.add(ph[u], pl[u], Cs, a0 + u);
      }
      if (kAhead) {
#pragma unroll
        for (int u = 0; u < kBatch; ++u) pv[u] = nv[u];
      } else {
        rows(pv, a0 + kBatch);
      }
    }
    sum.get(sh, sl);
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < nr) {
        const double y = df_join<false>(sh[r], sl[r]);
        Y[(long)r * N + g] = y;
        // the accumulator pair is the output in double-float form already
        // (it and y = sh + sl agree to 2^-53 relative)
        if (kTwinOut) Yt[(long)r * N + g] = make_float2(sh[r], sl[r]);
        if (partial) sacc[r] += y * y;
      }
  }
  if (!partial) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  packed_sums<NS, 1>(sacc, lane);
  if (lane % (32 / NS) == 0) red[warp][lane / (32 / NS)] = sacc[0];
  __syncthreads();
  if (threadIdx.x < nr) {
    double s = 0;
    for (int w = 0; w < kT / 32; ++w) s += red[w][threadIdx.x];
    partial[(long)blockIdx.x * nr + threadIdx.x] = s;
  }
  reduce_in_last_block(partial, nr, sq_out, 1, counter);
}

// out[o] = sum of partial[b*no + o] over the nb rows, in a fixed order (k_reduce_partials)
pg_status reduce(const double* partial, int nb, int no, double* out, bool sqrt_mode, cudaStream_t st,
                 const int* skip = nullptr, const PipPass* pass = nullptr, unsigned* counter = nullptr) {
  const int blocks = (no * 32 + kT - 1) / kT;
  if (pass) {
    PG_CUDA_TRY(launch_dependent(k_reduce_pip, dim3(blocks), dim3(kT), 0, st, partial, nb, no, out, skip, *pass,
                                 counter));
    return check_launch("k_reduce_pip");
  }
  PG_CUDA_TRY(launch_dependent(k_reduce_partials, dim3(blocks), dim3(kT), 0, st, partial, nb, no, out,
                               sqrt_mode ? 1 : 0, skip));
  return check_launch("k_reduce_partials");
}

}  // namespace

pg_status RedScratch::ensure(cudaStream_t st) {
  if (!partial.p) PG_TRY(partial.alloc((size_t)kRedBlocks * kMaxGramOut));
  if (!counter.p) {
    PG_TRY(counter.alloc(1));
    PG_TRY(zero_now(counter.p, sizeof(unsigned)));
  }
  return PG_OK;
}

// Double-float twins of count doubles: t[i] = (hi, lo) of x[i] (df_split);
// with y, also y[i] = x[i] (a copy and its twin in one pass).
__global__ void __launch_bounds__(kT) k_split_twin(long count, const double* __restrict__ x, float2* __restrict__ t,
                                                   double* __restrict__ y) {
  pdl_wait();
  pdl_release();
  for (long i = blockIdx.x * (long)kT + threadIdx.x; i < count; i += (long)gridDim.x * kT) {
    const double v = x[i];
    float h, l;
    df_split(v, h, l);
    t[i] = make_float2(h, l);
    if (y) y[i] = v;
  }
}

// 16-byte copies of point pairs: every row start 16-byte aligned
inline bool pair_ok(long N, const double* P, const double* Q) {
  return N % 2 == 0 && ((uintptr_t)P % 16) == 0 && ((uintptr_t)Q % 16) == 0;
}

// Shared-memory opt-in of the Gram kernels for a launch with smem dynamic bytes,
// once per kernel and device; launches within the default (48 KB with the
// static part) do without the look at the device.
static pg_status opt_in_smem(size_t smem) {
  if (smem <= 40 * 1024) return PG_OK;
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev));
  PG_CUDA_TRY(once_per_device(done, dev, [] {
    cudaError_t e = cudaFuncSetAttribute(k_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSmemMax);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_gram_df<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSmemMax);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_gram_df<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSmemMax);
    return e;
  }));
  return PG_OK;
}

// k_gram over the blocks of chunk points: 4, 2 or 1 tiles resident, as two
// buffers of them and the sums leave room for two blocks per SM (144 rows and
// 2048 outputs, more than any call has, fit with one).
static pg_status launch_gram(long N, long chunk, int blocks, const double* P, int na, const double* Q, int nb,
                             double* partial, const int* skip, cudaStream_t st) {
  const auto smem = [&](int logT) {
    return sizeof(double) * ((size_t)2 * (na + nb) * ((kTP << logT) + 1) + ((size_t)na * nb << logT));
  };
  int logT = 2;
  while (logT > 0 && smem(logT) > (size_t)kGramSmemMax) --logT;
  PG_TRY(opt_in_smem(smem(logT)));
  PG_CUDA_TRY(launch_dependent(k_gram, dim3(blocks), dim3(kT), smem(logT), st, N, chunk, P, na, Q, nb, logT, partial,
                               skip));
  return check_launch("k_gram");
}

pg_status gram(long N, const double* P, int na, const double* Q, int nb, double* out, RedScratch& rs,
               cudaStream_t st, bool dfloat, const double* Pt, const double* Qt, const int* skip, const PipPass* pass) {
  PG_ARG(na > 0 && nb > 0 && na * nb <= kMaxGramOut && na + nb <= 144, "gram: %d x %d outputs exceed the limits",
         na, nb);
  PG_TRY(rs.ensure(st));
  const long chunk = chunk_for(N, kRedBlocks, kTP);
  const int blocks = (int)((N + chunk - 1) / chunk);
  if (dfloat) {
    const GramGeom gg = gram_geometry(na, nb);
    PG_ARG(gg.nblk <= kT, "gram: %d output blocks", gg.nblk);  // at most ~160 within the limits above
    PG_TRY(opt_in_smem(gg.smem));
    const long dchunk = chunk_for(N, kRedBlocks, gg.tp);
    const int dblocks = (int)((N + dchunk - 1) / dchunk);
    const double* Ps = Pt ? Pt : P;
    const double* Qs = Qt ? Qt : Q;
    const int sp = Pt ? 1 : 0, sq = Qt ? 1 : 0;
    if (pair_ok(N, Ps, Qs))
      PG_CUDA_TRY(launch_dependent(k_gram_df<true>, dim3(dblocks), dim3(kT), gg.smem, st, N, dchunk, Ps, na, Qs, nb,
                                   gg.tp, gg.m, gg.S, gg.ablk, gg.nblk, sp, sq, rs.partial.p, skip));
    else
      PG_CUDA_TRY(launch_dependent(k_gram_df<false>, dim3(dblocks), dim3(kT), gg.smem, st, N, dchunk, Ps, na, Qs,
                                   nb, gg.tp, gg.m, gg.S, gg.ablk, gg.nblk, sp, sq, rs.partial.p, skip));
    PG_TRY(check_launch("k_gram_df"));
    return reduce(rs.partial.p, dblocks, na * nb, out, false, st, skip, pass, rs.counter.p);
  } else {
    PG_TRY(launch_gram(N, chunk, blocks, P, na, Q, nb, rs.partial.p, skip, st));
  }
  return reduce(rs.partial.p, blocks, na * nb, out, false, st, skip, pass, rs.counter.p);
}

// k_combine over blocks of chunk points; with P2 also Y2 from P2 (its blocks beside the others)
static pg_status launch_combine(long N, long chunk, int blocks, const double* P, const double* P2, int na,
                                const double* C, int ca, int cr, double cscale, const double* X, const double* alpha,
                                bool inv_sqrt, double* Y, double* Y2, int nr, double* sq, RedScratch& rs,
                                cudaStream_t st, const int* skip) {
  const size_t smem = sizeof(double) * (size_t)(na > 0 ? na : 1) * nr;
  // one kernel per number of outputs: an operation left out by a predicate
  // takes the FP64 pipe as long as any other (64 x 12 over 262144 points 570 us
  // as 16 outputs, 397 as 12; 40 x 5 186 as 8, 94 as 5)
#define PG_COMBINE(NRV)                                                                                             \
  case NRV:                                                                                                         \
    PG_CUDA_TRY(launch_dependent(k_combine<NRV>, dim3(blocks, P2 ? 2 : 1), dim3(kT), smem, st, N, chunk, P, P2, na, \
                                 C, ca, cr, cscale, X, alpha, inv_sqrt ? 1 : 0, Y, Y2, nr,                          \
                                 sq ? rs.partial.p : nullptr, sq, rs.counter.p, skip));                             \
    break
  switch (nr) {
    PG_COMBINE(1);
    PG_COMBINE(2);
    PG_COMBINE(3);
    PG_COMBINE(4);
    PG_COMBINE(5);
    PG_COMBINE(6);
    PG_COMBINE(7);
    PG_COMBINE(8);
    PG_COMBINE(9);
    PG_COMBINE(10);
    PG_COMBINE(11);
    PG_COMBINE(12);
    PG_COMBINE(13);
    PG_COMBINE(14);
    PG_COMBINE(15);
    PG_COMBINE(16);
  }
#undef PG_COMBINE
  return check_launch("k_combine");
}

pg_status combine_pair(long N, const double* P, const double* P2, int na, const double* C, int ca, int cr, double* Y,
                       double* Y2, int nr, double* sq, RedScratch& rs, cudaStream_t st) {
  PG_ARG(P && P2 && Y && Y2 && nr > 0 && nr <= kMaxCombine && na > 0 && na * nr <= 128 * kMaxCombine,
         "combine_pair: bad sizes na=%d nr=%d", na, nr);
  PG_TRY(rs.ensure(st));
  const long chunk = chunk_for(N, kStreamBlocks, kT);
  const int blocks = (int)((N + chunk - 1) / chunk);
  return launch_combine(N, chunk, blocks, P, P2, na, C, ca, cr, 1.0, nullptr, nullptr, false, Y, Y2, nr, sq, rs, st,
                        nullptr);
}

pg_status combine(long N, const double* P, int na, const double* C, int ca, int cr, double cscale, const double* X,
                  const double* alpha, bool inv_sqrt, double* Y, int nr, double* sq, RedScratch& rs,
                  cudaStream_t st, bool dfloat, const double* Pt, double* Yt, const int* skip) {
  PG_ARG(nr > 0 && nr <= kMaxCombine && na >= 0 && na * nr <= 128 * kMaxCombine, "combine: bad sizes na=%d nr=%d",
         na, nr);
  PG_TRY(rs.ensure(st));
  const long chunk = chunk_for(N, kStreamBlocks, kT);
  const int blocks = (int)((N + chunk - 1) / chunk);
  if (dfloat) {
#define PG_COMBINE_DF3(NRV, TI, TO)                                                                                \
  PG_CUDA_TRY(launch_dependent(k_combine_df<NRV, TI, TO>, dim3(blocks), dim3(kT), coef_bytes<NRV>(na), st, N, chunk, Pt ? Pt : P, na, \
                               C, ca, cr, cscale, X, alpha, inv_sqrt ? 1 : 0, Y, nr, reinterpret_cast<float2*>(Yt),  \
                               sq ? rs.partial.p : nullptr, sq, rs.counter.p, skip))
#define PG_COMBINE_DF(NRV)                                             \
  do {                                                                 \
    if (Pt && Yt) PG_COMBINE_DF3(NRV, true, true);                     \
    else if (Pt) PG_COMBINE_DF3(NRV, true, false);                     \
    else if (Yt) PG_COMBINE_DF3(NRV, false, true);                     \
    else PG_COMBINE_DF3(NRV, false, false);                            \
  } while (0)
    if (nr <= 1) PG_COMBINE_DF(1);
    else if (nr <= 2) PG_COMBINE_DF(2);
    else if (nr <= 4) PG_COMBINE_DF(4);
    else if (nr <= 6) PG_COMBINE_DF(6);
    else if (nr <= 8) PG_COMBINE_DF(8);
    else if (nr <= 10) PG_COMBINE_DF(10);
    else if (nr <= 12) PG_COMBINE_DF(12);
    else PG_COMBINE_DF(16);
#undef PG_COMBINE_DF
#undef PG_COMBINE_DF3
    PG_TRY(check_launch("k_combine_df"));
  } else {
    PG_TRY(launch_combine(N, chunk, blocks, P, nullptr, na, C, ca, cr, cscale, X, alpha, inv_sqrt, Y, nullptr, nr, sq,
                          rs, st, skip));
  }
  return PG_OK;  // with sq, the kernel's last block has reduced the norms
}

// The Ritz step of the mixed form in one pass: U_r = B v_r and
// W_r = Z v_r - lambda_r U_r in double-float from the twins of the m rows of
// B and Z (v_r = column r of V, leading dimension ldv), written as FP64, and
// |U_r|^2, |W_r|^2 (squares summed in FP32 per thread, in FP64 across threads)
// reduced by the last block into out[r] and out[nr + r].  On the FP32 pipe (24
// operations per output, row and point) next to the read of 16 bytes per row
// and point; the FP64 pipe only adds the norms.  4 roots over 262144 points,
// 8 / 30 / 60 rows: 27 / 61 / 102 us with FP64 additions per point, a read per
// coefficient and rows read as they are needed, now 23 / 47 / 80 (64 registers
// and four blocks per SM: 20 / 47 / 80, but 50 instead of 41 over 110592
// points and 60 rows, whose blocks all fit with three).
template <int NR>
__global__ void __launch_bounds__(kT, NR <= 4 ? 3 : 2) k_ritz_df(long N, long chunk, const double* Bt, const double* Zt,
                                                               int m, const double* __restrict__ V, int ldv,
                                                               const double* __restrict__ lam, double* U, double* W,
                                                               int nr, double* __restrict__ partial, double* out,
                                                               unsigned* counter) {
  constexpr bool kAhead = NR != 16;  // registers: 16 outputs spill
  constexpr int kRows = kBatch / 2;
  pdl_wait();
  pdl_release();
  extern __shared__ __align__(16) float smf[];
  float* Cs = smf;  // as in k_combine_df
  __shared__ float nlh[NR], nll[NR];
  __shared__ double red[kT / 32][2 * NR];
  load_coefs<NR>(Cs, m, nr, [&](int a, int r) { return V[(long)a + (long)r * ldv]; });
  if (threadIdx.x < nr) {
    float h, l;
    df_split(-lam[threadIdx.x], h, l);
    nlh[threadIdx.x] = h;
    nll[threadIdx.x] = l;
  }
  __syncthreads();
  float su[NR], sw[NR];  // about one point per thread: FP32 sums of the squares
#pragma unroll
  for (int r = 0; r < NR; ++r) su[r] = sw[r] = 0.f;
  const long g_begin = blockIdx.x * chunk;
  const long g_end = g_begin + chunk < N ? g_begin + chunk : N;
  for (long g = g_begin + threadIdx.x; g < g_end; g += kT) {
    float uh[NR], ul[NR], zh[NR], zl[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) uh[r] = ul[r] = zh[r] = zl[r] = 0.f;
    DfSums<NR> su2(uh, ul), sz2(zh, zl);
    // the next kRows rows of each are on their way while these are multiplied
    const double *rb = Bt + g, *rz = Zt + g;
    double pb[kRows], pz[kRows], nb[kRows], nz[kRows];
    auto rows = [&](double (&b)[kRows], double (&z)[kRows], int a0) {
#pragma unroll
      for (int u = 0; u < kRows; ++u) {
        b[u] = a0 + u < m ? rb[(long)(a0 + u) * N] : 0.0;
        z[u] = a0 + u < m ? rz[(long)(a0 + u) * N] : 0.0;
      }
    };
    rows(pb, pz, 0);
    for (int a0 = 0; a0 < m; a0 += kRows) {
      if (kAhead) rows(nb, nz, a0 + kRows);
#pragma unroll
      for (int u = 0; u < kRows; ++u) {
        if (a0 + u >= m) break;
        // the 8 bytes are a float2 (hi, lo): hi in the low word
        const float bh = __int_as_float(__double2loint(pb[u])), bl = __int_as_float(__double2hiint(pb[u]));
        const float qh = __int_as_float(__double2loint(pz[u])), ql = __int_as_float(__double2hiint(pz[u]));
        su2.add(bh, bl, Cs, a0 + u);
        sz2.add(qh, ql, Cs, a0 + u);
      }
      if (kAhead) {
#pragma unroll
        for (int u = 0; u < kRows; ++u) pb[u] = nb[u], pz[u] = nz[u];
      } else {
        rows(pb, pz, a0 + kRows);
      }
    }
    su2.get(uh, ul);
    sz2.get(zh, zl);
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r < nr) {
        df_fma(zh[r], zl[r], nlh[r], nll[r], uh[r], ul[r]);  // W = Z v - lambda U
        const double u = df_join<true>(uh[r], ul[r]);
        const double w = df_join<true>(zh[r], zl[r]);
        U[(long)r * N + g] = u;
        W[(long)r * N + g] = w;
        // the pair's sum in FP32 (after the cancellation in W its low part
        // need not be small against its high part), then its square
        const float uf = uh[r] + ul[r], wf = zh[r] + zl[r];
        su[r] = fmaf(uf, uf, su[r]);
        sw[r] = fmaf(wf, wf, sw[r]);
      }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // sums of 16 lanes in FP32 (2^-22 relative at most), the last step and
  // everything after it in FP64: few operations on the FP64 pipe
  float sq[2 * NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) sq[r] = su[r], sq[NR + r] = sw[r];
  packed_sums<2 * NR, 2>(sq, lane);
  constexpr int kRegs = NR == 16 ? 2 : 1;  // values per lane pair
#pragma unroll
  for (int i = 0; i < kRegs; ++i) {
    double a = f32_to_f64_int(sq[i]);
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    if (lane % (kRegs * 16 / NR) == 0) red[warp][lane * NR / 16 + i] = a;
  }
  __syncthreads();
  if (threadIdx.x < 2 * nr) {
    const int o = threadIdx.x < nr ? threadIdx.x : NR + threadIdx.x - nr;
    double t = 0;
    for (int w = 0; w < kT / 32; ++w) t += red[w][o];
    partial[(long)blockIdx.x * 2 * nr + threadIdx.x] = t;
  }
  reduce_in_last_block(partial, 2 * nr, out, 0, counter);
}

pg_status ritz_df(long N, const double* Bt, const double* Zt, int m, const double* V, int ldv, const double* lam,
                  double* U, double* W, int nr, double* sq, RedScratch& rs, cudaStream_t st) {
  PG_ARG(m > 0 && nr > 0 && nr <= kMaxCombine && m * nr <= 128 * kMaxCombine && Bt && Zt,
         "ritz_df: bad sizes m=%d nr=%d", m, nr);
  PG_TRY(rs.ensure(st));
  const long chunk = chunk_for(N, kStreamBlocks, kT);
  const int blocks = (int)((N + chunk - 1) / chunk);
#define PG_RITZ_DF(NRV)                                                                                           \
  PG_CUDA_TRY(launch_dependent(k_ritz_df<NRV>, dim3(blocks), dim3(kT), coef_bytes<NRV>(m), st, N, chunk, Bt, Zt, m, V, ldv, lam, U, \
                               W, nr, rs.partial.p, sq, rs.counter.p))
  if (nr <= 1) PG_RITZ_DF(1);
  else if (nr <= 2) PG_RITZ_DF(2);
  else if (nr <= 4) PG_RITZ_DF(4);
  else if (nr <= 8) PG_RITZ_DF(8);
  else PG_RITZ_DF(16);
#undef PG_RITZ_DF
  return check_launch("k_ritz_df");
}

pg_status split_twin(long count, const double* x, double* t, cudaStream_t st, double* copy) {
  if (count <= 0) return PG_OK;
  const long b = (count + kT - 1) / kT;
  PG_CUDA_TRY(launch_dependent(k_split_twin, dim3((unsigned)(b < 152L * 8 ? b : 152L * 8)), dim3(kT), 0, st, count, x,
                               reinterpret_cast<float2*>(t), copy));
  return check_launch("k_split_twin");
}


// The reduction scratch of the public block products: one per calling
// thread and device (a buffer allocated on one device is not used on another).
constexpr int kScratchDevices = 64;
pg_status thread_scratch(RedScratch** out) {
  static thread_local RedScratch rs[kScratchDevices];
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev));
  PG_ARG(dev >= 0 && dev < kScratchDevices, "block products: device %d out of range", dev);
  *out = &rs[dev];
  return PG_OK;
}

}  // namespace pg

extern "C" pg_status pg_block_gram(long n, const double* P, int np, const double* Q, int nq, double* out,
                                   int precision, void* stream) {
  PG_ARG(n > 0 && P && Q && out && np > 0 && nq > 0, "pg_block_gram: bad arguments");
  PG_ARG(precision == PG_FP64 || precision == PG_MIXED, "pg_block_gram: unknown precision");
  pg::RedScratch* rs = nullptr;
  PG_TRY(pg::thread_scratch(&rs));
  return pg::gram(n, P, np, Q, nq, out, *rs, pg::as_stream(stream), precision == PG_MIXED);
}

extern "C" pg_status pg_block_combine(long n, const double* P, int np, const double* C, int ny, double* Y,
                                      int precision, void* stream) {
  PG_ARG(n > 0 && P && C && Y && np > 0 && ny > 0, "pg_block_combine: bad arguments");
  PG_ARG(precision == PG_FP64 || precision == PG_MIXED, "pg_block_combine: unknown precision");
  pg::RedScratch* rs = nullptr;
  PG_TRY(pg::thread_scratch(&rs));
  return pg::combine(n, P, np, C, ny, 1, 1.0, nullptr, nullptr, false, Y, ny, nullptr, *rs, pg::as_stream(stream),
                     precision == PG_MIXED);
}

extern "C" pg_status pg_split_twin(long n, const double* x, double* twin, void* stream) {
  PG_ARG(n > 0 && x && twin && x != twin, "pg_split_twin: bad arguments");
  return pg::split_twin(n, x, twin, pg::as_stream(stream));
}

extern "C" pg_status pg_block_gram_twin(long n, const double* Pt, int np, const double* Qt, int nq, double* out,
                                        void* stream) {
  PG_ARG(n > 0 && Pt && Qt && out && np > 0 && nq > 0, "pg_block_gram_twin: bad arguments");
  pg::RedScratch* rs = nullptr;
  PG_TRY(pg::thread_scratch(&rs));
  return pg::gram(n, Pt, np, Qt, nq, out, *rs, pg::as_stream(stream), true, Pt, Qt);
}

extern "C" pg_status pg_block_combine_twin(long n, const double* Pt, int np, const double* C, int ny, double* Y,
                                           double* Yt, void* stream) {
  PG_ARG(n > 0 && Pt && C && Y && np > 0 && ny > 0, "pg_block_combine_twin: bad arguments");
  pg::RedScratch* rs = nullptr;
  PG_TRY(pg::thread_scratch(&rs));
  return pg::combine(n, Pt, np, C, ny, 1, 1.0, nullptr, nullptr, false, Y, ny, nullptr, *rs, pg::as_stream(stream),
                     true, Pt, Yt);
}

// ---------------------------------------------------------------------------
// pg_block_gram_noalloc: pg_block_gram for callers that may not allocate
// device memory.  The per-block partial sums live in a fixed file-scope
// device array instead of a cudaMalloc'd buffer; the kernels and the
// reduction order are pg_block_gram's, so the results are bit-identical.
namespace {

constexpr int kNoAllocMaxOut = 256;  // np * nq limit of this entry point
constexpr long kNoAllocPartials = (long)pg::kRedBlocks * kNoAllocMaxOut;  // 75,776 doubles = 592 KiB

// Nothing here needs to start at zero: each call writes every partial it
// reads back.  One array per device, shared by every caller of the entry point.
__device__ __align__(256) double g_noalloc_partial[kNoAllocPartials];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_m;
double* g_noalloc_ptr[kNoAllocMaxDevices] = {};

}  // namespace

extern "C" pg_status pg_block_gram_noalloc(long n, const double* P, int np, const double* Q, int nq, double* out,
                                           int precision, void* stream) {
  using namespace pg;
  PG_ARG(n > 0 && P && Q && out && np > 0 && nq > 0, "pg_block_gram_noalloc: bad arguments");
  PG_ARG(precision == PG_FP64 || precision == PG_MIXED, "pg_block_gram_noalloc: unknown precision");
  PG_ARG((long)np * nq <= kNoAllocMaxOut,
         "pg_block_gram_noalloc: %d x %d = %ld outputs exceed this entry point's fixed scratch (at most %d "
         "outputs; use pg_block_gram)",
         np, nq, (long)np * nq, kNoAllocMaxOut);
  PG_ARG(np + nq <= 144, "pg_block_gram_noalloc: np + nq = %d exceeds 144", np + nq);
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev));
  PG_ARG(dev >= 0 && dev < kNoAllocMaxDevices, "pg_block_gram_noalloc: device %d out of range", dev);
  double* partial = nullptr;
  {
    // first call on a device: the address of the scratch array in this
    // device's context (no allocation; done before any stream capture)
    std::lock_guard<std::mutex> l(g_noalloc_m);
    if (!g_noalloc_ptr[dev]) {
      void* addr = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_partial);
      if (e != cudaSuccess || !addr) {
        set_error("pg_block_gram_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        return PG_CUDA;
      }
      g_noalloc_ptr[dev] = static_cast<double*>(addr);
    }
    partial = g_noalloc_ptr[dev];
  }
  cudaStream_t st = as_stream(stream);
  const int no = np * nq;
  if (precision == PG_MIXED) {
    const GramGeom gg = gram_geometry(np, nq);
    PG_ARG(gg.nblk <= kT, "pg_block_gram_noalloc: %d output blocks", gg.nblk);
    PG_TRY(opt_in_smem(gg.smem));
    const long chunk = chunk_for(n, pg::kRedBlocks, gg.tp);
    const int blocks = (int)((n + chunk - 1) / chunk);
    if (pair_ok(n, P, Q))
      k_gram_df<true><<<blocks, kT, gg.smem, st>>>(n, chunk, P, np, Q, nq, gg.tp, gg.m, gg.S, gg.ablk, gg.nblk, 0,
                                                    0, partial, nullptr);
    else
      k_gram_df<false><<<blocks, kT, gg.smem, st>>>(n, chunk, P, np, Q, nq, gg.tp, gg.m, gg.S, gg.ablk, gg.nblk, 0,
                                                     0, partial, nullptr);
    PG_TRY(check_launch("k_gram_df"));
    return reduce(partial, blocks, no, out, false, st);
  }
  const long chunk = chunk_for(n, pg::kRedBlocks, kTP);
  const int blocks = (int)((n + chunk - 1) / chunk);
  PG_TRY(launch_gram(n, chunk, blocks, P, np, Q, nq, partial, nullptr, st));
  return reduce(partial, blocks, no, out, false, st);
}
