// FP64 products on the FP16 tensor cores by exact slicing.
//
// An FP64 value of a line (a row of the left operand) is taken as an integer
// F = x 2^s of at most 62 bits and sign, s from the line's largest exponent,
// and written in seven balanced digits of 9 bits, F = sum_i D_i 2^(9 (6-i)),
// -256 <= D_i < 256.  The digits are small integers, exact in FP16, and so
// are those of the right operand (one scale for the whole matrix).  The
// tensor core multiplies digit images and accumulates in FP32, where sums of
// integers below 2^24 are exact; products of equal weight (i + j = d) share
// one accumulator, and those with d > 6 (2^-60 of the operands' scale) are
// left out: 28 products.  The accumulators are put together with integer
// arithmetic and rounded once to FP64, so the product of a line and a matrix
// column is the sum of the operands quantised to 2^-62 of the line's (the
// matrix's) largest value with one rounding at the end, where a chain of
// FP64 multiply-adds rounds n times.  (Six digits, 2^-53, were not enough:
// on smooth vectors, whose kinetic terms cancel, the error was ten times
// that of FP64.)  This is the scheme of K. Ozaki, T. Ogita, S. Oishi, S. M.
// Rump, Numer. Algorithms 59 (2012) 95, with power-of-two line scales.
//
// Why: the FP64 pipe of this part issues a warp-wide instruction about every
// 74 cycles per SM sub-partition (0.55e12 lane operations a second, the FP32
// and integer pipes about 40e12), so conversions in integer arithmetic and
// 28 tensor-core products cost less than one FP64 multiply-add each.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

#include "pg_common.cuh"

namespace pg {

constexpr int kSliceAcc = 7;  // accumulators: digit products with i + j = 0 .. 6

constexpr int kSliceP = 9;                          // bits of a digit
constexpr int kSliceN = 7;                          // digits of a value
constexpr int kSliceGuard = kSliceN * kSliceP - 1 - 53;  // bits below the FP64 mantissa
constexpr int kSliceUnit = kSliceP * (2 * kSliceN - 2 - (kSliceAcc - 1));  // log2 of the weight of accumulator 6

// F of a value whose line has the largest biased exponent emax: mantissa
// 2^kGuard >> (emax - its own exponent), rounded to nearest, with the sign,
// plus the bias that makes every digit non-negative: digit i sits in bits
// [9 (6-i), 9 (7-i)) as D_i + 256 (the first one upwards of them).
__device__ __forceinline__ unsigned long long slice_fixed(double x, int emax) {
  constexpr unsigned long long kBias = [] {
    unsigned long long b = 0;
    for (int i = 0; i < kSliceN; ++i) b |= 1ull << (kSliceP * i + kSliceP - 1);
    return b;
  }();
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
  const int e = (int)((h >> 20) & 0x7ffu);
  uint32_t mh = (h & 0xfffffu) | (e ? 0x100000u : 0u), ml = l;
  mh = __funnelshift_l(ml, mh, kSliceGuard);
  ml <<= kSliceGuard;
  // right shift by s = emax - e with rounding to nearest (half up)
  int s = emax - (e ? e : 1);
  s = s > 63 ? 63 : s;
  const bool far = s >= 32;
  const uint32_t ss = (uint32_t)s & 31u;
  const uint32_t a1 = far ? 0u : mh, a0 = far ? mh : ml, am = far ? ml : 0u;
  const uint32_t r1 = a1 >> ss;
  const uint32_t r0 = __funnelshift_r(a0, a1, ss);
  const uint32_t rm = __funnelshift_r(am, a0, ss);  // the bits shifted out, left-aligned
  unsigned long long f = ((unsigned long long)r1 << 32 | r0) + (rm >> 31);
  f = (int)h < 0 ? 0ull - f : f;
  return f + kBias;
}

// Digit i of two biased values, as two FP16 integers.
__device__ __forceinline__ uint32_t slice_digit2(unsigned long long f0, unsigned long long f1, int i) {
  const int sh = kSliceP * (kSliceN - 1 - i);
  // the most significant digit may reach 256: it is not cut to kSliceP bits
  const uint32_t m = i > 0 ? (1u << kSliceP) - 1u : ~0u;
  const uint32_t d0 = (uint32_t)(f0 >> sh) & m, d1 = (uint32_t)(f1 >> sh) & m;
  // 1024 + digit as FP16 bits, then minus 1024 + 256: exact
  const uint32_t u = (d1 << 16) + d0 + 0x64006400u;
  const __half2 c = __half2half2(__ushort_as_half((unsigned short)(0x6400u + (1u << (kSliceP - 1)))));
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&u), c);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// sum_d acc_d 2^(kSliceP (6-d)) 2^e (acc_d integers below 2^24 in magnitude) rounded
// to FP64 with integer operations; the result's exponent must be in range.
__device__ __forceinline__ double slice_join(const float* acc, int e) {
  int a[kSliceAcc];
#pragma unroll
  for (int d = 0; d < kSliceAcc; ++d) a[d] = __float2int_rn(acc[d]);
  const long long t01 = (long long)a[0] * (1 << kSliceP) + a[1];
  const long long t23 = (long long)a[2] * (1 << kSliceP) + a[3];
  long long hi = (t01 << (2 * kSliceP)) + t23;
  const long long t45 = (long long)a[4] * (1 << kSliceP) + a[5];
  const long long lo = t45 * (1 << kSliceP) + a[6];
  hi += lo >> (3 * kSliceP);
  const uint32_t sgn = (uint32_t)(hi >> 63);
  // magnitude as the 96-bit word [m : l] with l left-aligned (one's complement of a negative sum)
  uint32_t l = ((uint32_t)lo & ((1u << (3 * kSliceP)) - 1u)) << (32 - 3 * kSliceP);
  uint32_t w2 = (uint32_t)((unsigned long long)hi >> 32) ^ sgn, w1 = (uint32_t)hi ^ sgn, w0 = l ^ sgn;
  int ex = e + 1023 + 63 + 3 * kSliceP;
  if (w2 == 0) {  // small against the line's largest value
    const bool two = w1 == 0;
    ex -= two ? 64 : 32;
    w2 = two ? w0 : w1;
    w1 = two ? 0u : w0;
    w0 = 0u;
  }
  const int lz = __clz((int)w2);
  ex -= lz;
  const uint32_t u1 = __funnelshift_l(w1, w2, lz & 31), u0 = __funnelshift_l(w0, w1, lz & 31);
  const unsigned long long u = (unsigned long long)u1 << 32 | u0;
  unsigned long long r = (u >> 11) + ((u >> 10) & 1ull) + ((unsigned long long)(uint32_t)(ex - 1) << 52);
  r |= (unsigned long long)(sgn & 0x80000000u) << 32;
  return __longlong_as_double(lz >= 32 ? 0ll : (long long)r);
}

// The images of every matrix of a grid (t_dev, q_dev, qb_dev), made on the
// device in one launch; equal matrices share one image.
pg_status slice_grid(pg_grid* g);

// Y (mode) = A x_axis X for nvec vectors of a grid of n points, FP64:
// mode 0: Y = A X, 1: Y += A X, 2: Y = V X + A X.
pg_status slice_axis(const pg_grid* g, int axis, const SliceMat& S, const double* A64, const double* v,
                     const double* x, double* y, int nvec, int mode, cudaStream_t st);

// Rows times a matrix: X is nlines x n (row-major), A n x n.
// kRowStore: Y = X A.  kRowDot: Y holds *rows rows of nlines values whose sum
// over the rows is x . (x A) for each line (at most slice_row_count(n)).
// A64 and the images (slice_rows_matrix) on the device; err as tc_err.
enum SliceRows { kRowStore = 0, kRowDot = 3 };
int slice_row_count(int n);
// shape and bytes of the images of an n x n matrix whose largest entry is big
size_t slice_rows_shape(int n, double big, SliceMat* S);
pg_status slice_rows_matrix(const double* A64, unsigned char* img, SliceMat* S, cudaStream_t st);
pg_status slice_rows(long nlines, const SliceMat& S, const double* A64, const double* x, double* y, SliceRows mode,
                     int* rows, int* err, cudaStream_t st);

}  // namespace pg
