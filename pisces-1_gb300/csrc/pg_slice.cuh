// FP64 products on the FP16 tensor cores by slicing both operands.
//
// An FP64 value of a line (a row of the left operand) is taken as an integer
// F = x 2^s of at most 79 bits and sign, s from the line's largest exponent,
// and written in ten balanced digits of 8 bits, F = sum_i D_i 2^(8 (9-i)),
// -128 <= D_i <= 128.  The digits are small integers, exact in FP16, and so
// are those of the right operand (one scale for the whole matrix).  The
// tensor core multiplies digit images and accumulates in FP32, where sums of
// integers up to 2^24 are exact: products of equal weight (i + j = d) share
// accumulator d, n values give at most n (d + 1) 2^14 there, and a launch
// takes no more than 96 values, 0.94 x 2^24 at the last accumulator (d = 9).
// Products with d > 9 are left out: 55 remain.  The accumulators are put
// together with integer arithmetic and rounded once to FP64.
//
// What a product of line and matrix column is off by, with u = 2^-53, X and A
// the largest values of the line and of the matrix and n the line's length:
//   - one rounding of the result, u |y| (and one per launch of 96 values that
//     is added up);
//   - the operands' rounding to 79 bits below their largest values,
//     2^-79 (X sum |a| + A sum |x|), nothing for values that keep their 53
//     bits there, i.e. within 2^26 of the largest;
//   - the products left out, below 2^-74.5 A X with random digits and n = 96
//     (2^-69 at the very worst).
// A chain of FP64 multiply-adds is off by up to n u sum |a x|.  On a sine-DVR
// axis no entry of T is below 2^-26 of the largest up to 160 points (there
// 2^-25.4; beyond, the grid takes the chain), so sum |a x| >= 2^-26 A X and a
// product is within two or three roundings of its own terms' magnitude, value
// by value, also in the tails of a wavefunction.  (62 bits, seven digits of 9,
// were not enough: near the norm they were better than the chain, in the tails
// of exp(-|r|) on 96 points 4e-12 against 2e-14, and their accumulators could
// pass 2^24.)  This is the scheme of K. Ozaki, T. Ogita, S. Oishi, S. M. Rump,
// Numer. Algorithms 59 (2012) 95, with power-of-two line scales.
//
// Why: the FP64 pipe of this part issues a warp-wide instruction about every
// 74 cycles per SM sub-partition (0.55e12 lane operations a second, the FP32
// and integer pipes about 40e12), so conversions in integer arithmetic and
// 55 tensor-core products cost less than one FP64 multiply-add each.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

#include "pg_common.cuh"

namespace pg {

constexpr int kSliceP = 8;                          // bits of a digit
constexpr int kSliceN = 10;                         // digits of a value
constexpr int kSliceAcc = 10;                       // accumulators: digit products with i + j = 0 .. 9
constexpr int kSliceK = 96;                         // values of a launch: sums of an accumulator stay below 2^24
constexpr int kSliceGuard = kSliceN * kSliceP - 1 - 53;  // bits below the FP64 mantissa
constexpr int kSliceUnit = kSliceP * (2 * kSliceN - 2 - (kSliceAcc - 1));  // log2 of the weight of accumulator 9
constexpr int kSliceBits = 97;                      // of a product put together, in units of accumulator 9
static_assert((long long)kSliceK * kSliceAcc << (2 * (kSliceP - 1)) <= 1ll << 24, "sums of an accumulator are exact");

// F + 128 (1 + 2^8 + .. + 2^72): digit i sits in byte 9 - i as D_i + 128 (the
// first one upwards of it: it may reach 256).
struct SliceInt {
  uint32_t w0, w1, w2;
};

// F of a value whose line has the largest biased exponent emax: mantissa
// 2^kSliceGuard >> (emax - its own exponent), rounded to nearest, with the
// sign.
__device__ __forceinline__ SliceInt slice_fixed(double x, int emax) {
  static_assert(kSliceGuard == 26 && kSliceP == 8 && kSliceN == 10, "words and bytes below");
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
  const int e = (int)((h >> 20) & 0x7ffu);
  const uint32_t mh = (h & 0xfffffu) | (e ? 0x100000u : 0u);
  const uint32_t w0 = l << 26, w1 = __funnelshift_l(l, mh, 26), w2 = mh >> 6;
  // right shift by s = emax - e, rounded to nearest (half up)
  int s = emax - (e ? e : 1);
  s = s > 127 ? 127 : s;
  const bool s32 = s >= 32, s64 = s >= 64, s96 = s >= 96;
  const uint32_t ss = (uint32_t)s & 31u;
  const uint32_t a2 = s32 ? 0u : w2, a1 = s32 ? (s64 ? 0u : w2) : w1;
  const uint32_t a0 = s32 ? (s64 ? (s96 ? 0u : w2) : w1) : w0, am = s32 ? (s64 ? (s96 ? 0u : w1) : w0) : 0u;
  const uint32_t r2 = a2 >> ss, r1 = __funnelshift_r(a1, a2, ss), r0 = __funnelshift_r(a0, a1, ss);
  const uint32_t rm = __funnelshift_r(am, a0, ss);  // the bits shifted out, left-aligned
  // two's complement of a negative value: the carry of ~r + 1 and the rounding together
  const uint32_t sg = (uint32_t)((int)h >> 31), c = (rm >> 31) ^ (sg & 1u);
  const unsigned long long bias = 0x8080808080808080ull + c;
  const unsigned long long lo = ((unsigned long long)(r1 ^ sg) << 32 | (r0 ^ sg)) + bias;
  return SliceInt{(uint32_t)lo, (uint32_t)(lo >> 32), (r2 ^ sg) + 0x8080u + (lo < bias ? 1u : 0u)};
}

// Digit i of two values, as two FP16 integers.
__device__ __forceinline__ uint32_t slice_digit2(const SliceInt& f0, const SliceInt& f1, int i) {
  const int b = kSliceN - 1 - i;
  uint32_t u;
  if (i == 0) {  // bits 72 .. 80
    u = __byte_perm(f0.w2, f1.w2, 0x6521) + 0x64006400u;
  } else {
    const uint32_t p = b < 4 ? f0.w0 : (b < 8 ? f0.w1 : f0.w2), q = b < 4 ? f1.w0 : (b < 8 ? f1.w1 : f1.w2);
    const unsigned k = (unsigned)b & 3u;
    u = (__byte_perm(p, q, k | k << 4 | (4u + k) << 8 | (4u + k) << 12) & 0x00ff00ffu) | 0x64006400u;
  }
  // 1024 + byte as FP16 bits, then minus 1024 + 128: exact
  const __half2 c = __half2half2(__ushort_as_half((unsigned short)(0x6400u + (1u << (kSliceP - 1)))));
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&u), c);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// sum_d acc_d 2^(8 (9-d)) 2^e (acc_d integers up to 2^24 in magnitude) rounded
// to FP64 with integer operations; e in [-1022, 1023 - kSliceBits], so that the
// result is zero or a normal number.
__device__ __forceinline__ double slice_join(const float* acc, int e) {
  long long t[kSliceAcc / 2];
#pragma unroll
  for (int d = 0; d < kSliceAcc / 2; ++d)
    t[d] = (long long)__float2int_rn(acc[2 * d]) * (1 << kSliceP) + __float2int_rn(acc[2 * d + 1]);
  // words of 32 bits: four digits each, the first two at the top
  const long long l = (t[3] << 16) + t[4];
  const long long m = (t[1] << 16) + t[2] + (l >> 32);
  const long long q = t[0] + (m >> 32);
  const uint32_t sg = (uint32_t)(q >> 63);
  unsigned long long lo = ((unsigned long long)((uint32_t)m ^ sg) << 32 | ((uint32_t)l ^ sg)) + (sg & 1u);
  unsigned long long hi = ((unsigned long long)q ^ ((unsigned long long)sg << 32 | sg)) + (sg && lo == 0 ? 1u : 0u);
  // the leading word to the top of [v3 : v2 : v1 : v0]
  uint32_t v3 = (uint32_t)(hi >> 32), v2 = (uint32_t)hi, v1 = (uint32_t)(lo >> 32);
  const uint32_t v0 = (uint32_t)lo;
  int ex = e + 1023 + 127;
  const bool up = v3 == 0;
  ex -= up ? 32 : 0;
  v3 = up ? v2 : v3;
  v2 = up ? v1 : v2;
  v1 = up ? v0 : v1;
  if (v3 == 0) {  // small against the line's largest value; up, so v1 = v0
    const bool two = v2 == 0;
    ex -= two ? 64 : 32;
    v3 = two ? v1 : v2;
    v2 = two ? 0u : v1;
    v1 = 0u;
  }
  const int lz = __clz((int)v3);
  ex -= lz;
  const uint32_t u1 = __funnelshift_l(v2, v3, lz & 31), u0 = __funnelshift_l(v1, v2, lz & 31);
  const unsigned long long u = (unsigned long long)u1 << 32 | u0;
  unsigned long long r = (u >> 11) + ((u >> 10) & 1ull) + ((unsigned long long)(uint32_t)(ex - 1) << 52);
  r |= (unsigned long long)(sg & 0x80000000u) << 32;
  return __longlong_as_double(lz >= 32 ? 0ll : (long long)r);
}

// SMs of a device.
int sm_count(int device);

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
// A64 and the images (slice_rows_matrix) on the device of g.
enum SliceRows { kRowStore = 0, kRowDot = 3 };
int slice_row_count(int n);
// Shape and bytes of the images of an n x n matrix whose largest entry is big
// and whose columns that are not zero all reach low.  A column far below the
// largest would keep few of its bits (one scale for the matrix): from 2^-20 on,
// as for entries outside the slices' range, every line goes by multiply-adds.
size_t slice_rows_shape(int n, double big, double low, SliceMat* S);
pg_status slice_rows_matrix(const double* A64, unsigned char* img, SliceMat* S, cudaStream_t st);
pg_status slice_rows(const pg_grid* g, long nlines, const SliceMat& S, const double* A64, const double* x, double* y,
                     SliceRows mode, int* rows, cudaStream_t st);

}  // namespace pg
