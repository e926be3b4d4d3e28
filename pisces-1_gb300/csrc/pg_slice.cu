// One axis contraction Y (+)= A x_axis X in FP64 on the tensor cores, from
// exact FP16 slices of both operands (pg_slice.cuh); the H*X product and the
// kinetic preconditioner of the FP64 form are three and six of these.
//
// Grid lines along the axis are the rows of the left operand: a CTA takes
// 128 of them (fewer on small grids), converts their values to digit images
// once (each line scaled by its own largest exponent; above 64 points once
// per 48 outputs), and multiplies them with the matrix's digit images, which
// the bulk copy engine fetches from L2.  The tensor core's accumulators (10 x
// nc columns of TMEM) are read back one line per lane.
//
// Bounds: per point and axis about 40 integer operations to make the digits,
// 95 to join the accumulators and one or two FP64 operations (V X, the sum
// into Y), against n FP64 multiply-adds before; the FP64 pipe is about 60
// times slower than the integer pipes here.  No one part sets the time: of an
// axis of 64^3 x 4 (a tile per CTA) the products cost 6 % beside the rest, the
// joins 11 %, the digits 9 %; the others are the latencies of the lines' loads,
// of each N chunk's read-out and of its sum into Y.
//
// H X, us, FP64 multiply-adds / slices of seven 9-bit digits (whose operands
// and sums were not exact, pg_slice.cuh) / as here: 32^3 34.0 / 19.9 / 21.3,
// 64^3 x 4 344 / 53.0 / 62.8, 83x90x71 x 6 1816 / 173 / 307, 96^3 x 8 3320 / 341
// / 581, 160^3 x 16 (K chunks, two launches an axis) 63100 / 5505 / 10360.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "pg_slice.cuh"
#include "pg_tc16.cuh"

namespace {

// Polls of a barrier after which its waiters carry on by multiply-adds.
#ifndef PG_SLICE_POLLS
#define PG_SLICE_POLLS (1l << 26)
#endif
#ifndef PG_SLICE_POLLS_ISSUE
#define PG_SLICE_POLLS_ISSUE (1l << 26)
#endif
template <long kPolls>
__device__ __forceinline__ bool wait_for(uint32_t bar, uint32_t parity) {
  for (long it = 0; it < kPolls; ++it)
    if (mbar_try(bar, parity)) return true;
  return false;
}

constexpr int kLines = 128;  // MMA M
constexpr int kST = 512;     // threads that fill and read out
constexpr int kTransMost = (kST / 32) * 32 * 5 * 8;  // transpose buffer: 32 lines x 4 columns per warp

// A line whose largest exponent lies outside [exp_lo, exp_hi] (subnormal or
// huge values, infinities, NaN, products that could leave the range of normal
// numbers) is multiplied with FP64 multiply-adds instead.

struct SliceArgs {
  long nlines;   // lines of all vectors
  long inner;    // stride of the axis
  long npts;     // points of one vector (index of V)
  int n, kc, nnc, nc;
  int lc;        // lines per CTA: 128, or 64 or 32 where that still leaves one CTA per SM at most
  int h0, nch;   // K chunks [h0, h0 + nch) of this launch
  int plain;     // every line by FP64 multiply-adds
  int exp_lo, exp_hi;
  int nc_per;    // N chunks per CTA (blockIdx.y takes the next ones)
  int scale;     // exponent of accumulator 9: kSliceUnit - tau - 1075 - kSliceGuard
  uint32_t block_bytes;  // one (K, N) block of the matrix image
  uint32_t off_b, off_t; // shared-memory offsets of the matrix blocks and the transpose buffer
  int tc;                // columns transposed at a time: 4, or 2 where shared memory is short
  uint32_t tmem_cols;
  int mode;              // 0: y = K, 1: y += K, 2: y = v x + K, 3: row dots x . K
  long out0;             // mode 3: first output row of this launch, in values
  long sa, sb;           // strides of A64 (output, input index)
};

// kChunks false: the whole axis in one K chunk (n <= 64).  The lines' digits
// are made once; the matrix comes in chunks of nc columns, double buffered,
// into two halves of tensor memory, so that a chunk's products run while the
// one before is read out.
// kChunks true: K chunks of at most 48, N chunks of at most 48; the digits are
// made again for every N chunk.
// The products of the former are issued by a warp of its own (the 17th), which
// waits for the matrix blocks and for the accumulators to be read: issued
// by a thread that also reads out, two chunks of 64^3 took 5600 cycles before
// its read-out began.
// Every wait is bounded, and Y does not depend on them: where one runs out, the
// outputs that it was for are computed by FP64 multiply-adds, as for lines
// outside the slices' range.  Copies and products in flight are waited for
// again before the block gives its memory back.
template <int NU, bool kChunks>
__global__ void __launch_bounds__(kST + (kChunks ? 0 : 32), 1)
    k_slice_axis(const SliceArgs A, const unsigned char* __restrict__ img, const double* __restrict__ A64,
                 const double* __restrict__ v, const double* __restrict__ x, double* y) {
  constexpr int NS = pg::kSliceN;
  constexpr int kBuf = kChunks ? 1 : 2;  // matrix blocks and accumulator sets
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar_b[kBuf], bar_mma[kBuf], bar_read[kBuf];
  __shared__ uint32_t tmem_base;
  __shared__ int s_emax[kLines];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c_first = blockIdx.y * A.nc_per;
  const int c_end = c_first + A.nc_per < A.nnc ? c_first + A.nc_per : A.nnc;
  const uint32_t sA = smem_u32(smem), sB = sA + A.off_b;

  auto load_b = [&](int c, int h, int b) {  // one thread: block (h, c) of the matrix image into buffer b
    uint64_t state;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 %0, [%1], %2;"
                 : "=l"(state)
                 : "r"(smem_u32(&bar_b[b])), "r"(A.block_bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     sB + (uint32_t)b * A.block_bytes),
                 "l"(img + (size_t)((A.h0 + h) * A.nnc + c) * A.block_bytes), "r"(A.block_bytes),
                 "r"(smem_u32(&bar_b[b]))
                 : "memory");
  };
  if (tid == 0) {
    for (int b = 0; b < kBuf; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_b[b])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_mma[b])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&bar_read[b])), "r"(kST / 32));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // constant data: before the kernel ahead has finished
    for (int b = 0; b < kBuf && c_first + b < c_end; ++b) load_b(c_first + b, 0, b);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(A.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid < kLines) s_emax[tid] = 0;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pg::pdl_wait();
  pg::pdl_release();
  const uint32_t tmem = tmem_base;

  const bool contig = A.inner == 1;
  const long l0 = blockIdx.x * (long)A.lc;
  const int lend = A.nlines - l0 < A.lc ? (int)(A.nlines - l0) : A.lc;  // lines of this CTA
  // filling: this thread's line, and its octets part, part + parts, ...
  const int line = tid & (A.lc - 1), part = tid / A.lc, parts = kST / A.lc;
  // read-out: this thread's TMEM lane
  const int row = 32 * (warp & 3) + lane, wpart = warp >> 2;
  auto first_point = [&](int r) {  // of line r of the tile
    const long l = r < lend ? l0 + r : 0;
    return contig ? l * A.n : (l / A.inner) * A.inner * A.n + l % A.inner;
  };
  const int koct = A.kc >> 3;
  // Octets of a K chunk that hold values, in whole K steps: of several, the last
  // one may end early, and so may the last N chunk's batches (72^3 x 4 274 us with
  // the padding, 245 so; one chunk is the axis itself, and a bound that is not
  // the same for all its N chunks costs 64^3 x 4 63 -> 69).
  auto octets = [&](int h) {
    const int kn = A.n - (A.h0 + h) * A.kc;
    return kChunks && kn < A.kc ? ((kn + 15) >> 4) << 1 : koct;
  };
  const int k_end = (A.h0 + A.nch) * A.kc < A.n ? (A.h0 + A.nch) * A.kc : A.n;

  double val[NU][8];
  auto load_chunk = [&](int h) {
    const int k0 = (A.h0 + h) * A.kc;
    const int kn = A.n - k0 < A.kc ? A.n - k0 : A.kc;
    if (contig) {
      // the lines are contiguous: coalesced through shared memory (the digit
      // images' place), odd pitch
      double* raw = reinterpret_cast<double*>(smem);
      const int pitch = A.kc | 1;
      for (int r = warp; r < A.lc; r += kST / 32)
        for (int k = lane; k < A.kc; k += 32) {
          const bool in = r < lend && k < kn;
          const double* src = x + (in ? (l0 + r) * A.n + k0 + k : 0);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(sA + 8u * (uint32_t)(r * pitch + k)),
                       "l"(src), "r"(in ? 8 : 0)
                       : "memory");
        }
      asm volatile("cp.async.wait_all;" ::: "memory");
      named_sync(1, kST);
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int o = part + parts * u;
#pragma unroll
        for (int q = 0; q < 8; ++q) val[u][q] = o < koct ? raw[line * pitch + 8 * o + q] : 0.0;
      }
    } else {
      const double* src = x + first_point(line);
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int o = part + parts * u;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int k = 8 * o + q;
          val[u][q] = (line < lend && o < koct && k < kn) ? src[(long)(k0 + k) * A.inner] : 0.0;
        }
      }
    }
  };
  auto chunk_emax = [&] {
    uint32_t em = 0;
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t h = (uint32_t)__double2hiint(val[u][q]) & 0x7fffffffu;
        // a subnormal counts as exponent 0 but not as zero: 1 marks it
        const uint32_t t = h >= 0x100000u ? h >> 20 : ((h | (uint32_t)__double2loint(val[u][q])) ? 1u : 0u);
        em = t > em ? t : em;
      }
    if (em) atomicMax(&s_emax[line], (int)em);
  };
  // a line's scale, once its maximum is complete; slow: by FP64 multiply-adds
  auto is_slow = [&](int em) { return A.plain || (em != 0 && (em < A.exp_lo || em > A.exp_hi)); };
  const uint32_t lbo = 128, sbo = (uint32_t)koct * 128u;
  const uint32_t a_slice = (uint32_t)kLines * (uint32_t)A.kc * 2u;
  // digits: one 16-byte row of a core matrix per slice and octet
  auto convert = [&](int h) {
    const int ko = octets(h);
    const int em = s_emax[line];
    const bool slow = is_slow(em);
    const int emax = slow ? 0 : em;
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      const int o = part + parts * u;
      if (o < ko) {
        uint32_t w[NS][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const pg::SliceInt f0 = pg::slice_fixed(slow ? 0.0 : val[u][2 * q], emax);
          const pg::SliceInt f1 = pg::slice_fixed(slow ? 0.0 : val[u][2 * q + 1], emax);
#pragma unroll
          for (int i = 0; i < NS; ++i) w[i][q] = pg::slice_digit2(f0, f1, i);
        }
        const uint32_t dst = (uint32_t)((line >> 3) * koct + o) * 128u + (uint32_t)(line & 7) * 16u;
#pragma unroll
        for (int i = 0; i < NS; ++i)
          *reinterpret_cast<uint4*>(smem + (uint32_t)i * a_slice + dst) =
              make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  };
  // One thread: the products of the digits with matrix block b into
  // accumulator set b, once the block has landed.  Digit i of the lines meets
  // digits 0 .. 9 - i of the matrix, which lie one under the other in shared
  // memory as one operand of (10 - i) nc rows, in accumulators i .. 9, which
  // lie side by side: at most 256 columns an instruction (one product at a
  // time reads the lines' digits once for each).
  auto issue = [&](int b, uint32_t parity, int h) {
    if (!wait_for<PG_SLICE_POLLS_ISSUE>(smem_u32(&bar_b[b]), parity)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint64_t dA = smem_desc(sA, lbo, sbo), dB = smem_desc(sB + (uint32_t)b * A.block_bytes, lbo, sbo);
    const uint32_t id0 = (1u << 4) | ((uint32_t)(kLines >> 4) << 24);
    const uint32_t d0 = tmem + (uint32_t)b * (A.tmem_cols >> 1);
    const int steps = octets(h) >> 1;
    for (int kk = 0; kk < steps; ++kk) {
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        const uint64_t da = dA + (((uint32_t)i * a_slice + (uint32_t)kk * 256u) >> 4);
        const int all = (NS - i) * A.nc;
        const uint32_t acc = (h > 0 || kk > 0 || i > 0) ? 1u : 0u;
        mma_f16(d0 + (uint32_t)(i * A.nc), da, dB + (uint32_t)kk * 16u,
                id0 | ((uint32_t)((all < 256 ? all : 256) >> 3) << 17), acc);
        if (kChunks && all > 256)
          mma_f16(d0 + (uint32_t)(i * A.nc + 256), da, dB + (uint32_t)kk * 16u + (((256u >> 3) * sbo) >> 4),
                  id0 | ((uint32_t)((all - 256) >> 3) << 17), acc);
      }
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
        smem_u32(&bar_mma[b])));
    return true;
  };
  // One thread: copies and products that it has issued, `loads` and `products`
  // of them on the barriers of buffer b, are complete.
  auto drain = [&](int b, int loads, int products) {
    if (loads > 0) mbar_wait(smem_u32(&bar_b[b]), (uint32_t)((loads - 1) & 1));
    if (products > 0) mbar_wait(smem_u32(&bar_mma[b]), (uint32_t)((products - 1) & 1));
  };
  // The four outputs of a read-out batch, joined two at a time (the accumulators
  // of all four at once spilled: 64^3 x 4 73 us, so 63): four columns of the
  // thread's own line, or, where lines are contiguous and the batch is
  // transposed, columns of neighbouring lines; addresses p + step[q].
  const bool reads = 32 * (warp & 3) < A.lc;  // this warp's lanes hold lines
  const bool valid = row < lend;
  const long base = first_point(row);
  const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  const int tc = A.tc;
  double* tb = reinterpret_cast<double*>(smem + A.off_t) + warp * 32 * (tc + 1);
  const int nbatch = A.nc >> 2;
  const int tcol = lane & (tc - 1), tline = lane / tc;  // transposed: lane = (line of 32 / tc, column)
  const int rows_t = lend - 32 * (warp & 3) - tline;    // lines from this lane's on
  const long istep = contig ? 1 : A.inner;
  const long pbase = contig ? (l0 + 32 * (warp & 3) + tline) * A.n + tcol : base;
  const long vector0 = base - base % A.npts;  // a line lies within one vector
  const long step1 = !contig ? A.inner : (tc == 4 ? 8L : 16L) * A.n;
  const long step2 = !contig ? 2 * A.inner : (tc == 4 ? 16L * A.n : 2L);
  const long step3 = step1 + step2;
  auto outputs = [&](int i) {  // which of the four exist, column i on
    if (!contig) return valid ? (A.n - i >= 4 ? 15 : (1 << (A.n - i > 0 ? A.n - i : 0)) - 1) : 0;
    if (tc == 4) return i + tcol < A.n ? (rows_t > 0) | (rows_t > 8) << 1 | (rows_t > 16) << 2 | (rows_t > 24) << 3 : 0;
    const int lines = (rows_t > 0) | (rows_t > 16) << 1;
    return (i + tcol < A.n ? lines : 0) | (i + tcol + 2 < A.n ? lines << 2 : 0);
  };
  double dot = 0.0;     // mode 3
  double pa[4], pb[4];  // what the next batch is added to: y, or x and v
  auto prefetch = [&](int i, long p) {
    if ((A.mode != 1 && A.mode != 2) || !reads) return;
    const double* s = (A.mode == 1 ? y : x) + p;
    const int m = outputs(i);
    pa[0] = m & 1 ? s[0] : 0.0;
    pa[1] = m & 2 ? s[step1] : 0.0;
    pa[2] = m & 4 ? s[step2] : 0.0;
    pa[3] = m & 8 ? s[step3] : 0.0;
    if (A.mode == 2) {  // never with contiguous lines
      const double* w = v + (p - vector0);
      pb[0] = m & 1 ? w[0] : 0.0;
      pb[1] = m & 2 ? w[step1] : 0.0;
      pb[2] = m & 4 ? w[step2] : 0.0;
      pb[3] = m & 8 ? w[step3] : 0.0;
    }
  };
  // first column and address of this warp's first batch of N chunk c
  auto first_col = [&](int c) { return c * A.nc + 4 * wpart; };
  auto first_at = [&](int c) { return pbase + (long)first_col(c) * istep; };
  // mma false (the same for the lanes of a warp): without the accumulators
  auto readout = [&](int c, uint32_t tset, bool more, bool mma) {
    if (!reads) return;
    const int em = s_emax[row];
    const bool slow = is_slow(em) || !mma;
    const int emax = slow ? 0 : em;
    int i = first_col(c);
    long p = first_at(c);
    for (int bt = wpart; bt < nbatch && (!kChunks || i < A.n); bt += 4, i += 16, p += 16 * istep) {
      double a0[4], b0[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) a0[q] = pa[q], b0[q] = pb[q];
      if (bt + 4 < nbatch) prefetch(i + 16, p + 16 * istep);
      else if (more) prefetch(first_col(c + 1), first_at(c + 1));
      double k[4];
#pragma unroll
      for (int g = 0; g < 4; g += 2) {
        uint32_t r[pg::kSliceAcc][2];
        if (mma) {
#pragma unroll
          for (int d = 0; d < pg::kSliceAcc; ++d)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
                         : "=r"(r[d][0]), "=r"(r[d][1])
                         : "r"(trow + tset + (uint32_t)(d * A.nc + 4 * bt + g)));
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int d = 0; d < pg::kSliceAcc; ++d)  // the values are read after the wait
          asm volatile("" : "+r"(r[d][0]), "+r"(r[d][1]));
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float a[pg::kSliceAcc];
#pragma unroll
          for (int d = 0; d < pg::kSliceAcc; ++d) a[d] = __uint_as_float(r[d][q]);
          k[g + q] = pg::slice_join(a, A.scale + emax);
        }
      }
      if (slow && valid) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double s = 0.0;
#pragma unroll 1
          for (int b = A.h0 * A.kc; i + q < A.n && b < k_end; ++b)
            s = fma(A64[(i + q) * A.sa + b * A.sb], x[base + b * A.inner], s);
          k[q] = s;
        }
      }
      if (A.mode == 3) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (valid && i + q < A.n) dot = fma(x[base + i + q], k[q], dot);
        continue;
      }
      if (contig) {
        // through the warp's buffer, so that neighbouring lanes write
        // neighbouring values of a line
        if (tc == 4) {
#pragma unroll
          for (int q = 0; q < 4; ++q) tb[lane * 5 + q] = k[q];
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; ++q) k[q] = tb[(8 * q + tline) * 5 + tcol];
          __syncwarp();
        } else {
#pragma unroll
          for (int g = 0; g < 4; g += 2) {
            tb[lane * 3] = k[g];
            tb[lane * 3 + 1] = k[g + 1];
            __syncwarp();
            k[g] = tb[tline * 3 + tcol];
            k[g + 1] = tb[(16 + tline) * 3 + tcol];
            __syncwarp();
          }
        }
      }
      const int m = outputs(i);
      double* out = y + p;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (m >> q & 1) {
          const double w = A.mode == 0 ? k[q] : (A.mode == 1 ? a0[q] + k[q] : fma(b0[q], a0[q], k[q]));
          out[q == 0 ? 0 : (q == 1 ? step1 : (q == 2 ? step2 : step3))] = w;
        }
    }
  };
  bool ok = true;
  if constexpr (!kChunks) {
    if (warp < kST / 32) {
      load_chunk(0);
      chunk_emax();
      named_sync(1, kST);  // the maxima are complete, the staging area is read
      convert(0);
    }
    __syncthreads();
    if (warp < kST / 32) {
      prefetch(first_col(c_first), first_at(c_first));
      for (int c = c_first; c < c_end; ++c) {
        const int b = (c - c_first) & 1;
        if (ok)
          ok = __all_sync(0xffffffffu, wait_for<PG_SLICE_POLLS>(smem_u32(&bar_mma[b]),
                                                               (uint32_t)((c - c_first) >> 1 & 1)));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        __syncwarp();
        readout(c, (uint32_t)b * (A.tmem_cols >> 1), c + 1 < c_end, ok);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        // a warp that has given up is not counted: it may be chunks ahead
        if (ok && lane == 0) mbar_arrive(smem_u32(&bar_read[b]));
      }
    } else if (lane == 0) {
      int loads[2] = {1, c_first + 1 < c_end ? 1 : 0}, products[2] = {0, 0};
      for (int c = c_first; c < c_end && ok; ++c) {
        const int b = (c - c_first) & 1, use = (c - c_first) >> 1;
        if (use > 0) {
          // the matrix block is free once its products are done, the
          // accumulators once they are read
          ok = wait_for<PG_SLICE_POLLS_ISSUE>(smem_u32(&bar_mma[b]), (uint32_t)((use - 1) & 1));
          if (!ok) break;
          load_b(c, 0, b);
          ++loads[b];
          ok = wait_for<PG_SLICE_POLLS_ISSUE>(smem_u32(&bar_read[b]), (uint32_t)((use - 1) & 1));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        ok = issue(b, (uint32_t)(use & 1), 0);
        if (ok) ++products[b];
      }
      for (int b = 0; b < 2; ++b) drain(b, loads[b], products[b]);
    }
  } else {
    for (int h = 0; h < A.nch; ++h) {
      load_chunk(h);
      chunk_emax();
      __syncthreads();
    }
    int turn = 0, loads = 1, products = 0;
    for (int c = c_first; c < c_end; ++c) {
      for (int h = 0; h < A.nch && ok; ++h, ++turn) {
        load_chunk(h);
        __syncthreads();  // the staging area is read
        convert(h);
        __syncthreads();
        if (tid == 0) {
          if (issue(0, (uint32_t)turn & 1u, h)) ++products;
        }
        if (h + 1 == A.nch) prefetch(first_col(c), first_at(c));
        ok = __syncthreads_and(wait_for<PG_SLICE_POLLS>(smem_u32(&bar_mma[0]), (uint32_t)turn & 1u)) != 0;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (tid == 0 && ok && (h + 1 < A.nch || c + 1 < c_end)) {  // the next block while this one is read out
          load_b(h + 1 < A.nch ? c : c + 1, h + 1 < A.nch ? h + 1 : 0, 0);
          ++loads;
        }
      }
      if (!ok) prefetch(first_col(c), first_at(c));
      readout(c, 0u, false, ok);
      // the accumulators are read before products into them
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (tid == 0) drain(0, loads, products);
  }
  if (A.mode == 3) {
    // the four threads of a line, in order
    double* sd = reinterpret_cast<double*>(smem + A.off_t);
    __syncthreads();
    if (warp < kST / 32) sd[wpart * kLines + row] = dot;
    __syncthreads();
    if (wpart == 0 && valid)
      y[A.out0 + (long)blockIdx.y * A.nlines + l0 + row] =
          ((dot + sd[kLines + row]) + sd[2 * kLines + row]) + sd[3 * kLines + row];
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A.tmem_cols));
  }
}

// The digit images of up to nine n x n matrices, one thread per entry of the
// padded image; the images are zero-filled beforehand.
struct SliceBuild {
  const double* A[9];
  unsigned char* img[9];
  int emax[9];  // biased exponent of the matrix's largest value
  int n[9], kc[9], nc[9], nnc[9];
  int trans;    // the images are those of A^T
};
__global__ void k_slice_matrix(const SliceBuild B) {
  const int m = blockIdx.y, n = B.n[m], kc = B.kc[m], nc = B.nc[m];
  const size_t block = (size_t)pg::kSliceN * nc * kc * 2;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * n; e += gridDim.x * blockDim.x) {
    const int i = e / n, k = e - i * n;
    const pg::SliceInt f = pg::slice_fixed(B.A[m][B.trans ? k * n + i : e], B.emax[m]);
    const int c = i / nc, h = k / kc;
    unsigned char* p = B.img[m] + (size_t)(h * B.nnc[m] + c) * block + pg::tc16_kmajor_off(i - c * nc, k - h * kc, kc);
#pragma unroll
    for (int s = 0; s < pg::kSliceN; ++s)
      *reinterpret_cast<unsigned short*>(p + (size_t)s * nc * kc * 2) = (unsigned short)pg::slice_digit2(f, f, s);
  }
}

constexpr int kSmemMost = 226 * 1024;

template <int NU, bool kChunks>
cudaError_t launch_slice(const SliceArgs& a, dim3 grid, size_t smem, const unsigned char* img, const double* A64,
                         const double* v, const double* x, double* y, cudaStream_t st, int device) {
  static std::atomic<unsigned long long> done{0};
  const cudaError_t attr = pg::once_per_device(done, device, [] {
    return cudaFuncSetAttribute(k_slice_axis<NU, kChunks>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
  });
  if (attr != cudaSuccess) return attr;
  return pg::launch_dependent(k_slice_axis<NU, kChunks>, grid, dim3(kST + (kChunks ? 0 : 32)), smem, st, a,
                              img, A64, v, x, y);
}

}  // namespace

namespace pg {

// Up to 64 points: one K chunk, N chunks of 16 (two sets of 10 accumulators in
// 512 columns of tensor memory; the lines' digits and two blocks of the
// matrix's in shared memory).  Longer axes: K chunks and N chunks of at most
// 48 (10 x 48 columns; 169 KB of shared memory), whose products with all K
// chunks of a launch meet in one set of accumulators.
static void slice_shape(int n, SliceMat* S) {
  S->n = n;
  S->nch = n <= 64 ? 1 : (n + 47) / 48;
  S->kc = ((n + S->nch - 1) / S->nch + 15) / 16 * 16;
  const int npad = (n + 15) / 16 * 16;
  const int most = S->nch > 1 ? 48 : 16;
  S->nnc = (npad + most - 1) / most;
  S->nc = ((npad + S->nnc - 1) / S->nnc + 15) / 16 * 16;
}

// Whether a product from slices of this n x n matrix is as exact, value by
// value, as a chain of n multiply-adds may be: entries that are not zero no
// further than r bits below the largest, which the slices round by 2^(r - 26)
// of an FP64 rounding (kSliceGuard bits are to spare), two such roundings (T
// and the line) against n.  The sine DVR keeps to this up to about 750 points.
// big: the largest entry.
static bool slice_exact(const std::vector<double>& t, double* big) {
  // magnitudes compare as integers; the smallest above zero as bits - 1
  uint64_t most = 0, least = ~0ull;
  for (const double& x : t) {
    uint64_t u;
    memcpy(&u, &x, 8);
    u &= 0x7fffffffffffffffull;
    most = std::max(most, u);
    least = std::min(least, u - 1);
  }
  double small;
  memcpy(big, &most, 8);
  if (most >= 0x7ff0000000000000ull) return false;
  if (most == 0) return true;
  ++least;
  memcpy(&small, &least, 8);
  return *big < 1e270 && small > 1e-270 &&
         std::ilogb(*big) - std::ilogb(small) <= kSliceGuard + std::ilogb(sqrt((double)t.size())) - 1;
}

// T, Q^T and Q of the three axes; the host copies give the largest entry
// (|Q| <= 1, scaled as if it reached 1).
pg_status slice_grid(pg_grid* g) {
  SliceBuild B{};
  SliceMat* S[9];
  int share[9], count = 0;
  // an axis with the points and kinetic matrix of one before it has its images too
  int like[3] = {-1, -1, -1};
  double big[3];
  g->t_sliced = true;
  for (int a = 0; a < 3; ++a) {
    for (int b = 0; b < a && like[a] < 0; ++b)
      if (g->n[b] == g->n[a] && like[b] < 0 && g->t[b] == g->t[a]) like[a] = b;
    if (like[a] >= 0) big[a] = big[like[a]];
    else g->t_sliced &= slice_exact(g->t[a], &big[a]);
  }
  g->same_t = like[1] == 0 && like[2] == 0;
  size_t off[9], total = 0;
  for (int m = 0; m < 9; ++m) {
    const int a = m % 3;
    S[m] = m < 3 ? &g->t_sl[a] : (m < 6 ? &g->q_sl[a] : &g->qb_sl[a]);
    slice_shape(g->n[a], S[m]);
    share[m] = like[a] >= 0 ? m - a + like[a] : -1;
    if (share[m] < 0 && m >= 6 && g->dvrtype != 3) share[m] = m - 3;  // the DST-I is symmetric
    while (share[m] >= 0 && share[share[m]] >= 0) share[m] = share[share[m]];
    if (m < 3 && !g->t_sliced) continue;  // no images of T
    off[m] = total;
    if (share[m] < 0) total += ((size_t)S[m]->nch * S[m]->nnc * S[m]->block_bytes() + 255) / 256 * 256;
  }
  PG_TRY(g->sl_img.alloc(total));
  PG_CUDA_TRY(cudaMemsetAsync(g->sl_img.p, 0, total, 0));
  int most = 0;
  for (int m = 0; m < 9; ++m) {
    const int a = m % 3;
    if (m < 3 && !g->t_sliced) continue;
    int ex = 0;
    frexp(m < 3 ? big[a] : 1.0, &ex);  // big < 2^ex, its biased exponent ex + 1022
    S[m]->tau = kSliceN * kSliceP - 1 - ex;
    S[m]->img = g->sl_img.p + (share[m] < 0 ? off[m] : off[share[m]]);
    if (share[m] >= 0) continue;
    B.A[count] = m < 3 ? g->t_dev[a].p : (m < 6 ? g->q_dev[a].p : g->qb_dev[a].p);
    B.img[count] = g->sl_img.p + off[m];
    B.emax[count] = ex + 1022;
    B.n[count] = S[m]->n;
    B.kc[count] = S[m]->kc;
    B.nc[count] = S[m]->nc;
    B.nnc[count] = S[m]->nnc;
    most = std::max(most, S[m]->n);
    ++count;
  }
  const int blocks = (most * most + 255) / 256;
  k_slice_matrix<<<dim3((unsigned)blocks, (unsigned)count), 256, 0, 0>>>(B);
  PG_TRY(check_launch("k_slice_matrix"));
  PG_CUDA_TRY(cudaStreamSynchronize(0));  // the grid may be used on any stream
  return PG_OK;
}

int sm_count(int device) {
  static std::atomic<int> known[64];
  int n = 0;
  const bool slot = device >= 0 && device < 64;
  if (slot && (n = known[device].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) return 152;
  if (slot) known[device].store(n, std::memory_order_relaxed);
  return n;
}

namespace {

// Launches the contraction of nlines lines (stride inner); mode 3 writes
// *rows rows of nlines partial dots.
pg_status slice_launch(long nlines, long inner, long npts, const SliceMat& S, const double* A64, bool trans,
                       const double* v, const double* x, double* y, int mode, int* rows, cudaStream_t st, int device) {
  SliceArgs a{};
  a.n = S.n;
  a.inner = inner;
  a.npts = npts;
  a.nlines = nlines;
  a.plain = S.plain;
  a.kc = S.kc;
  a.nnc = S.nnc;
  a.nc = S.nc;
  a.sa = trans ? 1 : S.n;
  a.sb = trans ? S.n : 1;
  a.scale = kSliceUnit - kSliceGuard - S.tau - 1075;
  // lines whose products stay normal numbers with this matrix (slice_join)
  a.exp_lo = std::max(2, -1022 - a.scale);
  a.exp_hi = std::min(2046, 1023 - kSliceBits - a.scale);
  a.block_bytes = (uint32_t)S.block_bytes();
  const bool chunks = S.nch > 1;
  a.off_b = (uint32_t)(kSliceN * kLines * S.kc * 2);
  const size_t images = a.off_b + (size_t)(chunks ? 1 : 2) * a.block_bytes;
  // with K chunks the digits are made again for every N chunk: the transpose
  // buffer may take their place
  a.tc = chunks || images + kTransMost <= (size_t)kSmemMost ? 4 : 2;
  a.off_t = chunks ? 0u : (uint32_t)images;
  const size_t smem = images + (chunks ? 0 : (size_t)(kST / 32) * 32 * (a.tc + 1) * 8);
  a.tmem_cols = 32;
  while (a.tmem_cols < (uint32_t)(kSliceAcc * S.nc)) a.tmem_cols <<= 1;
  if (!chunks) a.tmem_cols <<= 1;  // two sets
  // Few lines: the N chunks of a tile go to CTAs of their own, then fewer lines
  // to a CTA, as long as there is an SM for each.  In this order: a CTA's
  // read-out takes as long for 32 lines as for 128 (TMEM lanes belong to one
  // scheduler's warps), its digits do not (64^3 x 1: 44 us with the lines
  // first, 34 so; 80^3 x 1 62 / 48, 160x60x60 x 1 91 / 63).
  const long full = (nlines + kLines - 1) / kLines;
  const int sms = sm_count(device);
  const int groups = (int)std::max<long>(1, std::min<long>(S.nnc, sms / full));
  a.nc_per = (S.nnc + groups - 1) / groups;
  const int split = (S.nnc + a.nc_per - 1) / a.nc_per;
  a.lc = kLines;
  while (a.lc > 32 && (nlines + a.lc / 2 - 1) / (a.lc / 2) * split <= sms) a.lc /= 2;
  const long tiles = (nlines + a.lc - 1) / a.lc;
  const dim3 grid((unsigned)tiles, (unsigned)split);
  // at most kSliceK values (two K chunks) per launch, so that the sums of one
  // accumulator stay below 2^24; a longer axis adds up in Y
  int launches = 0;
  for (int h0 = 0; h0 < S.nch; h0 += 2, ++launches) {
    a.h0 = h0;
    a.nch = std::min(2, S.nch - h0);
    a.mode = h0 == 0 || mode == 3 ? mode : 1;
    a.out0 = (long)launches * split * nlines;
    cudaError_t e;
    if (chunks) e = launch_slice<2, true>(a, grid, smem, S.img, A64, v, x, y, st, device);
    else if (S.kc <= 32) e = launch_slice<1, false>(a, grid, smem, S.img, A64, v, x, y, st, device);
    else e = launch_slice<2, false>(a, grid, smem, S.img, A64, v, x, y, st, device);
    PG_CUDA_TRY(e);
    PG_TRY(check_launch("k_slice_axis"));
  }
  if (rows) *rows = launches * split;
  return PG_OK;
}

}  // namespace

pg_status slice_axis(const pg_grid* g, int axis, const SliceMat& S, const double* A64, const double* v,
                     const double* x, double* y, int nvec, int mode, cudaStream_t st) {
  PG_ARG(S.img && S.n == g->n[axis], "slice_axis: no operand images");
  const long inner = axis == 0 ? 1 : (axis == 1 ? g->n[0] : (long)g->n[0] * g->n[1]);
  return slice_launch(g->N / S.n * nvec, inner, g->N, S, A64, false, v, x, y, mode, nullptr, st, g->device);
}

int slice_row_count(int n) {
  SliceMat S;
  slice_shape(n, &S);
  return (S.nch + 1) / 2 * S.nnc;
}

size_t slice_rows_shape(int n, double big, double low, SliceMat* S) {
  slice_shape(n, S);
  S->plain = !std::isfinite(big) || (big != 0 && (big > 1e270 || low < 1e-270 || low < std::ldexp(big, -20)));
  int ex = 0;
  if (!S->plain) frexp(big, &ex);
  S->tau = kSliceN * kSliceP - 1 - ex;
  return (size_t)S->nch * S->nnc * S->block_bytes();
}

pg_status slice_rows_matrix(const double* A64, unsigned char* img, SliceMat* S, cudaStream_t st) {
  PG_CUDA_TRY(cudaMemsetAsync(img, 0, (size_t)S->nch * S->nnc * S->block_bytes(), st));
  SliceBuild B{};
  B.A[0] = A64;
  B.img[0] = img;
  B.emax[0] = kSliceN * kSliceP - 1 - S->tau + 1022;
  B.n[0] = S->n;
  B.kc[0] = S->kc;
  B.nc[0] = S->nc;
  B.nnc[0] = S->nnc;
  B.trans = 1;
  S->img = img;
  k_slice_matrix<<<dim3((unsigned)std::min(4096, (S->n * S->n + 255) / 256), 1), 256, 0, st>>>(B);
  return check_launch("k_slice_matrix");
}

pg_status slice_rows(const pg_grid* g, long nlines, const SliceMat& S, const double* A64, const double* x, double* y,
                     SliceRows mode, int* rows, cudaStream_t st) {
  return slice_launch(nlines, 1, nlines * S.n, S, A64, true, nullptr, x, y, mode, rows, st, g->device);
}

}  // namespace pg
