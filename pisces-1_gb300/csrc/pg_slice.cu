// One axis contraction Y (+)= A x_axis X in FP64 on the tensor cores, from
// exact FP16 slices of both operands (pg_slice.cuh); the H*X product and the
// kinetic preconditioner of the FP64 form are three and six of these.
//
// Grid lines along the axis are the rows of the left operand: a CTA takes
// 128 of them, converts their values to digit images once (each line scaled
// by its own largest exponent), and multiplies them with the matrix's digit
// images, which the bulk copy engine fetches from L2.  The tensor core's
// accumulators (7 x nc columns of TMEM) are read back one line per lane.
//
// Bounds: per point and axis about 35 integer operations to make the digits,
// 60 to join the accumulators and one or two FP64 operations (V X, the sum
// into Y), against n FP64 multiply-adds before; the FP64 pipe is about 60
// times slower than the integer pipes here.
#include <algorithm>
#include <cmath>

#include "pg_slice.cuh"
#include "pg_tc16.cuh"

namespace {

constexpr int kLines = 128;  // MMA M
constexpr int kST = 512;     // threads: four per line
constexpr int kTransPitch = 5;
constexpr int kTransBytes = (kST / 32) * 32 * kTransPitch * 8;  // 32 lines x 4 columns per warp

// A line whose largest exponent lies outside [kExpLo, kExpHi] (subnormal or
// huge values, infinities, NaN) is multiplied with FP64 multiply-adds instead.
constexpr int kExpLo = 200, kExpHi = 1900;

struct SliceArgs {
  long nlines;   // lines of all vectors
  long inner;    // stride of the axis
  long npts;     // points of one vector (index of V)
  int n, kc, nnc, nc;
  int h0, nch;   // K chunks [h0, h0 + nch) of this launch
  int plain;     // every line by FP64 multiply-adds
  int rebuild;   // more than one K chunk per axis: the digit images are rebuilt for every N chunk
  int nc_per;    // N chunks per CTA (blockIdx.y takes the next ones)
  int scale;     // exponent of accumulator 6: kSliceUnit - tau - 1075 - kSliceGuard
  uint32_t block_bytes;  // one (K, N) block of the matrix image
  uint32_t slice_b;      // bytes of one slice in it
  uint32_t off_b, off_t; // shared-memory offsets of the matrix block and the transpose buffer
  uint32_t tmem_cols;
  int mode;              // 0: y = K, 1: y += K, 2: y = v x + K, 3: row dots x . K
  long out0;             // mode 3: first output row of this launch, in values
  long sa, sb;           // strides of A64 (output, input index)
};

template <int NU>
__global__ void __launch_bounds__(kST, 1)
    k_slice_axis(const SliceArgs A, const unsigned char* __restrict__ img, const double* __restrict__ A64,
                 const double* __restrict__ v, const double* __restrict__ x, double* y, int* __restrict__ err) {
  constexpr int NS = pg::kSliceN;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar_b, bar_mma;
  __shared__ uint32_t tmem_base;
  __shared__ int s_emax[kLines];
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int line = tid & (kLines - 1), part = tid >> 7;
  const int c_first = blockIdx.y * A.nc_per;
  const int c_end = c_first + A.nc_per < A.nnc ? c_first + A.nc_per : A.nnc;
  const uint32_t sA = smem_u32(smem), sB = sA + A.off_b;

  auto load_b = [&](int c, int h) {  // one thread: block (h, c) of the matrix image
    uint64_t state;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 %0, [%1], %2;"
                 : "=l"(state)
                 : "r"(smem_u32(&bar_b)), "r"(A.block_bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sB),
                 "l"(img + (size_t)((A.h0 + h) * A.nnc + c) * A.block_bytes), "r"(A.block_bytes), "r"(smem_u32(&bar_b))
                 : "memory");
  };
  if (tid == 0) {
    s_fail = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_b)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_mma)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    load_b(c_first, 0);  // constant data: before the kernel ahead has finished
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

  const long l0 = blockIdx.x * (long)kLines;
  const bool contig = A.inner == 1;
  const bool valid = l0 + line < A.nlines;
  const long base = [&] {  // first point of this thread's line
    const long l = valid ? l0 + line : 0;
    return contig ? l * A.n : (l / A.inner) * A.inner * A.n + l % A.inner;
  }();
  const int koct = A.kc >> 3;
  const int k_end = (A.h0 + A.nch) * A.kc < A.n ? (A.h0 + A.nch) * A.kc : A.n;

  double val[NU][8];
  // this thread's octets (part, part + 4, ...) of K chunk h
  auto load_chunk = [&](int h) {
    const int k0 = (A.h0 + h) * A.kc;
    const int kn = A.n - k0 < A.kc ? A.n - k0 : A.kc;
    if (contig) {
      // the lines are contiguous: coalesced through shared memory (the digit
      // images' place), odd pitch
      double* raw = reinterpret_cast<double*>(smem);
      const int pitch = A.kc | 1;
      const long lend = A.nlines - l0 < kLines ? A.nlines - l0 : kLines;
      for (int r = warp; r < kLines; r += kST / 32)
        for (int k = lane; k < A.kc; k += 32) {
          const bool in = r < lend && k < kn;
          const double* src = x + (in ? (l0 + r) * A.n + k0 + k : 0);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(sA + 8u * (uint32_t)(r * pitch + k)),
                       "l"(src), "r"(in ? 8 : 0)
                       : "memory");
        }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int o = part + 4 * u;
#pragma unroll
        for (int q = 0; q < 8; ++q) val[u][q] = o < koct ? raw[line * pitch + 8 * o + q] : 0.0;
      }
    } else {
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int o = part + 4 * u;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int k = 8 * o + q;
          val[u][q] = (valid && o < koct && k < kn) ? x[base + (long)(k0 + k) * A.inner] : 0.0;
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

  // The four outputs of a read-out batch are y[p + q step], q < cnt: four
  // columns of the thread's own line, or, where lines are contiguous and the
  // batch is transposed, one column of four lines.
  struct Out {
    long p;
    int cnt;
  };
  const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  double* tb = reinterpret_cast<double*>(smem + A.off_t) + warp * 32 * kTransPitch;
  const int nbatch = A.nc >> 2;
  const long lt = l0 + 32 * (warp & 3) + (lane >> 2);
  const long ostep = contig ? 8L * A.n : A.inner;
  const int rows_left = lt < A.nlines ? (int)((A.nlines - lt + 7) / 8 < 4 ? (A.nlines - lt + 7) / 8 : 4) : 0;
  auto out_of = [&](int c, int bt) {
    Out o;
    const int i = c * A.nc + 4 * bt;
    if (contig) {
      o.p = lt * A.n + i + (lane & 3);
      o.cnt = i + (lane & 3) < A.n ? rows_left : 0;
    } else {
      o.p = base + i * A.inner;
      o.cnt = valid ? (A.n - i < 4 ? A.n - i : 4) : 0;
    }
    return o;
  };
  double dot = 0.0;     // mode 3
  double pa[4], pb[4];  // what the next batch is added to: y, or x and v
  auto prefetch = [&](const Out& o) {
    const double* s = A.mode == 1 ? y : x;
    if (A.mode == 1 || A.mode == 2) {
#pragma unroll
      for (int q = 0; q < 4; ++q) pa[q] = q < o.cnt ? s[o.p + q * ostep] : 0.0;
    }
    if (A.mode == 2) {
      const long pv = o.p % A.npts;  // a line lies within one vector
#pragma unroll
      for (int q = 0; q < 4; ++q) pb[q] = q < o.cnt ? v[pv + q * ostep] : 0.0;
    }
  };

  bool ok = true;
  int waits_b = 0, waits_m = 0;
  int emax = 0;
  bool slow = false;
  auto settle = [&] {  // after the line maxima are complete
    emax = s_emax[line];
    slow = A.plain || (emax != 0 && (emax < kExpLo || emax > kExpHi));
    if (slow) emax = 0;
  };
  if (A.nch > 1) {
    for (int h = 0; h < A.nch; ++h) {
      load_chunk(h);
      chunk_emax();
      __syncthreads();
    }
    settle();
  }
  const uint32_t lbo = 128, sbo = (uint32_t)koct * 128u;
  const uint32_t a_slice = (uint32_t)kLines * (uint32_t)A.kc * 2u;
  for (int c = c_first; c < c_end && ok; ++c) {
    for (int h = 0; h < A.nch && ok; ++h) {
      if (A.rebuild || c == c_first) {
        load_chunk(h);
        if (A.nch == 1) chunk_emax();
        __syncthreads();  // the staging area is read; with one chunk also the maxima
        if (A.nch == 1) settle();
        // digits: one 16-byte row of a core matrix per slice and octet
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          const int o = part + 4 * u;
          if (o < koct) {
            uint32_t w[NS][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const unsigned long long f0 = pg::slice_fixed(slow ? 0.0 : val[u][2 * q], emax);
              const unsigned long long f1 = pg::slice_fixed(slow ? 0.0 : val[u][2 * q + 1], emax);
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
      }
      __syncthreads();
      if (tid == 0) {
        if (mbar_wait(smem_u32(&bar_b), (uint32_t)(waits_b & 1))) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // digit i of the lines against digits 0 .. 6 - i of the matrix,
          // which lie one under the other in shared memory as one operand of
          // (7 - i) nc rows, into accumulators i .. 6, which lie side by side:
          // at most 256 columns an instruction (one product at a time read
          // the lines' digits 28 times instead of 10: 7700 cycles a tile
          // of 64 x 64 against 6600)
          for (int kk = 0; kk < (koct >> 1); ++kk) {
#pragma unroll
            for (int i = 0; i < NS; ++i) {
              const uint64_t da = smem_desc(sA + (uint32_t)i * a_slice + (uint32_t)kk * 256u, lbo, sbo);
              for (int c0 = 0; c0 < (NS - i) * A.nc; c0 += 256) {
                const int cols = (NS - i) * A.nc - c0 < 256 ? (NS - i) * A.nc - c0 : 256;
                const uint32_t idesc =
                    (1u << 4) | ((uint32_t)(cols >> 3) << 17) | ((uint32_t)(kLines >> 4) << 24);
                mma_f16(tmem + (uint32_t)(i * A.nc + c0), da,
                        smem_desc(sB + (uint32_t)(c0 >> 3) * sbo + (uint32_t)kk * 256u, lbo, sbo), idesc,
                        (h > 0 || kk > 0 || i > 0) ? 1u : 0u);
              }
            }
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_u32(&bar_mma)));
        } else {
          s_fail = 1;
          mbar_arrive(smem_u32(&bar_mma));  // nothing was issued: release the others
        }
      }
      ++waits_b;
      if (h + 1 == A.nch) prefetch(out_of(c, part));
      ok = __syncthreads_and(mbar_wait(smem_u32(&bar_mma), (uint32_t)(waits_m & 1)) && !*(volatile int*)&s_fail) != 0;
      ++waits_m;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tid == 0 && ok) {  // the next block while this one is read out
        if (h + 1 < A.nch) load_b(c, h + 1);
        else if (c + 1 < c_end) load_b(c + 1, 0);
      }
    }
    if (!ok) {
      if (tid == 0) atomicExch(err, 1);
      break;
    }
    // read-out: this thread's line (its TMEM lane), four columns at a time
    for (int bt = part; bt < nbatch; bt += 4) {
      uint32_t r[pg::kSliceAcc][4];
#pragma unroll
      for (int d = 0; d < pg::kSliceAcc; ++d)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[d][0]), "=r"(r[d][1]), "=r"(r[d][2]), "=r"(r[d][3])
                     : "r"(trow + (uint32_t)(d * A.nc + 4 * bt)));
      double a0[4], b0[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) a0[q] = pa[q], b0[q] = pb[q];
      const Out o = out_of(c, bt);
      if (bt + 4 < nbatch) prefetch(out_of(c, bt + 4));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int d = 0; d < pg::kSliceAcc; ++d)  // the values are read after the wait
        asm volatile("" : "+r"(r[d][0]), "+r"(r[d][1]), "+r"(r[d][2]), "+r"(r[d][3]));
      double k[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float a[pg::kSliceAcc];
#pragma unroll
        for (int d = 0; d < pg::kSliceAcc; ++d) a[d] = __uint_as_float(r[d][q]);
        k[q] = pg::slice_join(a, A.scale + emax);
      }
      if (slow && valid) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = c * A.nc + 4 * bt + q;
          double s = 0.0;
#pragma unroll 1
          for (int b = A.h0 * A.kc; i < A.n && b < k_end; ++b) s = fma(A64[i * A.sa + b * A.sb], x[base + b * A.inner], s);
          k[q] = s;
        }
      }
      if (A.mode == 3) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = c * A.nc + 4 * bt + q;
          if (valid && i < A.n) dot = fma(x[base + i], k[q], dot);
        }
        continue;
      }
      if (contig) {
        // 32 lines x 4 columns through the warp's buffer, so that four lanes
        // write one line's 32 bytes
#pragma unroll
        for (int q = 0; q < 4; ++q) tb[lane * kTransPitch + q] = k[q];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) k[q] = tb[(8 * q + (lane >> 2)) * kTransPitch + (lane & 3)];
        __syncwarp();
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q < o.cnt) {
          double* p = y + o.p + q * ostep;
          if (A.mode == 0) *p = k[q];
          else if (A.mode == 1) *p = a0[q] + k[q];
          else *p = fma(b0[q], a0[q], k[q]);
        }
    }
    // the accumulators are read before the next chunk's products
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (A.mode == 3) {
    // the four threads of a line, in order
    double* sd = reinterpret_cast<double*>(smem + A.off_t);
    __syncthreads();
    sd[part * kLines + line] = dot;
    __syncthreads();
    if (part == 0 && valid)
      y[A.out0 + (long)blockIdx.y * A.nlines + l0 + line] =
          ((dot + sd[kLines + line]) + sd[2 * kLines + line]) + sd[3 * kLines + line];
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
    const unsigned long long f = pg::slice_fixed(B.A[m][B.trans ? k * n + i : e], B.emax[m]);
    const int c = i / nc, h = k / kc;
    unsigned char* p = B.img[m] + (size_t)(h * B.nnc[m] + c) * block + pg::tc16_kmajor_off(i - c * nc, k - h * kc, kc);
#pragma unroll
    for (int s = 0; s < pg::kSliceN; ++s)
      *reinterpret_cast<unsigned short*>(p + (size_t)s * nc * kc * 2) = (unsigned short)pg::slice_digit2(f, f, s);
  }
}

template <int NU>
cudaError_t launch_slice(const SliceArgs& a, dim3 grid, size_t smem, const unsigned char* img, const double* A64,
                         const double* v, const double* x, double* y, int* err, cudaStream_t st) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(k_slice_axis<NU>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
  if (attr != cudaSuccess) return attr;
  return pg::launch_dependent(k_slice_axis<NU>, grid, dim3(kST), smem, st, a, img, A64, v, x, y, err);
}

}  // namespace

namespace pg {

static void slice_shape(int n, SliceMat* S) {
  S->n = n;
  // K chunks of at most 80: 128 lines' digits and 64 matrix rows' fit shared memory
  S->nch = (n + 79) / 80;
  S->kc = ((n + S->nch - 1) / S->nch + 15) / 16 * 16;
  const int npad = (n + 15) / 16 * 16;
  S->nnc = (npad + 63) / 64;  // 7 accumulators of at most 64 columns in TMEM
  S->nc = ((npad + S->nnc - 1) / S->nnc + 15) / 16 * 16;
}

// T, Q^T and Q of the three axes; the host copies give the largest entry
// (|Q| <= 1, scaled as if it reached 1).
pg_status slice_grid(pg_grid* g) {
  SliceBuild B{};
  SliceMat* S[9];
  int share[9], count = 0;
  size_t off[9], total = 0;
  for (int m = 0; m < 9; ++m) {
    const int a = m % 3;
    S[m] = m < 3 ? &g->t_sl[a] : (m < 6 ? &g->q_sl[a] : &g->qb_sl[a]);
    slice_shape(g->n[a], S[m]);
    // an axis with the points and kinetic matrix of one before it has its images too
    share[m] = -1;
    for (int b = 0; b < a && share[m] < 0; ++b)
      if (g->n[b] == g->n[a] && g->t[b] == g->t[a]) share[m] = m - a + b;
    if (share[m] < 0 && m >= 6 && g->dvrtype != 3) share[m] = m - 3;  // the DST-I is symmetric
    while (share[m] >= 0 && share[share[m]] >= 0) share[m] = share[share[m]];
    off[m] = total;
    if (share[m] < 0) total += ((size_t)S[m]->nch * S[m]->nnc * S[m]->block_bytes() + 255) / 256 * 256;
  }
  PG_TRY(g->sl_img.alloc(total));
  PG_CUDA_TRY(cudaMemsetAsync(g->sl_img.p, 0, total, 0));
  int most = 0;
  for (int m = 0; m < 9; ++m) {
    const int a = m % 3;
    double big = 1.0;
    if (m < 3) {
      big = 0;
      for (double t : g->t[a]) big = std::max(big, fabs(t));
    }
    int ex = 0;
    frexp(big, &ex);  // big < 2^ex, its biased exponent ex + 1022
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

namespace {

// Launches the contraction of nlines lines (stride inner); mode 3 writes
// *rows rows of nlines partial dots.
pg_status slice_launch(long nlines, long inner, long npts, const SliceMat& S, const double* A64, bool trans,
                       const double* v, const double* x, double* y, int mode, int* rows, int* err, cudaStream_t st) {
  SliceArgs a{};
  a.n = S.n;
  a.inner = inner;
  a.npts = npts;
  a.nlines = nlines;
  a.plain = S.plain;
  a.rebuild = S.nch > 1;
  a.kc = S.kc;
  a.nnc = S.nnc;
  a.nc = S.nc;
  a.sa = trans ? 1 : S.n;
  a.sb = trans ? S.n : 1;
  a.scale = kSliceUnit - kSliceGuard - S.tau - 1075;
  a.block_bytes = (uint32_t)S.block_bytes();
  a.slice_b = (uint32_t)(S.nc * S.kc * 2);
  const uint32_t abytes = (uint32_t)(kSliceN * kLines * S.kc * 2);
  a.off_b = abytes;
  // with several K chunks the digit images are rebuilt for every N chunk, so
  // the transpose buffer may take their place
  a.off_t = S.nch > 1 ? 0u : abytes + a.block_bytes;
  const size_t smem = abytes + a.block_bytes + (S.nch > 1 ? 0 : kTransBytes);
  a.tmem_cols = 32;
  while (a.tmem_cols < (uint32_t)(kSliceAcc * S.nc)) a.tmem_cols <<= 1;
  const long tiles = (a.nlines + kLines - 1) / kLines;
  // few tiles: the N chunks of a tile go to CTAs of their own
  const int split = tiles * S.nnc <= 152 ? S.nnc : 1;
  a.nc_per = (S.nnc + split - 1) / split;
  const dim3 grid((unsigned)tiles, (unsigned)split);
  // at most two K chunks (160 values) per launch, so that the sums of one
  // accumulator stay below 2^24; a longer axis adds up in Y
  int launches = 0;
  for (int h0 = 0; h0 < S.nch; h0 += 2, ++launches) {
    a.h0 = h0;
    a.nch = std::min(2, S.nch - h0);
    a.mode = h0 == 0 || mode == 3 ? mode : 1;
    a.out0 = (long)launches * split * nlines;
    cudaError_t e;
    if (S.kc <= 32) e = launch_slice<1>(a, grid, smem, S.img, A64, v, x, y, err, st);
    else if (S.kc <= 64) e = launch_slice<2>(a, grid, smem, S.img, A64, v, x, y, err, st);
    else e = launch_slice<3>(a, grid, smem, S.img, A64, v, x, y, err, st);
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
  return slice_launch(g->N / S.n * nvec, inner, g->N, S, A64, false, v, x, y, mode, nullptr, g->tc_err.p, st);
}

int slice_row_count(int n) {
  SliceMat S;
  slice_shape(n, &S);
  return (S.nch + 1) / 2 * S.nnc;
}

size_t slice_rows_shape(int n, double big, SliceMat* S) {
  slice_shape(n, S);
  S->plain = !std::isfinite(big) || big > 1e200 || (big != 0 && big < 1e-200);
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

pg_status slice_rows(long nlines, const SliceMat& S, const double* A64, const double* x, double* y, SliceRows mode,
                     int* rows, int* err, cudaStream_t st) {
  return slice_launch(nlines, 1, nlines * S.n, S, A64, true, nullptr, x, y, mode, rows, err, st);
}

}  // namespace pg
