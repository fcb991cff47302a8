// tlr_oz.cu -- FP64 products of the complex128 factorisation on the tensor
// cores: the Schur updates F22 -= L21 U12 of the fronts and the products by the
// inverses of the diagonal blocks that rewrite the finished factor, by exact
// integer slices (the splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms
// 59 (2012); tcgen05 has no FP64 kind, and GB300's FP64 pipe runs at about 1.1
// TFLOP/s).
//
// For an update C -= A B (A = L21, B = U12) every operand entry becomes a
// 56-bit fixed-point number relative to its row's (A) or column's (B) largest
// entry, written as seven signed base-256 digits d_0 (top) .. d_6, each exact in
// bfloat16 (the rewrite: 64 bits, eight digits).  The product of
// slice s of A and slice t of B has weight 256^-(s + t); all products of
// one weight class g = s + t accumulate in one FP32 TMEM accumulator.  They
// are exact: at most 8 pairs x 64 real terms x 2^14 < 2^24.  Classes 0 .. 7
// are kept (34 of the 49 pairs, 36 of 64; class 8 starts at 2^-64 of the largest
// product), summed as 64-bit integers, and enter F22 with one FP64 FMA, i.e.
// one rounding instead of one per term.  Pivot rows of very different scale
// would waste bits (a small entry of A meets a large row of B), so row k of B is
// first scaled by the power of two of its largest entry and column k of A by the
// inverse.  L' = L inv(L_cc) takes the largest entries of L's columns instead: of
// rows scaled by d, L has entries like d_i / d_k and the inverse like d_k / d_j,
// whose diagonal of ones says nothing about d.  D_b = inv(U_bb) inv(L_bb) has no
// such scaling for rows and columns of any scale and stays in FP64, as do the
// products by blocks of fewer than 32 columns, whose FP64 chains are short and
// round less.
//
// An entry far below the largest of its line keeps fewer bits than FP64 would, and a
// product of such entries alone loses by it.  A factor does not: pivoting bounds the
// multipliers, and a line's largest products carry the rounding of either kind.
// Backward errors of solves in extended precision, sliced / FMA: grids of 30 x 18 to
// 130 x 60 points 0.37 to 0.91 normwise (0.33 to 1.28 by rows), pencils of order 25 to
// 600 0.81 to 1.24, with entries spread over 2 to 16 decades without structure 0.70 to
// 1.26 (by rows 0.66 to 1.44), with rows or columns over 6 and 12 decades 0.67 to 1.92.
//
// Complex products as in tlr_tc.cu: A = [Lr | Li] (128 rows), B = [Ur; -Ui]
// and [Ui; Ur] (32 + 32 "rows"), K chunks of 8 complex columns = 16 real =
// one MMA step of kind::f16.
#include <algorithm>
#include <cstdint>

#include "tlr_async.cuh"
#include "tlr_complex.cuh"
#include "tlr_internal.h"
#include "tlr_lu.h"

namespace tlr {
namespace {

constexpr int kM = 128, kN = 32;          // complex tile
constexpr int kK = kOzPanel;              // panel columns (complex)
constexpr int kChunks = kK / 8;
constexpr int kClasses = 8;               // weight classes
constexpr int kAStep = 128 * 32, kBStep = 64 * 32;  // bytes of one slice, one chunk
constexpr int kSmem = 226 * 1024;                   // dynamic shared memory at most
constexpr int kThreads = 320;
constexpr int kExpNone = -(1 << 20);

// unbiased exponent of the larger part; kExpNone for zero, 1024 when not finite
__device__ __forceinline__ int exp_of(double2 v) {
  const int a = (__double2hiint(v.x) >> 20) & 0x7ff, b = (__double2hiint(v.y) >> 20) & 0x7ff;
  const int e = max(a, b);
  return e == 0 ? kExpNone : e - 1023;  // subnormals count as zero
}

// v 2^(BITS - e) rounded to an integer (|v| < 2^(e + 1)); zero below its last bit
template <int BITS>
__device__ __forceinline__ long long fixed_of(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int x = (int)((b >> 52) & 0x7ff);
  if (x == 0) return 0;
  const long long mant = (b & 0xfffffffffffffll) | (1ll << 52);
  const int sh = x - 1023 - 52 + BITS - e;  // mant 2^sh, sh <= BITS - 52
  long long r;
  if (sh >= 0)
    r = mant << sh;
  else if (sh > -55)
    r = (mant + (1ll << (-sh - 1))) >> -sh;
  else
    r = 0;
  return b < 0 ? -r : r;
}

// the lowest signed base-256 digit; x is left with the rest
__device__ __forceinline__ int take_digit(long long &x) {
  const int d = (int)(signed char)(x & 0xff);
  x = (x - d) >> 8;
  return d;
}

__device__ __forceinline__ uint32_t bf16_pair(int a, int b) {  // exact for |a|, |b| <= 256
  return (__float_as_uint((float)a) >> 16) | (__float_as_uint((float)b) & 0xffff0000u);
}

__device__ __forceinline__ int find_front(const int *__restrict__ prefix, int nf, int t) {
  int lo = 0, hi = nf;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (prefix[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// One product: C (rows x cols) from A (rows x kw) and B (kw x cols), kw <= kK,
// all column-major.
struct View {
  const double2 *a, *b;
  double2 *c;
  int lda, ldb, ldc, rows, cols, kw;
  bool by_a;  // k scaled by the columns of A, else by the rows of B
};

// The products of a launch: panel step s of a level's fronts (C -= A B), or the
// rewrite of the factor (C = A B, later passes C += A B).  kS: slices.  The
// rewrite has no large C to round into, and seven slices (54 bits below the
// largest entry) would lose up to 1.5 times as much as FP64 FMAs there.
struct PanelStep {
  static constexpr bool kUpdate = true;
  static constexpr int kS = 7;
  const int *fl;
  const DevFront *fr;
  double2 *pool;
  int s, w;
  __device__ __forceinline__ View view(int q) const {
    const DevFront f = fr[fl[q]];
    const int k0 = s * w, ww = min(w, f.p - k0), base = k0 + ww;
    double2 *F = pool + f.off;
    return {F + (long long)k0 * f.m + base, F + (long long)base * f.m + k0,
            F + (long long)base * f.m + base, f.m, f.m, f.m, f.m - base, f.m - base, ww, false};
  }
};

struct Rewrite {
  static constexpr bool kUpdate = false;
  static constexpr int kS = 8;
  const OzJob *jobs;
  double2 *pool;
  const double2 *linv, *uinv;
  __device__ __forceinline__ View view(int q) const {
    const OzJob j = jobs[q];
    return {(j.kind ? uinv : pool) + j.a, (j.kind ? pool : linv) + j.b, pool + j.c, j.lda, j.ldb,
            j.ldc, j.rows, j.cols, j.kw, j.kind == 0};
  }
};

template <class S>
struct Size {
  static constexpr int kAImg = kChunks * S::kS * kAStep;  // 114688 for seven slices
  static constexpr int kBChunk = S::kS * kBStep;          // 14336
  static constexpr int kBImg = kChunks * kBChunk;         // 57344
  static constexpr int kStages = (kSmem - kAImg) / kBChunk;  // ring of B chunks: 8 (8 slices: 6)
};

// rexp[q kK + k] = largest exponent of row k of B (lane = row, a warp per
// column) or of column k of A (lane = row) of product q; the caller has set it
// below every exponent
template <class S>
__global__ void __launch_bounds__(256) k_oz_rowexp(S src, int *__restrict__ rexp) {
  const View v = src.view(blockIdx.y);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  if (v.by_a) {
    for (int k = wp; k < v.kw; k += 8) {
      int e = kExpNone;
      for (int r = blockIdx.x * 32 + lane; r < v.rows; r += gridDim.x * 32) {
        const int x = exp_of(v.a[(long long)k * v.lda + r]);
        if (x < 1024) e = max(e, x);
      }
      e = __reduce_max_sync(0xffffffffu, e);
      if (lane == 0 && e > kExpNone) atomicMax(rexp + blockIdx.y * kK + k, e);
    }
    return;
  }
  int e = kExpNone;
  for (int c = blockIdx.x * 8 + wp; c < v.cols; c += gridDim.x * 8)
    if (lane < v.kw) {
      const int x = exp_of(v.b[(long long)c * v.ldb + lane]);
      if (x < 1024) e = max(e, x);
    }
  if (lane < v.kw && e > kExpNone) atomicMax(rexp + blockIdx.y * kK + lane, e);
}

// Operand images of the products of one launch.  Grid atiles + btiles: an A
// tile is 128 rows of A, a B tile 32 columns of B.  Image: [chunk][slice][row groups
// of 8][two 8 x 16-byte core matrices]; scale[row or column]: the power of two
// of its fixed-point numbers (NaN when an entry is not finite).
template <class S>
__global__ void __launch_bounds__(256)
    k_oz_split(S src, const int *__restrict__ pa, const int *__restrict__ pb, int nf,
               const int *__restrict__ rexp, unsigned char *__restrict__ img_a, unsigned char *__restrict__ img_b,
               double *__restrict__ scale_a, double *__restrict__ scale_b, int atiles) {
  constexpr int kS = S::kS, kAImg = Size<S>::kAImg, kBImg = Size<S>::kBImg;
  __shared__ int smax[256];
  __shared__ int re[kK];
  const int tid = threadIdx.x;
  const bool is_a = (int)blockIdx.x < atiles;
  const int t = is_a ? blockIdx.x : blockIdx.x - atiles;
  const int lo = find_front(is_a ? pa : pb, nf, t);
  const View v = src.view(lo);
  const double2 *M = is_a ? v.a : v.b;
  const long long ldl = is_a ? 1 : v.ldb, ldk = is_a ? v.lda : 1;  // a line's, a k's distance
  const int nl = is_a ? v.rows : v.cols;
  if (tid < kK) {
    const int e = max(rexp[lo * kK + tid], -1100);  // an empty row or column: any scale
    re[tid] = v.by_a ? -e : e;
  }
  __syncthreads();
  // thread: one line (A row / B column) and its chunks
  const int lines = is_a ? kM : kN;
  const int line = tid % lines, part = tid / lines;  // A: 2 parts of 2 chunks, B: 4 of 1
  const int cpp = is_a ? kChunks / 2 : 1;
  const bool act = is_a || part < kChunks;
  const int g = (t - (is_a ? pa[lo] : pb[lo])) * lines + line;
  auto entry = [&](int k) {  // scaled exponents aside
    if (!act || g >= nl || k >= v.kw) return make_double2(0.0, 0.0);
    return M[g * ldl + k * ldk];
  };
  int e = kExpNone;
  bool bad = false;
  if (act)
    for (int k = part * cpp * 8; k < (part + 1) * cpp * 8; ++k) {
      const int x = exp_of(entry(k));
      bad |= x >= 1024;
      if (x > kExpNone) e = max(e, is_a ? x + re[k] : x - re[k]);
    }
  smax[tid] = bad ? 1 << 20 : e;
  __syncthreads();
  e = smax[line];
  for (int q = 1; q < (is_a ? 2 : kChunks); ++q) e = max(e, smax[line + q * lines]);
  bad = e >= 1 << 20;
  if (act && part == 0) {
    double *sc = is_a ? scale_a + (long long)t * kM : scale_b + (long long)t * kN;
    sc[line] = bad ? nan("") : e == kExpNone ? 0.0 : scalbn(1.0, e - 27);
  }
  if (!act) return;
  if (bad || e == kExpNone) e = 1 << 14;  // every fixed-point number is zero
  for (int c = part * cpp; c < (part + 1) * cpp; ++c) {
    long long xr[8], xi[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = 8 * c + j;
      const double2 x = entry(k);
      const int ek = is_a ? e - re[k] : e + re[k];
      xr[j] = fixed_of<8 * kS - 2>(x.x, ek);
      xi[j] = fixed_of<8 * kS - 2>(x.y, ek);
    }
    unsigned char *im = is_a ? img_a + (long long)t * kAImg + c * kS * kAStep
                             : img_b + (long long)t * kBImg + c * kS * kBStep;
#pragma unroll
    for (int sl = kS - 1; sl >= 0; --sl) {
      int dr[8], di[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // the top slice takes what is left: |x| <= 2^(8 kS - 1) leaves at most 2^7
        dr[j] = sl ? take_digit(xr[j]) : (int)xr[j];
        di[j] = sl ? take_digit(xi[j]) : (int)xi[j];
      }
      const uint4 r4 = make_uint4(bf16_pair(dr[0], dr[1]), bf16_pair(dr[2], dr[3]),
                                  bf16_pair(dr[4], dr[5]), bf16_pair(dr[6], dr[7]));
      const uint4 i4 = make_uint4(bf16_pair(di[0], di[1]), bf16_pair(di[2], di[3]),
                                  bf16_pair(di[4], di[5]), bf16_pair(di[6], di[7]));
      auto at = [](int row) { return (row >> 3) * 256 + (row & 7) * 16; };
      if (is_a) {
        unsigned char *p = im + sl * kAStep + at(line);
        *reinterpret_cast<uint4 *>(p) = r4;
        *reinterpret_cast<uint4 *>(p + 128) = i4;
      } else {
        const uint4 n4 = make_uint4(i4.x ^ 0x80008000u, i4.y ^ 0x80008000u, i4.z ^ 0x80008000u,
                                    i4.w ^ 0x80008000u);  // sign flips: exact
        unsigned char *p = im + sl * kBStep + at(line), *q = im + sl * kBStep + at(kN + line);
        *reinterpret_cast<uint4 *>(p) = r4;        // Cr: [Ur ; -Ui]
        *reinterpret_cast<uint4 *>(p + 128) = n4;
        *reinterpret_cast<uint4 *>(q) = i4;        // Ci: [Ui ; Ur]
        *reinterpret_cast<uint4 *>(q + 128) = r4;
      }
    }
  }
}

__device__ __forceinline__ uint64_t desc(uint32_t saddr) {  // K-major, LBO 128, SBO 256
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128u >> 4) << 16) |
         ((uint64_t)(256u >> 4) << 32) | (1ull << 46);
}

// kind::f16: D f32, A and B bf16, K-major, M = 128, N = 64
constexpr uint32_t kIdescBf16 = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) |
                                ((128u >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(kIdescBf16), "r"(acc));
}

__device__ __forceinline__ void commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_addr(bar))
               : "memory");
}

#define TLR_OZ_LD8(taddr, r)                                                                    \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"        \
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),        \
                 "=r"(r[6]), "=r"(r[7])                                                         \
               : "r"(taddr))

// The eight class sums of 8 accumulator columns at `col` as integers of
// weight 2^-42 of class 0 (at most 2^62): classes 6 and 7 are rounded in.
__device__ __forceinline__ void class_sums(uint32_t taddr, long long (&v)[8]) {
  uint32_t r[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0;
#pragma unroll
  for (int g = 0; g < 6; ++g) {
    TLR_OZ_LD8(taddr + 64 * g, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j)
      v[j] = (v[j] << 8) + __float2int_rn(__uint_as_float(r[j]));
  }
  int lowc[8];
  TLR_OZ_LD8(taddr + 64 * 6, r);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) lowc[j] = __float2int_rn(__uint_as_float(r[j]));
  TLR_OZ_LD8(taddr + 64 * 7, r);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c7 = __float2int_rn(__uint_as_float(r[j]));
    v[j] = (v[j] << 2) + ((lowc[j] * 256 + c7 + 8192) >> 14);
  }
}

// Persistent, warp-specialised: each CTA takes a contiguous range of the
// tiles [tbase, tbase + tiles) (column tiles of one row tile in a row, so the 112
// KB A image stays in shared memory and only the 56 KB B images stream, through
// a ring of 8-column chunks).
//   warp 8 (one thread): bulk copies; warp 9 (one thread): the 136 (eight
//   slices: 144) MMAs of a tile into eight 64-column accumulators (all 512 TMEM columns);
//   warps 0..7: read the accumulators into 64-bit integers, release TMEM, and
//   update C in FP64 while the next tile's MMAs run.  Warp w owns rows
//   32 (w % 4) + lane and columns 16 (w / 4) .. +15.
// The eight accumulators fill TMEM, so the MMAs of a tile start when the last
// one's class sums have been read: at 100 x 50 (the largest updates, 696 us) the
// tensor pipe is active 48% of the time, the FP64 pipe of the epilogue (two
// conversions and two FMAs per entry) 55%, DRAM is 31% busy; the rewrite (188 us):
// 47%, 52%, 17 to 28%.  32-column panels keep the A image resident and the class
// sums exact with every pair kept.  Measured against the CUDA-core FP64 kernel
// (a 64 x 64 tile is 524 K FMAs, 125 us on an SM): complex128 factorisation
// 123 -> 55 ms at 60 x 32, 1191 -> 272 ms at 150 x 64 with the updates here, 42
// and 188 ms with the rewrite here too (its CUDA-core kernels took 102 of the
// 272 ms; with faster panels 32 and 167 ms now).  Waits are bounded as in
// tlr_tc.cu.
template <class S>
__global__ void __launch_bounds__(kThreads, 1)
    k_oz_gemm(S src, const int *__restrict__ prefix, const int *__restrict__ pa,
              const int *__restrict__ pb, int nf, int tbase, int tiles, bool add, const unsigned char *__restrict__ img_a, const unsigned char *__restrict__ img_b,
              const double *__restrict__ scale_a, const double *__restrict__ scale_b,
              int *__restrict__ err) {
  extern __shared__ __align__(1024) unsigned char oz_smem[];
  constexpr int kS = S::kS, kAImg = Size<S>::kAImg, kBImg = Size<S>::kBImg;
  constexpr int kBChunk = Size<S>::kBChunk, kStages = Size<S>::kStages;
  __shared__ __align__(8) uint64_t afull, aempty, bfull[kStages], bempty[kStages], tfull, tempty;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ int issued_a, issued_b, used_a, used_b, committed_b, committed_t;
  unsigned char *sa = oz_smem, *sb = oz_smem + kAImg;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    mbar_init(&afull, 1);
    mbar_init(&aempty, 1);
    for (int q = 0; q < kStages; ++q) {
      mbar_init(&bfull[q], 1);
      mbar_init(&bempty[q], 1);
    }
    mbar_init(&tfull, 1);
    mbar_init(&tempty, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    issued_a = issued_b = used_a = used_b = committed_b = committed_t = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const int t0 = tbase + (int)((long long)tiles * blockIdx.x / gridDim.x);
  const int t1 = tbase + (int)((long long)tiles * (blockIdx.x + 1) / gridDim.x);

  struct Tile {
    double2 *C;  // its first entry
    int ld, nr, nc, at, bt;  // leading dimension, rows and columns left, image indices
  };
  auto decode = [&](int t) {
    Tile d;
    const int lo = find_front(prefix, nf, t);
    const View v = src.view(lo);
    const int ntc = (v.cols + kN - 1) / kN;
    const int lt = t - prefix[lo];
    const int rt = lt / ntc, ct = lt - rt * ntc;
    d.C = v.c + (long long)ct * kN * v.ldc + rt * kM;
    d.ld = v.ldc;
    d.nr = v.rows - rt * kM;
    d.nc = v.cols - ct * kN;
    d.at = pa[lo] + rt;
    d.bt = pb[lo] + ct;
    return d;
  };
  auto wait_bar = [&](uint64_t *bar, uint32_t parity) -> bool {
    for (unsigned it = 0; it < kWaitLimit; ++it) {
      if (mbar_test(bar, parity)) return true;
      if (abort_flag) return false;
    }
    abort_flag = 1;
    atomicExch(err, 1);
    return false;
  };

  if (warp == 8) {
    if (lane == 0) {  // copies
      int na = 0, nb = 0, cur = -1;  // nb: chunks of B
      for (int t = t0; t < t1 && !abort_flag; ++t) {
        const Tile d = decode(t);
        if (d.at != cur) {  // a new row tile: once the MMAs of the old one are done
          if (na > 0 && !wait_bar(&aempty, (na - 1) & 1)) break;
          mbar_expect_tx(&afull, kAImg);
          bulk_g2s(sa, img_a + (long long)d.at * kAImg, kAImg, &afull);
          cur = d.at;
          ++na;
        }
        for (int c = 0; c < kChunks; ++c, ++nb) {
          const int g = nb % kStages;
          if (nb >= kStages && !wait_bar(&bempty[g], (nb / kStages - 1) & 1)) break;
          mbar_expect_tx(&bfull[g], kBChunk);
          bulk_g2s(sb + g * kBChunk, img_b + (long long)d.bt * kBImg + c * kBChunk, kBChunk,
                   &bfull[g]);
        }
      }
      issued_a = na;
      issued_b = nb;
    }
  } else if (warp == 9) {
    if (lane == 0) {  // MMAs
      int na = 0, nb = 0, cur = -1, ti = 0;
      bool fine = true;
      for (int t = t0; t < t1 && fine && !abort_flag; ++t) {
        const Tile d = decode(t);
        if (d.at != cur) {
          if (!wait_bar(&afull, na & 1)) break;
          cur = d.at;
          ++na;
        }
        if (ti >= 1 && !wait_bar(&tempty, (ti - 1) & 1)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = smem_addr(sa);
        for (int c = 0; c < kChunks; ++c, ++nb) {
          const int st = nb % kStages;
          fine = wait_bar(&bfull[st], (nb / kStages) & 1);
          if (!fine) break;
          const uint32_t ac = a0 + c * kS * kAStep, bc = smem_addr(sb) + st * kBChunk;
#pragma unroll
          for (int g = 0; g < kClasses; ++g)
#pragma unroll
            for (int sl = 0; sl < kS; ++sl) {
              const int tl = g - sl;
              if (tl < 0 || tl >= kS) continue;
              const bool first = sl == (g < kS ? 0 : g - kS + 1);
              mma_bf16(tmem + 64 * g, desc(ac + sl * kAStep), desc(bc + tl * kBStep),
                       c == 0 && first ? 0u : 1u);
            }
          commit(&bempty[st]);
        }
        if (!fine) break;
        commit(&tfull);
        ++ti;
        // the next tile has another row tile: this commit frees A
        if (t + 1 < t1 && decode(t + 1).at != cur) commit(&aempty);
      }
      committed_b = nb;
      committed_t = ti;
      used_a = na;
      used_b = nb;
    }
  } else {
    const int q4 = warp & 3, h2 = warp >> 2;
    const int row = 32 * q4 + lane;
    int ti = 0;
    for (int t = t0; t < t1; ++t, ++ti) {
      const Tile d = decode(t);
      const bool row_ok = row < d.nr;
      const double sr = scale_a[(long long)d.at * kM + row];
      bool ok = true;
      if (lane == 0) ok = wait_bar(&tfull, ti & 1);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t base = tmem + ((uint32_t)(32 * q4) << 16) + 16 * h2;
      long long vr[16], vi[16];
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        long long x[8];
        class_sums(base + 8 * part, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) vr[8 * part + j] = x[j];
        class_sums(base + 32 + 8 * part, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) vi[8 * part + j] = x[j];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&tempty))
                     : "memory");
      const double *scb = scale_b + (long long)d.bt * kN + 16 * h2;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2 f22[8];
        double2 *p = d.C + (long long)(16 * h2 + 8 * h) * d.ld + row;
        const int nc = row_ok ? d.nc - (16 * h2 + 8 * h) : 0;  // columns left
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < nc) f22[j] = S::kUpdate || add ? p[(long long)j * d.ld] : make_double2(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < nc) {
            const double sc = S::kUpdate ? -sr * scb[8 * h + j] : sr * scb[8 * h + j];
            f22[j].x = fma((double)vr[8 * h + j], sc, f22[j].x);
            f22[j].y = fma((double)vi[8 * h + j], sc, f22[j].y);
            p[(long long)j * d.ld] = f22[j];
          }
      }
    }
  }
  __syncthreads();
  if (tid == 0 && abort_flag) {
    // let the copies and MMAs already issued land before TMEM is released
    for (int g = used_a; g < issued_a; ++g) mbar_wait(&afull, g & 1);
    for (int g = used_b; g < issued_b; ++g) mbar_wait(&bfull[g % kStages], (g / kStages) & 1);
    if (committed_b > 0)
      mbar_wait(&bempty[(committed_b - 1) % kStages], ((committed_b - 1) / kStages) & 1);
    if (committed_t > 0) mbar_wait(&tfull, (committed_t - 1) & 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

struct Images {
  unsigned char *a, *b;
  double *sa, *sb;
};

template <class S>
Images images(unsigned char *planes, int atiles, int btiles) {
  Images im;
  im.a = planes;
  im.b = planes + (size_t)atiles * Size<S>::kAImg;
  im.sa = reinterpret_cast<double *>(im.b + (size_t)btiles * Size<S>::kBImg);
  im.sb = im.sa + (size_t)atiles * kM;
  return im;
}

template <class S>
size_t image_bytes(size_t atiles, size_t btiles) {
  return atiles * (Size<S>::kAImg + kM * sizeof(double)) +
         btiles * (Size<S>::kBImg + kN * sizeof(double));
}

template <class S>
int split_images(tlr_ctx *ctx, S src, const int *pa, const int *pb, int nf, int max_len,
                 int atiles, int btiles, const Images &im, int *rexp, cudaStream_t st) {
  TLR_CUDA(ctx, cudaMemsetAsync(rexp, 0x80, sizeof(int) * kK * nf, st));
  { k_oz_rowexp<S><<<dim3(std::min(64, blocks_for(max_len, 32)), nf), 256, 0, st>>>(src,
                                                                                     rexp); count_launches(); }
  { k_oz_split<S><<<atiles + btiles, 256, 0, st>>>(src, pa, pb, nf, rexp, im.a, im.b, im.sa, im.sb,
                                                   atiles); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

template <class S>
int gemm(tlr_ctx *ctx, S src, const int *prefix, const int *pa, const int *pb, int nf, int tbase,
         int tiles, bool add, const Images &im, int *err, cudaStream_t st) {
  if (tiles <= 0) return TLR_OK;
  const int smem = Size<S>::kAImg + Size<S>::kStages * Size<S>::kBChunk;
  TLR_CUDA(ctx,
           cudaFuncSetAttribute(k_oz_gemm<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int grid = std::max(1, std::min(tiles, std::max(sms, 1)));
  { k_oz_gemm<S><<<grid, kThreads, smem, st>>>(src, prefix, pa, pb, nf, tbase, tiles, add, im.a,
                                               im.b, im.sa, im.sb, err); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

}  // namespace

size_t oz_update_bytes(size_t atiles, size_t btiles) {
  return image_bytes<PanelStep>(atiles, btiles);
}
size_t oz_rewrite_bytes(size_t atiles, size_t btiles) {
  return image_bytes<Rewrite>(atiles, btiles);
}

int launch_gemm_oz(tlr_ctx *ctx, const int *fl, const int *prefix, const int *pa, const int *pb,
                   int nf, int s, int w, int max_ext, double2 *pool, const DevFront *fr, int tiles,
                   int atiles, int btiles, unsigned char *planes, int *rexp, int *err,
                   cudaStream_t st) {
  if (tiles <= 0) return TLR_OK;
  const PanelStep src{fl, fr, pool, s, w};
  const Images im = images<PanelStep>(planes, atiles, btiles);
  int rc = split_images(ctx, src, pa, pb, nf, max_ext, atiles, btiles, im, rexp, st);
  if (!rc) rc = gemm(ctx, src, prefix, pa, pb, nf, 0, tiles, true, im, err, st);
  return rc;
}

int launch_rewrite_oz(tlr_ctx *ctx, const OzBatch &b, const OzJob *jobs, const int *prefix,
                      double2 *pool, const double2 *linv, const double2 *uinv,
                      unsigned char *planes, int *rexp, int *err, cudaStream_t st) {
  const Rewrite src{jobs + b.job_off, pool, linv, uinv};
  const int *pt = prefix + b.prefix_off, *pa = pt + b.jobs + 1, *pb = pa + b.jobs + 1;
  const Images im = images<Rewrite>(planes, b.atiles, b.btiles);
  int rc = split_images(ctx, src, pa, pb, b.jobs, b.max_len, b.atiles, b.btiles, im, rexp, st);
  for (int q = 0; q < kOzPasses && !rc; ++q)
    rc = gemm(ctx, src, pt, pa, pb, b.jobs, b.pass[q], b.pass[q + 1] - b.pass[q], q > 0, im, err,
              st);
  return rc;
}

}  // namespace tlr
