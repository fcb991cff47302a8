// tlr_kvec.cu -- Krylov basis primitives: block inner products, basis
// updates, basis combinations, scaling and axpy on complex128 vectors.
//
// These replace what SLEPc does inside EPSSolve with BLAS (EigenSolver.cpp:72:
// classical Gram-Schmidt against the basis, Ritz vectors V Y, thick-restart
// bases V Q).  Everything runs on the context stream and leaves its results in
// device memory, so an Arnoldi step needs no host round trip: the Gram-Schmidt
// coefficients, ||w|| and the next basis vector w / ||w|| are all formed on the
// device, and the host reads the projected matrix once per restart.
//
// The basis V is column-major (vector q at V + q * ldv).  Every kernel is bound
// by HBM: each reads each basis vector it touches once.  Inner products are
// reduced in a fixed order (per-CTA partials, summed in CTA order by the CTA
// that finishes last), so results are bitwise reproducible.
#include <algorithm>

#include "tlr_complex.cuh"
#include "tlr_ff.cuh"
#include "tlr_internal.h"

namespace tlr {
namespace {

constexpr int kThreads = 256;
// result vectors per CTA of a basis combination: FP64 FMAs bound it (four per
// 16 bytes and result), so few results per CTA and more CTAs; 16 of them left
// 38 CTAs at 60 x 32 (95 us per restart)
constexpr int kChunk = 4;

// conj(v) * w
__device__ __forceinline__ double2 cdotc(double2 acc, double2 v, double2 w) {
  acc.x = fma(v.x, w.x, acc.x);
  acc.x = fma(v.y, w.y, acc.x);
  acc.y = fma(v.x, w.y, acc.y);
  acc.y = fma(-v.y, w.x, acc.y);
  return acc;
}

constexpr int kDotCols = 8;  // basis vectors per CTA of the inner products

__device__ __forceinline__ double2 shfl_xor2(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// whether this CTA is the last of `total` to arrive at the counter (which it
// then clears for the next launch); the others' global writes are visible
__device__ __forceinline__ bool last_arrival(int *ctr, int total) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ctr, 1) == total - 1;
    if (last) *ctr = 0;
    __threadfence();
  }
  __syncthreads();
  return last != 0;
}

// h[k] = sum_i conj(V_k[i]) w[i] for k = blockIdx.y * kDotCols + (0 ..
// kDotCols-1) < nk: this CTA's rows, then the partial sums of all CTAs of the
// column group in CTA order.  FP64 issue bounds the products (four FMAs per
// 16 bytes of basis); a warp folds its eight sums by halving (nine exchanges
// of a pair instead of forty).
__global__ void __launch_bounds__(kThreads)
    k_dot(long long n, const double2 *__restrict__ V, long long ldv, int nk,
          const double2 *__restrict__ w, double2 *__restrict__ part, int ldp,
          double2 *__restrict__ h, int *__restrict__ ctr) {
  __shared__ double2 red[kThreads / 32][kDotCols];
  const int k0 = blockIdx.y * kDotCols;
  const int kc = min(kDotCols, nk - k0);
  double2 acc[kDotCols];
#pragma unroll
  for (int q = 0; q < kDotCols; ++q) acc[q] = make_double2(0.0, 0.0);
  const double2 *Vb = V + (long long)k0 * ldv;
  for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < n;
       i += (long long)gridDim.x * kThreads) {
    const double2 wi = w[i];
    double2 v[kDotCols];
#pragma unroll
    for (int q = 0; q < kDotCols; ++q) v[q] = Vb[min(q, kc - 1) * ldv + i];
#pragma unroll
    for (int q = 0; q < kDotCols; ++q)
      if (q < kc) acc[q] = cdotc(acc[q], v[q], wi);
  }
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  // halving: after the steps of 16, 8 and 4 lanes, lane l holds column
  // 4 (l >> 4 & 1) + 2 (l >> 3 & 1) + (l >> 2 & 1) summed over eight lanes
#pragma unroll
  for (int o = 16, c = kDotCols / 2; c > 0; o >>= 1, c >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < c; ++q) {
      const double2 send = up ? acc[q] : acc[q + c];
      const double2 keep = up ? acc[q + c] : acc[q];
      acc[q] = cadd(keep, shfl_xor2(send, o));
    }
  }
  acc[0] = cadd(acc[0], shfl_xor2(acc[0], 2));
  acc[0] = cadd(acc[0], shfl_xor2(acc[0], 1));
  if ((lane & 3) == 0) red[wp][(lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1)] = acc[0];
  __syncthreads();
  if (threadIdx.x < kc) {
    double2 s = make_double2(0.0, 0.0);
#pragma unroll
    for (int p = 0; p < kThreads / 32; ++p) s = cadd(s, red[p][threadIdx.x]);
    part[(long long)blockIdx.x * ldp + k0 + threadIdx.x] = s;
  }
  if (!last_arrival(ctr + blockIdx.y, gridDim.x)) return;
  // warp q sums column q over the CTAs
  if (wp < kc) {
    double2 s = make_double2(0.0, 0.0);
    for (int b = lane; b < (int)gridDim.x; b += 32)
      s = cadd(s, __ldcg(part + (long long)b * ldp + k0 + wp));
    for (int o = 16; o > 0; o >>= 1) s = cadd(s, shfl_xor2(s, o));
    if (lane == 0) h[k0 + wp] = s;
  }
}

// Column j of the projected matrix = the two Gram-Schmidt passes and beta,
// then g1 = H h and g2 = H g1(0 : j+1), the combinations the pipelined
// applications need (OP V h = V g1; OP V g1 = V g2 + g1(j+1) OP v_{j+1}).
// Run by one CTA, four lanes per row; sh: 2 (j + 2) values.
__device__ void projected_column(const KvColumn &c, double beta, double2 *sh) {
  const int m = c.j + 2;  // rows of the column
  double2 *gs = sh + m;
  for (int i = threadIdx.x; i < c.ldh; i += kThreads) {
    double2 v = make_double2(0.0, 0.0);
    if (i <= c.j) {
      v = cadd(c.h1[i], c.h2[i]);
      sh[i] = v;
    } else if (i == c.j + 1) {
      v.x = beta;
    }
    c.H[(long long)c.j * c.ldh + i] = v;
  }
  __syncthreads();
  const int part = threadIdx.x & 3;
  for (int pass = 0; pass < 2; ++pass) {
    const double2 *x = pass ? gs : sh;
    for (int r0 = 0; r0 < m; r0 += kThreads / 4) {
      const int i = r0 + threadIdx.x / 4;
      double2 acc = make_double2(0.0, 0.0);
      if (i < m)
#pragma unroll 4
        for (int q = part; q <= c.j; q += 4) acc = cfma(acc, c.H[(long long)q * c.ldh + i], x[q]);
      acc = cadd(acc, shfl_xor2(acc, 1));
      acc = cadd(acc, shfl_xor2(acc, 2));
      if (part == 0 && i < m) {
        if (!pass) gs[i] = acc;
        c.g[pass * c.ldh + i] = ff_split(acc);
      }
    }
    __syncthreads();
  }
}

// w[i] -= sum_k V_k[i] h[k]; with npart, also *norm = ||w|| of the result
// (per-CTA partial sums, added in CTA order by the last CTA) and, with a
// column, the projected matrix's new column.
__global__ void __launch_bounds__(kThreads)
    k_update(long long n, const double2 *__restrict__ V, long long ldv, int nk,
             const double2 *__restrict__ h, double2 *__restrict__ w, double *__restrict__ npart,
             double *__restrict__ norm, int *__restrict__ ctr, KvColumn column) {
  extern __shared__ double2 hs[];
  __shared__ double red[kThreads / 32];
  for (int k = threadIdx.x; k < nk; k += kThreads) hs[k] = h[k];
  __syncthreads();
  double s2 = 0.0;
  for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < n;
       i += (long long)gridDim.x * kThreads) {
    double2 acc = w[i];
    const double2 *Vi = V + i;
    int k = 0;
    for (; k + 4 <= nk; k += 4) {  // four independent loads in flight
      const double2 v0 = Vi[(long long)k * ldv], v1 = Vi[(long long)(k + 1) * ldv];
      const double2 v2 = Vi[(long long)(k + 2) * ldv], v3 = Vi[(long long)(k + 3) * ldv];
      acc = cfms(acc, v0, hs[k]);
      acc = cfms(acc, v1, hs[k + 1]);
      acc = cfms(acc, v2, hs[k + 2]);
      acc = cfms(acc, v3, hs[k + 3]);
    }
    for (; k < nk; ++k) acc = cfms(acc, Vi[(long long)k * ldv], hs[k]);
    w[i] = acc;
    s2 = fma(acc.x, acc.x, s2);
    s2 = fma(acc.y, acc.y, s2);
  }
  if (!npart) return;
  for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int p = 0; p < kThreads / 32; ++p) t += red[p];
    npart[blockIdx.x] = t;
  }
  if (!last_arrival(ctr, gridDim.x)) return;
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) s += __ldcg(npart + b);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) {
      red[0] = sqrt(s);
      *norm = red[0];
    }
  }
  __syncthreads();
  if (column.H) projected_column(column, red[0], hs);
}

// out[:, j] = sum_q V[:, q] Y(q, j) for j in this CTA's chunk of kChunk
// columns; Y column-major with leading dimension ldy.
__global__ void __launch_bounds__(kThreads)
    k_combine(long long n, const double2 *__restrict__ V, long long ldv, int nq,
              const double2 *__restrict__ Y, int ldy, int nl, double2 *__restrict__ out,
              long long ldo) {
  extern __shared__ double2 ys[];  // [nq][kChunk]
  const int j0 = blockIdx.y * kChunk;
  const int jc = min(kChunk, nl - j0);
  for (int x = threadIdx.x; x < nq * kChunk; x += kThreads) {
    const int q = x / kChunk, jj = x % kChunk;
    ys[x] = jj < jc ? Y[(long long)(j0 + jj) * ldy + q] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < n;
       i += (long long)gridDim.x * kThreads) {
    double2 acc[kChunk];
#pragma unroll
    for (int jj = 0; jj < kChunk; ++jj) acc[jj] = make_double2(0.0, 0.0);
    for (int q = 0; q < nq; ++q) {
      const double2 v = V[(long long)q * ldv + i];
#pragma unroll
      for (int jj = 0; jj < kChunk; ++jj) acc[jj] = cfma(acc[jj], v, ys[q * kChunk + jj]);
    }
#pragma unroll
    for (int jj = 0; jj < kChunk; ++jj)
      if (jj < jc) out[(long long)(j0 + jj) * ldo + i] = acc[jj];
  }
}

// dst = src * s / *dnorm (dnorm may be null: dst = src * s).  A zero or
// non-finite norm writes zeros; the host sees that norm and reports the
// breakdown.
__global__ void k_scale(long long n, const double2 *src, const double *dnorm, double s,
                        double2 *dst) {  // src and dst may be the same vector
  double f = s;
  if (dnorm) {
    const double d = *dnorm;
    f = (d > 0.0 && d < INFINITY) ? s / d : 0.0;
  }
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double2 v = src[i];
    dst[i] = make_double2(v.x * f, v.y * f);
  }
}

__global__ void k_axpy(long long n, double2 a, const double2 *__restrict__ x,
                       double2 *__restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = cfma(y[i], a, x[i]);
}

int row_blocks(tlr_ctx *ctx, long long n) {
  return (int)std::max<long long>(1, std::min<long long>(ctx->partial_blocks,
                                                         (n + kThreads - 1) / kThreads));
}

}  // namespace

int arrival_counters(tlr_ctx *ctx, int count) {
  if (ctx->kv_ctr && ctx->kv_ctr_n >= count) return TLR_OK;
  TLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  cudaFree(ctx->kv_ctr);
  ctx->kv_ctr = nullptr;
  const int cap = std::max(count, 64);
  TLR_CUDA(ctx, dev_malloc(&ctx->kv_ctr, sizeof(int) * cap));
  TLR_CUDA(ctx, cudaMemsetAsync(ctx->kv_ctr, 0, sizeof(int) * cap, ctx->stream));
  ctx->kv_ctr_n = cap;
  return TLR_OK;
}

int pinned_words(tlr_ctx *ctx) {
  if (!ctx->pin)
    TLR_CUDA(ctx, pin_malloc(&ctx->pin, sizeof(double) * kPinWords));
  return TLR_OK;
}

int kv_dot(tlr_ctx *ctx, long long n, const double2 *V, long long ldv, int nk,
           const double2 *w, double2 *part, double2 *h) {
  if (nk <= 0) return TLR_OK;
  const int nb = row_blocks(ctx, n);
  const dim3 grid(nb, (nk + kDotCols - 1) / kDotCols);
  if (const int rc = arrival_counters(ctx, (int)grid.y)) return rc;
  { k_dot<<<grid, kThreads, 0, ctx->stream>>>(n, V, ldv, nk, w, part, nk, h, ctx->kv_ctr); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int kv_update(tlr_ctx *ctx, long long n, const double2 *V, long long ldv, int nk,
              const double2 *h, double2 *w, double *npart, double *norm, const KvColumn *column) {
  const int nb = row_blocks(ctx, n);
  if (const int rc = arrival_counters(ctx, 1)) return rc;
  const KvColumn c = column ? *column : KvColumn{};
  // 3072 vectors are the most that the update takes (48 KB of coefficients); the
  // column's two stages are as long as this basis, whatever the largest one so far
  if (nk > 3072)
    return fail(ctx, TLR_ERR_CUDA, "Gram-Schmidt takes at most 3072 basis vectors");
  const size_t sm = sizeof(double2) * std::max({nk, 1, column ? 2 * (c.j + 2) : 0});
  if (sm > 47 * 1024) TLR_CUDA(ctx, allow_dynamic_smem(k_update));
  { k_update<<<nb, kThreads, sm, ctx->stream>>>(n, V, ldv, nk, h, w, norm ? npart : nullptr, norm,
                                                ctx->kv_ctr, c); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int kv_combine(tlr_ctx *ctx, long long n, const double2 *V, long long ldv, int nq,
               const double2 *Y, int ldy, int nl, double2 *out, long long ldo) {
  if (nl <= 0) return TLR_OK;
  const int nb = row_blocks(ctx, n);
  const dim3 grid(nb, (nl + kChunk - 1) / kChunk);
  const size_t sm = (size_t)nq * kChunk * sizeof(double2);
  if (sm > 48 * 1024) {
    // more than 768 basis vectors: the shared-memory stage needs opting in
    TLR_CUDA(ctx, allow_dynamic_smem(k_combine));
  }
  { k_combine<<<grid, kThreads, sm, ctx->stream>>>(n, V, ldv, nq, Y, ldy, nl, out, ldo); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int kv_scale(tlr_ctx *ctx, long long n, const double2 *src, const double *dnorm, double s,
             double2 *dst) {
  const int nb = row_blocks(ctx, n);
  { k_scale<<<nb, kThreads, 0, ctx->stream>>>(n, src, dnorm, s, dst); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int kv_axpy(tlr_ctx *ctx, long long n, double2 a, const double2 *x, double2 *y) {
  const int nb = row_blocks(ctx, n);
  { k_axpy<<<nb, kThreads, 0, ctx->stream>>>(n, a, x, y); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

}  // namespace tlr
