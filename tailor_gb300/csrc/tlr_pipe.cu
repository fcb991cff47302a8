// tlr_pipe.cu -- kernels of the pipelined refined applications (tlr_pipe.h).
//
// No counterpart in the reference: PCLU applies MUMPS's FP64 factor once per
// application (EigenSolver.cpp:61-71).
#include <algorithm>

#include "tlr_complex.cuh"
#include "tlr_ff.cuh"
#include "tlr_pipe.h"

namespace tlr {
namespace {

// The element-wise kernels own whole grid nodes (five unknowns), because
// they end in a product with the block-diagonal B: 51 nodes per CTA.
constexpr int kNodes = 51, kRows = 5 * kNodes, kThreads = 256;
constexpr int kWarpRows = 8;  // block rows (warps) per CTA of the A products

__device__ __forceinline__ double2 block_row(const double2 *__restrict__ Bb, const double2 *s) {
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < 5; ++q) acc = cfma(acc, Bb[q], s[q]);
  return acc;
}

// Targets of x and y and the right-hand side of u, for this thread's row:
// tx = b + sigma B x, ty = B x + sigma B y, u's right-hand side B y.
__device__ __forceinline__ void targets(long long i, const double2 *__restrict__ Bb,
                                        const double2 *xs, const double2 *ys, double2 b,
                                        double2 sg, double2 *__restrict__ tx,
                                        double2 *__restrict__ ty, float2 *__restrict__ by32) {
  const double2 bx = block_row(Bb, xs), by = block_row(Bb, ys);
  tx[i] = cfma(b, sg, bx);
  ty[i] = cfma(bx, sg, by);
  by32[i] = make_float2((float)by.x, (float)by.y);
}

// this CTA's sum of |b|^2
__device__ __forceinline__ void block_sum_sq(double s, double *out) {
  __shared__ double red[kThreads / 32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int p = 0; p < kThreads / 32; ++p) t += red[p];
    *out = t;
  }
}

__global__ void __launch_bounds__(kThreads)
    k_pipe_start(long long n, const double2 *__restrict__ v, const double2 *__restrict__ B,
                 float4 *__restrict__ vff, double2 *__restrict__ x, double2 *__restrict__ y,
                 float4 *__restrict__ xyff, double2 *__restrict__ b, double2 *__restrict__ tx,
                 double2 *__restrict__ ty, float2 *__restrict__ by32, double *__restrict__ bpart) {
  __shared__ double2 vs[kRows];
  const int t = threadIdx.x;
  const long long i = (long long)blockIdx.x * kRows + t;
  const bool ok = t < kRows && i < n;
  double2 vi = make_double2(0.0, 0.0);
  if (ok) {
    vi = v[i];
    vs[t] = vi;
    vff[i] = ff_split(vi);
    x[i] = y[i] = make_double2(0.0, 0.0);
    xyff[2 * i] = xyff[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  double s2 = 0.0;
  if (ok) {
    const double2 bi = block_row(B + (i / 5) * 25 + (t % 5) * 5, vs + t / 5 * 5);
    b[i] = bi;
    tx[i] = bi;
    ty[i] = make_double2(0.0, 0.0);
    by32[i] = make_float2(0.f, 0.f);
    s2 = bi.x * bi.x + bi.y * bi.y;
  }
  block_sum_sq(s2, bpart + blockIdx.x);
}

__global__ void k_pipe_split(long long n, const double2 *__restrict__ a, float4 *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = ff_split(a[i]);
}

// Column j of H = the two Gram-Schmidt passes and beta, then g1 = H h and
// g2 = H g1(0 : j+1) (OP V h = V g1; OP V g1 = V g2 + g1(j+1) OP v_{j+1}).
// One CTA: four lanes per row.
__global__ void __launch_bounds__(kThreads)
    k_pipe_coef(int j, int ldh, const double2 *__restrict__ h1, const double2 *__restrict__ h2,
                const double *__restrict__ beta, double2 *__restrict__ H,
                float4 *__restrict__ g) {
  extern __shared__ double2 sh[];  // [2][ldh]: h, then g1
  double2 *gs = sh + ldh;
  const int m = j + 2;  // rows of the column
  for (int i = threadIdx.x; i < ldh; i += kThreads) {
    double2 v = make_double2(0.0, 0.0);
    if (i <= j) {
      v = cadd(h1[i], h2[i]);
      sh[i] = v;
    } else if (i == j + 1) {
      v.x = *beta;
    }
    H[(long long)j * ldh + i] = v;
  }
  __syncthreads();
  const int part = threadIdx.x & 3;
  for (int pass = 0; pass < 2; ++pass) {
    const double2 *c = pass ? gs : sh;
    for (int r0 = 0; r0 < m; r0 += kThreads / 4) {
      const int i = r0 + threadIdx.x / 4;
      double2 acc = make_double2(0.0, 0.0);
      if (i < m)
        for (int q = part; q <= j; q += 4) acc = cfma(acc, H[(long long)q * ldh + i], c[q]);
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
      }
      if (part == 0 && i < m) {
        if (!pass) gs[i] = acc;
        g[pass * ldh + i] = ff_split(acc);
      }
    }
    __syncthreads();
  }
}

// v_{j+1} = w / beta, x' = (y - V g1) / beta, y' = (u - V g2 - g1(j+1) x') /
// beta over the nk = j + 1 old basis vectors and the new one, then B v, the
// targets of x' and y' and B y'.  Bound by reading the basis: the products
// run in float-float on the FP32 pipe (they only make the guesses that the
// refinement corrects; FP64 FMAs would take ten times the reading).  The
// new basis vector itself is formed in FP64.
__global__ void __launch_bounds__(kThreads)
    k_pipe_shift(long long n, int nk, int ldh, const float4 *__restrict__ vff,
                 const float4 *__restrict__ g, const double *__restrict__ beta,
                 const double2 *__restrict__ B, double2 sg, double2 *__restrict__ x,
                 double2 *__restrict__ y, double2 *__restrict__ vnew,
                 float4 *__restrict__ vffnew, float4 *__restrict__ xyff,
                 double2 *__restrict__ b, double2 *__restrict__ tx, double2 *__restrict__ ty,
                 const float2 *__restrict__ u, float2 *__restrict__ by32,
                 double *__restrict__ bpart) {
  extern __shared__ float4 gsh[];  // [2][nk + 1]
  __shared__ double2 vs[kRows], xs[kRows], ys[kRows];
  float4 *g1 = gsh, *g2 = gsh + nk + 1;
  const int t = threadIdx.x;
  for (int k = t; k <= nk; k += kThreads) {
    g1[k] = g[k];
    g2[k] = g[ldh + k];
  }
  __syncthreads();
  const long long i = (long long)blockIdx.x * kRows + t;
  const bool ok = t < kRows && i < n;
  if (ok) {
    FFC a1{0.f, 0.f, 0.f, 0.f}, a2{0.f, 0.f, 0.f, 0.f};
    const float4 *Vi = vff + i;
    int k = 0;
    for (; k + 4 <= nk; k += 4) {
      float4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = Vi[(long long)(k + q) * n];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ffc_mac(a1, v[q], g1[k + q]);
        ffc_mac(a2, v[q], g2[k + q]);
      }
    }
    for (; k < nk; ++k) {
      const float4 v = Vi[(long long)k * n];
      ffc_mac(a1, v, g1[k]);
      ffc_mac(a2, v, g2[k]);
    }
    const double d = *beta;
    const double f = (d > 0.0 && d < INFINITY) ? 1.0 / d : 0.0;
    const double2 w = x[i];
    const double2 v = make_double2(w.x * f, w.y * f);
    const float4 vf = ff_split(v);
    ffc_mac(a1, vf, g1[nk]);
    ffc_mac(a2, vf, g2[nk]);
    const double2 s1 = ffc_value(a1), s2 = ffc_value(a2), yi = y[i];
    const float2 ui = u[i];
    const float4 gn = g1[nk];
    const double2 gd = make_double2((double)gn.x + (double)gn.y, (double)gn.z + (double)gn.w);
    const double2 xn = make_double2((yi.x - s1.x) * f, (yi.y - s1.y) * f);
    double2 yn = cfms(make_double2((double)ui.x - s2.x, (double)ui.y - s2.y), gd, xn);
    yn.x *= f;
    yn.y *= f;
    vnew[i] = v;
    vffnew[i] = vf;
    x[i] = xn;
    y[i] = yn;
    xyff[2 * i] = ff_split(xn);
    xyff[2 * i + 1] = ff_split(yn);
    vs[t] = v;
    xs[t] = xn;
    ys[t] = yn;
  }
  __syncthreads();
  double s2 = 0.0;
  if (ok) {
    const double2 *Bb = B + (i / 5) * 25 + (t % 5) * 5;
    const int q = t / 5 * 5;
    const double2 bi = block_row(Bb, vs + q);
    b[i] = bi;
    s2 = bi.x * bi.x + bi.y * bi.y;
    targets(i, Bb, xs + q, ys + q, bi, sg, tx, ty, by32);
  }
  block_sum_sq(s2, bpart + blockIdx.x);
}

// x += c_x, y += c_y (with corrections), their splits and targets.
__global__ void __launch_bounds__(kThreads)
    k_pipe_targets(long long n, int correct, const double2 *__restrict__ B, double2 sg,
                   double2 *__restrict__ x, double2 *__restrict__ y, float4 *__restrict__ xyff,
                   const double2 *__restrict__ b, double2 *__restrict__ tx,
                   double2 *__restrict__ ty, const float2 *__restrict__ rhs,
                   float2 *__restrict__ by32) {
  __shared__ double2 xs[kRows], ys[kRows];
  const int t = threadIdx.x;
  const long long i = (long long)blockIdx.x * kRows + t;
  const bool ok = t < kRows && i < n;
  if (ok) {
    double2 xi = x[i], yi = y[i];
    if (correct) {
      const float2 cx = rhs[i], cy = rhs[n + i];
      xi.x += cx.x;
      xi.y += cx.y;
      yi.x += cy.x;
      yi.y += cy.y;
      x[i] = xi;
      y[i] = yi;
    }
    xyff[2 * i] = ff_split(xi);
    xyff[2 * i + 1] = ff_split(yi);
    xs[t] = xi;
    ys[t] = yi;
  }
  __syncthreads();
  if (ok) {
    const double2 *Bb = B + (i / 5) * 25 + (t % 5) * 5;
    const int q = t / 5 * 5;
    targets(i, Bb, xs + q, ys + q, b[i], sg, tx, ty, by32);
  }
}

// A times x (NV = 1) or x and y (NV = 2) in float-float, subtracted from
// the targets.  Warp per block row, lane 5 r + c holds entry (r, c) of each
// block; the operator is read once for both vectors.  NV = 2 writes the
// three right-hand sides, NV = 1 this CTA's sum of |r|^2.
template <int NV>
__global__ void __launch_bounds__(32 * kWarpRows)
    k_pipe_residual(int nrows, const int *__restrict__ row_ptr, const int *__restrict__ col,
                    const float4 *__restrict__ aff, const float4 *__restrict__ xyff,
                    const double2 *__restrict__ tx, const double2 *__restrict__ ty,
                    const float2 *__restrict__ by32, float2 *__restrict__ rhs, long long n,
                    double *__restrict__ rpart) {
  __shared__ double red[kWarpRows];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int row = blockIdx.x * kWarpRows + wp;
  const int c = lane % 5;
  const bool active = lane < 25;
  double s2 = 0.0;
  if (row < nrows) {
    FFC s[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = FFC{0.f, 0.f, 0.f, 0.f};
    const int k0 = row_ptr[row], k1 = row_ptr[row + 1];
    constexpr int kU = NV == 1 ? 8 : 5;
    for (int k = k0; k < k1; k += kU) {
      float4 a[kU], xv[kU][NV];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const bool ok = active && k + u < k1;
        a[u] = ok ? __ldcs(aff + (size_t)(k + u) * 25 + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 *p = xyff + (ok ? 2 * ((size_t)col[k + u] * 5 + c) : 0);
#pragma unroll
        for (int v = 0; v < NV; ++v) xv[u][v] = ok ? p[v] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int v = 0; v < NV; ++v) ffc_mac(s[v], a[u], xv[u][v]);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int d = 1; d < 5; ++d) {
        const float h1 = __shfl_down_sync(0xffffffffu, s[v].rh, d);
        const float l1 = __shfl_down_sync(0xffffffffu, s[v].rl, d);
        const float h2 = __shfl_down_sync(0xffffffffu, s[v].ih, d);
        const float l2 = __shfl_down_sync(0xffffffffu, s[v].il, d);
        if (c == 0) {
          ff_add(s[v].rh, s[v].rl, h1, l1);
          ff_add(s[v].ih, s[v].il, h2, l2);
        }
      }
    }
    if (active && c == 0) {
      const size_t i = (size_t)row * 5 + lane / 5;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double2 a = ffc_value(s[v]), tg = v ? ty[i] : tx[i];
        const double2 r = make_double2(tg.x - a.x, tg.y - a.y);
        if (NV == 1)
          s2 = r.x * r.x + r.y * r.y;
        else
          rhs[v * n + i] = make_float2((float)r.x, (float)r.y);
      }
      if (NV == 2) rhs[2 * n + i] = by32[i];
    }
  }
  if (NV == 1) {
    for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    if (lane == 0) red[wp] = s2;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int p = 0; p < kWarpRows; ++p) t += red[p];
      rpart[blockIdx.x] = t;
    }
  }
}

// out = sqrt of the two partial sums, summed in a fixed order
__global__ void __launch_bounds__(512)
    k_pipe_norms(int nr, const double *__restrict__ rpart, int nb,
                 const double *__restrict__ bpart, double *__restrict__ out) {
  __shared__ double red[2][16];
  double s[2] = {0.0, 0.0};
  for (int i = threadIdx.x; i < nr; i += 512) s[0] += rpart[i];
  for (int i = threadIdx.x; i < nb; i += 512) s[1] += bpart[i];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = s[k];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int p = 0; p < 16; ++p) t += red[threadIdx.x][p];
    out[threadIdx.x] = sqrt(t);
  }
}

int node_blocks(const Pipe &p) { return blocks_for(p.nn, kNodes); }
int row_blocks(const Pipe &p) { return blocks_for(p.nn, kWarpRows); }

}  // namespace

int pipe_alloc(tlr_ctx *ctx, Pipe &p, int ncv) {
  p.nn = ctx->nn;
  p.n = 5LL * ctx->nn;
  p.ncv = ncv;
  p.ldh = ncv + 2;
  const size_t n = (size_t)p.n;
  TLR_CUDA(ctx, cudaMalloc(&p.vff, sizeof(float4) * n * (ncv + 1)));
  TLR_CUDA(ctx, cudaMalloc(&p.xyff, sizeof(float4) * 2 * n));
  TLR_CUDA(ctx, cudaMalloc(&p.y, sizeof(double2) * n));
  TLR_CUDA(ctx, cudaMalloc(&p.b, sizeof(double2) * n));
  TLR_CUDA(ctx, cudaMalloc(&p.tx, sizeof(double2) * n));
  TLR_CUDA(ctx, cudaMalloc(&p.ty, sizeof(double2) * n));
  TLR_CUDA(ctx, cudaMalloc(&p.by32, sizeof(float2) * n));
  TLR_CUDA(ctx, cudaMalloc(&p.H, sizeof(double2) * p.ldh * ncv));
  TLR_CUDA(ctx, cudaMalloc(&p.g, sizeof(float4) * 2 * p.ldh));
  TLR_CUDA(ctx, cudaMalloc(&p.bpart, sizeof(double) * node_blocks(p)));
  TLR_CUDA(ctx, cudaMalloc(&p.rpart, sizeof(double) * row_blocks(p)));
  TLR_CUDA(ctx, cudaHostAlloc(&p.hup, sizeof(double2) * p.ldh * ncv, cudaHostAllocDefault));
  return TLR_OK;
}

void pipe_free(Pipe &p) {
  cudaFree(p.vff); cudaFree(p.xyff); cudaFree(p.y); cudaFree(p.b); cudaFree(p.tx);
  cudaFree(p.ty); cudaFree(p.by32); cudaFree(p.H); cudaFree(p.g); cudaFree(p.bpart); cudaFree(p.rpart);
  cudaFreeHost(p.hup);
  p = Pipe();
}

int pipe_start(tlr_ctx *ctx, Pipe &p, const double2 *v, double2 *x) {
  { k_pipe_start<<<node_blocks(p), kThreads, 0, ctx->stream>>>(
      p.n, v, ctx->B, p.vff, x, p.y, p.xyff, p.b, p.tx, p.ty, p.by32, p.bpart); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_split_basis(tlr_ctx *ctx, Pipe &p, const double2 *V, int nk) {
  const long long n = p.n * nk;
  { k_pipe_split<<<blocks_for(n, 256), 256, 0, ctx->stream>>>(n, V, p.vff); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_upload_h(tlr_ctx *ctx, Pipe &p, int l) {
  TLR_CUDA(ctx, cudaMemcpyAsync(p.H, p.hup, sizeof(double2) * p.ldh * l, cudaMemcpyHostToDevice,
                                ctx->stream));
  return TLR_OK;
}

int pipe_coefficients(tlr_ctx *ctx, Pipe &p, int j, const double2 *h1, const double2 *h2,
                      const double *beta) {
  const size_t sm = sizeof(double2) * 2 * p.ldh;
  if (sm > 48 * 1024)
    TLR_CUDA(ctx, cudaFuncSetAttribute(k_pipe_coef, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sm));
  { k_pipe_coef<<<1, kThreads, sm, ctx->stream>>>(j, p.ldh, h1, h2, beta, p.H, p.g); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_shift(tlr_ctx *ctx, Pipe &p, int j, const double *beta, double sr, double si,
               double2 *x, double2 *vnew, const float2 *rhs) {
  const size_t sm = sizeof(float4) * 2 * (j + 2);
  if (sm > 32 * 1024)  // the static arrays take 12 KB of the 48 KB
    TLR_CUDA(ctx, cudaFuncSetAttribute(k_pipe_shift, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sm));
  { k_pipe_shift<<<node_blocks(p), kThreads, sm, ctx->stream>>>(
      p.n, j + 1, p.ldh, p.vff, p.g, beta, ctx->B, make_double2(sr, si), x, p.y, vnew,
      p.vff + (size_t)(j + 1) * p.n, p.xyff, p.b, p.tx, p.ty, rhs + 2 * p.n,
      p.by32, p.bpart); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_residuals(tlr_ctx *ctx, Pipe &p, float2 *rhs) {
  { k_pipe_residual<2><<<row_blocks(p), 32 * kWarpRows, 0, ctx->stream>>>(
      p.nn, ctx->row_ptr, ctx->col, ctx->aff, p.xyff, p.tx, p.ty, p.by32, rhs, p.n, nullptr); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_targets(tlr_ctx *ctx, Pipe &p, double sr, double si, double2 *x, const float2 *rhs,
                 bool correct) {
  { k_pipe_targets<<<node_blocks(p), kThreads, 0, ctx->stream>>>(
      p.n, correct ? 1 : 0, ctx->B, make_double2(sr, si), x, p.y, p.xyff, p.b, p.tx, p.ty, rhs,
      p.by32); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_accept(tlr_ctx *ctx, Pipe &p, double *out) {
  { k_pipe_residual<1><<<row_blocks(p), 32 * kWarpRows, 0, ctx->stream>>>(
      p.nn, ctx->row_ptr, ctx->col, ctx->aff, p.xyff, p.tx, p.ty, p.by32, nullptr, p.n, p.rpart); count_launches(); }
  { k_pipe_norms<<<1, 512, 0, ctx->stream>>>(row_blocks(p), p.rpart, node_blocks(p), p.bpart, out); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

}  // namespace tlr
