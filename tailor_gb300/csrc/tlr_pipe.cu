// tlr_pipe.cu -- kernels of the pipelined refined applications (tlr_pipe.h).
//
// No counterpart in the reference: PCLU applies MUMPS's FP64 factor once per
// application (EigenSolver.cpp:61-71).
#include <algorithm>

#include "tlr_async.cuh"
#include "tlr_complex.cuh"
#include "tlr_ff.cuh"
#include "tlr_pipe.h"

namespace tlr {
namespace {

// The element-wise kernels own whole grid nodes (five unknowns), because
// they end in a product with the block-diagonal B: 12 nodes per CTA of 64
// threads, so that the smallest grids still fill the SMs.
constexpr int kNodes = 12, kRows = 5 * kNodes, kThreads = 64;
// the shift: 10 nodes per CTA, five threads per row sharing the basis
// vectors (one thread per row left 38 CTAs of 20 dependent steps at 60 x 32:
// 15 us)
constexpr int kSNodes = 10, kSRows = 5 * kSNodes, kSGroups = 5, kSThreads = 256;
// A products: one CTA of 16 warps per SM, each warp with a ring of five
// stages of six blocks in shared memory (192 KB)
constexpr int kRWarps = 16, kRStages = 5, kRBlocks = 6, kRStage = 25 * kRBlocks;
constexpr size_t kRSmem = sizeof(float4) * kRWarps * kRStages * kRStage;

__device__ __forceinline__ double2 block_row(const double2 *Bb, const double2 *s) {
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < 5; ++q) acc = cfma(acc, Bb[q], s[q]);
  return acc;
}

// Targets of x and y and the right-hand side of u, for this thread's row:
// tx = b + sigma B x, ty = B x + sigma B y, u's right-hand side B y (FP32, the
// factor's precision; FP64 only where sigma needs it: the FP64 pipe is what
// these kernels are short of).  xs: x of the node, ys: y of the node as
// float-float.
__device__ __forceinline__ void targets(long long i, const double2 *Bb, const float2 *B32,
                                        const double2 *xs, const float4 *ys, double2 b,
                                        double2 sg, double2 *__restrict__ tx,
                                        double2 *__restrict__ ty, float2 *__restrict__ by32) {
  const double2 bx = block_row(Bb, xs);
  if (sg.x == 0.0 && sg.y == 0.0) {
    float2 by = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 5; ++q) by = cfma(by, B32[q], make_float2(ys[q].x, ys[q].z));
    tx[i] = b;
    ty[i] = bx;
    by32[i] = by;
  } else {
    double2 yd[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) yd[q] = ff_value(ys[q]);
    const double2 by = block_row(Bb, yd);
    tx[i] = cfma(b, sg, bx);
    ty[i] = cfma(bx, sg, by);
    by32[i] = make_float2((float)by.x, (float)by.y);
  }
}

// this CTA's sum of |b|^2
template <int THREADS>
__device__ __forceinline__ void block_sum_sq(double s, double *out) {
  __shared__ double red[THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int p = 0; p < THREADS / 32; ++p) t += red[p];
    *out = t;
  }
}

__global__ void __launch_bounds__(kSThreads)
    k_pipe_start(long long n, const double2 *__restrict__ v, const double2 *__restrict__ B,
                 float4 *__restrict__ vff, double2 *__restrict__ x,
                 float4 *__restrict__ xyff, double2 *__restrict__ b, double2 *__restrict__ tx,
                 double2 *__restrict__ ty, float2 *__restrict__ by32, double *__restrict__ bpart) {
  __shared__ double2 vs[kSRows];
  const int t = threadIdx.x;
  const long long i = (long long)blockIdx.x * kSRows + t;
  const bool ok = t < kSRows && i < n;
  double2 vi = make_double2(0.0, 0.0);
  if (ok) {
    vi = v[i];
    vs[t] = vi;
    vff[i] = ff_split(vi);
    x[i] = make_double2(0.0, 0.0);
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
  block_sum_sq<kSThreads>(s2, bpart + blockIdx.x);
}

__global__ void k_pipe_b32(long long n, const double2 *__restrict__ B, float2 *__restrict__ B32) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) B32[i] = make_float2((float)B[i].x, (float)B[i].y);
}

__global__ void k_pipe_split(long long n, const double2 *__restrict__ a, float4 *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = ff_split(a[i]);
}

// v_{j+1} = w / beta, x' = (y - V g1) / beta, y' = (u - V g2 - g1(j+1) x') /
// beta over the nk = j + 1 old basis vectors and the new one, then B v, the
// targets of x' and y' and B y'.  A large basis is bound by reading it: the
// products run in float-float on the FP32 pipe (they only make the guesses that
// the refinement corrects; FP64 FMAs would take ten times the reading).  The
// new basis vector itself is formed in FP64.  A small one is bound by the chain of
// one CTA: 21 vectors at 100 x 50 take 20 us with DRAM 8%, the FP64 pipe (B's
// products) 41% and the FP32 pipe 15% busy, a third of the stalls at barriers.
__global__ void __launch_bounds__(kSThreads, 3)
    k_pipe_shift(long long n, int nk, int ldh, const float4 *__restrict__ vff,
                 const float4 *__restrict__ g, const double *__restrict__ beta,
                 const double2 *__restrict__ B, const float2 *__restrict__ B32, double2 sg,
                 double2 *__restrict__ x, double2 *__restrict__ vnew,
                 float4 *__restrict__ vffnew, float4 *__restrict__ xyff,
                 double2 *__restrict__ b, double2 *__restrict__ tx, double2 *__restrict__ ty,
                 const float2 *__restrict__ u, float2 *__restrict__ by32,
                 double *__restrict__ bpart) {
  extern __shared__ float4 gsh[];  // [2][nk + 1]
  __shared__ double2 vs[kSRows], xs[kSRows];
  __shared__ float4 ys[kSRows];
  __shared__ FFC part[kSGroups - 1][2][kSRows];
  float4 *g1 = gsh, *g2 = gsh + nk + 1;
  const int t = threadIdx.x;
  for (int k = t; k <= nk; k += kSThreads) {
    g1[k] = g[k];
    g2[k] = g[ldh + k];
  }
  const int grp = t / kSRows, r = t - grp * kSRows;
  const long long i = (long long)blockIdx.x * kSRows + r;
  const bool ok = grp < kSGroups && i < n;
  const bool own = ok && grp == 0;
  // the owner's operands go out before the basis products
  double2 w = make_double2(0.0, 0.0), bl[5];
  float4 yi = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 ui = make_float2(0.f, 0.f), b32[5];
  const double d = *beta;
  if (own) {
    w = x[i];
    yi = xyff[2 * i + 1];
    ui = u[i];
    const long long bo = (i / 5) * 25 + (r % 5) * 5;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      bl[q] = B[bo + q];
      b32[q] = B32[bo + q];
    }
  }
  __syncthreads();
  FFC a1{0.f, 0.f, 0.f, 0.f}, a2{0.f, 0.f, 0.f, 0.f};
  if (ok) {  // basis vectors grp, grp + 5, ...
    const float4 *Vi = vff + i;
    int k = grp;
    for (; k + 3 * kSGroups < nk; k += 4 * kSGroups) {
      float4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = Vi[(long long)(k + q * kSGroups) * n];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ffc_mac(a1, v[q], g1[k + q * kSGroups]);
        ffc_mac(a2, v[q], g2[k + q * kSGroups]);
      }
    }
    for (; k < nk; k += kSGroups) {
      const float4 v = Vi[(long long)k * n];
      ffc_mac(a1, v, g1[k]);
      ffc_mac(a2, v, g2[k]);
    }
    if (grp > 0) {
      part[grp - 1][0][r] = a1;
      part[grp - 1][1][r] = a2;
    }
  }
  __syncthreads();
  if (own) {
#pragma unroll
    for (int q = 0; q < kSGroups - 1; ++q) {
      const FFC p1 = part[q][0][r], p2 = part[q][1][r];
      ff_add(a1.rh, a1.rl, p1.rh, p1.rl);
      ff_add(a1.ih, a1.il, p1.ih, p1.il);
      ff_add(a2.rh, a2.rl, p2.rh, p2.rl);
      ff_add(a2.ih, a2.il, p2.ih, p2.il);
    }
    const double f = (d > 0.0 && d < INFINITY) ? 1.0 / d : 0.0;
    const double2 v = make_double2(w.x * f, w.y * f);
    const float4 vf = ff_split(v);
    ffc_mac(a1, vf, g1[nk]);
    ffc_mac(a2, vf, g2[nk]);
    // the guesses stay on the FP32 pipe (float-float)
    const float fh = (float)f, fl = (float)(f - (double)fh);
    const float4 xn = ffc_scale(ffc_sub(yi, a1), fh, fl);
    ffc_mac(a2, xn, g1[nk]);
    const float4 yn =
        ffc_scale(ffc_sub(make_float4(ui.x, 0.f, ui.y, 0.f), a2), fh, fl);
    const double2 xd = ff_value(xn);
    vnew[i] = v;
    vffnew[i] = vf;
    x[i] = xd;
    xyff[2 * i] = xn;
    xyff[2 * i + 1] = yn;
    vs[r] = v;
    xs[r] = xd;
    ys[r] = yn;
  }
  __syncthreads();
  double s2 = 0.0;
  if (own) {
    const int q = r / 5 * 5;
    const double2 bi = block_row(bl, vs + q);
    b[i] = bi;
    s2 = bi.x * bi.x + bi.y * bi.y;
    targets(i, bl, b32, xs + q, ys + q, bi, sg, tx, ty, by32);
  }
  block_sum_sq<kSThreads>(s2, bpart + blockIdx.x);
}

// x += c_x, y += c_y and u = c_u, or u += c_u where the round refined u
// (correct 1, 2; 0: none), their splits and targets; u's target is B y + sigma
// B u, in FP32.
__global__ void __launch_bounds__(kThreads)
    k_pipe_targets(long long n, int correct, const double2 *__restrict__ B,
                   const float2 *__restrict__ B32, double2 sg, double2 *__restrict__ x,
                   float4 *__restrict__ xyff,
                   const double2 *__restrict__ b, double2 *__restrict__ tx,
                   double2 *__restrict__ ty, float2 *__restrict__ rhs,
                   float2 *__restrict__ by32, float2 *__restrict__ u32,
                   float2 *__restrict__ tu32) {
  __shared__ double2 xs[kRows];
  __shared__ float4 ys[kRows];
  __shared__ float2 us[kRows];
  const int t = threadIdx.x;
  const long long i = (long long)blockIdx.x * kRows + t;
  const bool ok = t < kRows && i < n;
  double2 bl[5], bi = make_double2(0.0, 0.0);
  float2 b32[5];
  if (ok) {
    double2 xi = x[i];
    float4 yi = xyff[2 * i + 1];
    const long long bo = (i / 5) * 25 + (t % 5) * 5;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      bl[q] = B[bo + q];
      b32[q] = B32[bo + q];
    }
    bi = b[i];
    if (correct) {
      const float2 cx = rhs[i], cy = rhs[n + i];
      xi.x += cx.x;
      xi.y += cx.y;
      ff_add(yi.x, yi.y, cy.x, 0.f);
      ff_add(yi.z, yi.w, cy.y, 0.f);
      ff_norm(yi.x, yi.y);
      ff_norm(yi.z, yi.w);
      x[i] = xi;
      xyff[2 * i + 1] = yi;
    }
    float2 ui = correct ? rhs[2 * n + i] : u32[i];
    if (correct == 2) {
      const float2 uo = u32[i];
      ui.x += uo.x;
      ui.y += uo.y;
      rhs[2 * n + i] = ui;
    }
    if (correct) u32[i] = ui;
    xyff[2 * i] = ff_split(xi);
    xs[t] = xi;
    ys[t] = yi;
    us[t] = ui;
  }
  __syncthreads();
  if (ok) {
    const int q = t / 5 * 5;
    targets(i, bl, b32, xs + q, ys + q, bi, sg, tx, ty, by32);
    float2 tu = by32[i];
    if (sg.x != 0.0 || sg.y != 0.0) {
      float2 bu = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 5; ++k) bu = cfma(bu, b32[k], us[q + k]);
      tu = cfma(tu, make_float2((float)sg.x, (float)sg.y), bu);
    }
    tu32[i] = tu;
  }
}

// A times x (NV = 1), x and y (NV = 2) or x, y and u (NV = 3) in float-float,
// subtracted from the targets.  Bound by reading the operator (NV = 1: 5.3 TB/s at
// 300 x 192) and by the float-float arithmetic on the FP32 pipe (NV = 2, 96
// instructions per entry).  At 100 x 50, two or three block rows per warp, neither is
// reached: 49 us at 41% of DRAM's rate and 62 us with the FP32 pipe 47% busy, the
// last rows of a CTA's warps its tail.  A block
// row's blocks are contiguous, so each warp streams its rows (row gw, gw + W,
// ...) through its own ring with bulk copies of six blocks, issued by its
// first lane five stages ahead and across rows.  Lane 5 b + r multiplies row r
// of block b: 30 of 32 lanes work (25 with a lane per entry of one block), a
// lane's five entries are 80 consecutive bytes (no bank conflicts), and a row
// is summed over six lanes at its end.  Every wait is bounded: on a timeout
// the warp raises the error flag, waits once more for its copies in flight
// and stops.  NV = 2 and 3 write the three right-hand sides, NV = 1 the norms
// out[0] = |r|, out[1] = |b| (b's partial sums: bpart).
template <int NV>
__global__ void __launch_bounds__(32 * kRWarps, 1)
    k_pipe_residual(int nrows, const int *__restrict__ row_ptr, const int *__restrict__ col,
                    const float4 *__restrict__ aff, const float4 *__restrict__ xyff,
                    const double2 *__restrict__ tx, const double2 *__restrict__ ty,
                    const float2 *__restrict__ by32, const float2 *__restrict__ u32,
                    float2 *__restrict__ rhs, long long n, double *__restrict__ rpart, int nb,
                    const double *__restrict__ bpart,
                    int *__restrict__ arrived, double *__restrict__ out, int *__restrict__ err) {
  extern __shared__ __align__(128) float4 ring_all[];
  __shared__ __align__(8) uint64_t full_all[kRWarps][kRStages];
  __shared__ double red[2][kRWarps];
  __shared__ int last;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  float4 *ring = ring_all + wp * kRStages * kRStage;
  uint64_t *full = full_all[wp];
  const int W = gridDim.x * kRWarps, gw = wp * gridDim.x + blockIdx.x;
  if (lane == 0) {
    for (int q = 0; q < kRStages; ++q) mbar_init(&full[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // producer cursor (first lane): the next blocks [pk, pe) of row prow
  int prow = gw - W, pk = 0, pe = 0, issued = 0;
  auto issue = [&]() {
    while (pk >= pe) {
      prow += W;
      if (prow >= nrows) {
        prow -= W;  // stay here: nothing left
        return;
      }
      pk = row_ptr[prow];
      pe = row_ptr[prow + 1];
    }
    const int nb = min(kRBlocks, pe - pk), st = issued % kRStages;
    mbar_expect_tx(&full[st], nb * 400);
    bulk_g2s(ring + st * kRStage, aff + (size_t)pk * 25, nb * 400, &full[st]);
    pk += nb;
    ++issued;
  };
  if (lane == 0)
    for (int q = 0; q < kRStages; ++q) issue();
  const int l = min(lane, 29), bl = l / 5, rr = l % 5;
  int consumed = 0;
  bool fine = true;
  double s2 = 0.0;
  for (int row = gw; row < nrows && fine; row += W) {
    const int k0 = row_ptr[row], k1 = row_ptr[row + 1];
    FFC s[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = FFC{0.f, 0.f, 0.f, 0.f};
    // the columns of 30 blocks at a time, x one stage ahead
    int mycol = lane < 30 && k0 + lane < k1 ? col[k0 + lane] : 0;
    for (int kb = k0; kb < k1 && fine; kb += 30) {
      const int nxcol = lane < 30 && kb + 30 + lane < k1 ? col[kb + 30 + lane] : 0;
      constexpr int NF = NV < 3 ? NV : 2;  // vectors held as float-float
      float4 xv[NF][5];
      float2 uv[NV == 3 ? 5 : 1];
      auto load_x = [&](int j) {  // stage j of this group of 30 blocks
        const int c = __shfl_sync(0xffffffffu, mycol, min(j * kRBlocks + bl, 29));
        const float4 *p = xyff + (size_t)c * 10;
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
          for (int v = 0; v < NF; ++v) xv[v][q] = p[2 * q + v];
        if (NV == 3)
#pragma unroll
          for (int q = 0; q < 5; ++q) uv[q % (NV == 3 ? 5 : 1)] = u32[(size_t)c * 5 + q];
      };
      load_x(0);
      for (int j = 0; j < 5 && kb + j * kRBlocks < k1; ++j) {
        const int st = consumed % kRStages;
        if (!mbar_wait(&full[st], (consumed / kRStages) & 1)) fine = false;
        fine = __all_sync(0xffffffffu, fine);
        if (!fine) break;
        if (kb + j * kRBlocks + bl < k1) {
          const float4 *ap = ring + st * kRStage + l * 5;
#pragma unroll
          for (int q = 0; q < 5; ++q) {
            const float4 av = ap[q];
#pragma unroll
            for (int v = 0; v < NF; ++v) ffc_mac(s[v], av, xv[v][q]);
            if (NV == 3) {
              const float2 ui = uv[q % (NV == 3 ? 5 : 1)];
              ffc_mac(s[NV - 1], av, make_float4(ui.x, 0.f, ui.y, 0.f));
            }
          }
        }
        __syncwarp();
        ++consumed;
        if (lane == 0) issue();
        if (j < 4) load_x(j + 1);
      }
      mycol = nxcol;
    }
    // lanes r, r + 5, ..., r + 25 hold row r
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int o = d == 0 ? 15 : 5;
        const float h1 = __shfl_down_sync(0xffffffffu, s[v].rh, o * (d == 2 ? 2 : 1));
        const float l1 = __shfl_down_sync(0xffffffffu, s[v].rl, o * (d == 2 ? 2 : 1));
        const float h2 = __shfl_down_sync(0xffffffffu, s[v].ih, o * (d == 2 ? 2 : 1));
        const float l2 = __shfl_down_sync(0xffffffffu, s[v].il, o * (d == 2 ? 2 : 1));
        if (d == 0 ? lane < 15 : lane < 5) {
          ff_add(s[v].rh, s[v].rl, h1, l1);
          ff_add(s[v].ih, s[v].il, h2, l2);
        }
      }
    }
    if (lane < 5) {
      const size_t i = (size_t)row * 5 + rr;
#pragma unroll
      for (int v = 0; v < (NV < 3 ? NV : 2); ++v) {
        const double2 av = ffc_value(s[v]), tg = v ? ty[i] : tx[i];
        const double2 r = make_double2(tg.x - av.x, tg.y - av.y);
        if (NV == 1) {
          s2 = fma(r.x, r.x, s2);
          s2 = fma(r.y, r.y, s2);
        } else {
          rhs[v * n + i] = make_float2((float)r.x, (float)r.y);
        }
      }
      if (NV == 2) rhs[2 * n + i] = by32[i];
      if (NV == 3) {  // by32: the target of u
        const double2 au = ffc_value(s[NV - 1]);
        const float2 tu = by32[i];
        rhs[2 * n + i] = make_float2((float)(tu.x - au.x), (float)(tu.y - au.y));
      }
    }
  }
  if (!fine && lane == 0) {
    atomicExch(err, 1);
    for (int q = consumed; q < issued; ++q) mbar_wait(&full[q % kRStages], (q / kRStages) & 1);
  }
  if (NV == 1) {
    for (int o = 4; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);  // lanes 0 .. 4
    if (lane == 0) red[0][wp] = s2;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int p = 0; p < kRWarps; ++p) t += red[0][p];
      rpart[blockIdx.x] = t;
      __threadfence();
      last = atomicAdd(arrived, 1) == (int)gridDim.x - 1;
      if (last) *arrived = 0;
      __threadfence();
    }
    __syncthreads();
    if (!last) return;
    // the last CTA: both norms, the partial sums added in a fixed order
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 32 * kRWarps) a += __ldcg(rpart + i);
    for (int i = threadIdx.x; i < nb; i += 32 * kRWarps) b += bpart[i];
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      red[0][wp] = a;
      red[1][wp] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      double t = 0.0;
      for (int p = 0; p < kRWarps; ++p) t += red[threadIdx.x][p];
      out[threadIdx.x] = sqrt(t);
    }
  }
}

int node_blocks(const Pipe &p) { return blocks_for(p.nn, kNodes); }
int shift_blocks(const Pipe &p) { return blocks_for(p.nn, kSNodes); }
int row_blocks(const Pipe &p) { return std::min(p.sms, blocks_for(p.nn, kRWarps)); }

int alloc_buffers(tlr_ctx *ctx, Pipe &p, int ncv) {
  p.nn = ctx->nn;
  p.n = 5LL * ctx->nn;
  p.ncv = ncv;
  p.ldh = ncv + 2;
  p.sms = 1;
  cudaDeviceGetAttribute(&p.sms, cudaDevAttrMultiProcessorCount, ctx->device);
  TLR_CUDA(ctx, cudaFuncSetAttribute(k_pipe_residual<1>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRSmem));
  TLR_CUDA(ctx, cudaFuncSetAttribute(k_pipe_residual<2>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRSmem));
  TLR_CUDA(ctx, cudaFuncSetAttribute(k_pipe_residual<3>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRSmem));
  const size_t n = (size_t)p.n;
  auto dev = [](auto **q, size_t bytes) { return dev_malloc(q, bytes) == cudaSuccess; };
  if (!(dev(&p.vff, sizeof(float4) * n * (ncv + 1)) &&
        dev(&p.xyff, sizeof(float4) * 2 * n) &&
        dev(&p.B32, sizeof(float2) * 5 * n) &&
        dev(&p.b, sizeof(double2) * n) &&
        dev(&p.tx, sizeof(double2) * n) &&
        dev(&p.ty, sizeof(double2) * n) &&
        dev(&p.by32, sizeof(float2) * n) &&
        dev(&p.u32, sizeof(float2) * n) &&
        dev(&p.tu32, sizeof(float2) * n) &&
        dev(&p.H, sizeof(double2) * p.ldh * ncv) &&
        dev(&p.g, sizeof(float4) * 2 * p.ldh) &&
        dev(&p.bpart, sizeof(double) * shift_blocks(p)) &&
        dev(&p.rpart, sizeof(double) * row_blocks(p)) &&
        dev(&p.arrived, sizeof(int)) &&
        pin_malloc(&p.hup, sizeof(double2) * p.ldh * ncv) == cudaSuccess))
    return fail(ctx, TLR_ERR_NOMEM, "no memory for the pipelined applications");
  TLR_CUDA(ctx, cudaMemsetAsync(p.arrived, 0, sizeof(int), ctx->stream));
  return TLR_OK;
}

}  // namespace

int pipe_alloc(tlr_ctx *ctx, Pipe &p, int ncv) {
  const int rc = alloc_buffers(ctx, p, ncv);
  if (rc) pipe_free(p);  // all of them or none: vff says which
  return rc;
}

void pipe_free(Pipe &p) {
  cudaFree(p.vff); cudaFree(p.xyff); cudaFree(p.B32); cudaFree(p.b); cudaFree(p.tx);
  cudaFree(p.ty); cudaFree(p.by32); cudaFree(p.u32); cudaFree(p.tu32); cudaFree(p.H); cudaFree(p.g);
  cudaFree(p.bpart); cudaFree(p.rpart); cudaFree(p.arrived);
  cudaFreeHost(p.hup);
  p = Pipe();
}

int pipe_start(tlr_ctx *ctx, Pipe &p, const double2 *v, double2 *x) {
  { k_pipe_b32<<<blocks_for(5 * p.n, 256), 256, 0, ctx->stream>>>(5 * p.n, ctx->B, p.B32); count_launches(); }
  { k_pipe_start<<<shift_blocks(p), kSThreads, 0, ctx->stream>>>(
      p.n, v, ctx->B, p.vff, x, p.xyff, p.b, p.tx, p.ty, p.by32, p.bpart); count_launches(); }
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

int pipe_shift(tlr_ctx *ctx, Pipe &p, int j, const double *beta, double sr, double si,
               double2 *x, double2 *vnew, const float2 *rhs) {
  const size_t sm = sizeof(float4) * 2 * (j + 2);
  if (sm > 38 * 1024)  // the static arrays take 9 KB of the 48 KB
    TLR_CUDA(ctx, allow_dynamic_smem(k_pipe_shift));
  { k_pipe_shift<<<shift_blocks(p), kSThreads, sm, ctx->stream>>>(
      p.n, j + 1, p.ldh, p.vff, p.g, beta, ctx->B, p.B32, make_double2(sr, si), x, vnew,
      p.vff + (size_t)(j + 1) * p.n, p.xyff, p.b, p.tx, p.ty, rhs + 2 * p.n,
      p.by32, p.bpart); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_residuals(tlr_ctx *ctx, Pipe &p, float2 *rhs, bool refine_u, int *err) {
  if (refine_u)
    { k_pipe_residual<3><<<row_blocks(p), 32 * kRWarps, kRSmem, ctx->stream>>>(
        p.nn, ctx->row_ptr, ctx->col, ctx->aff, p.xyff, p.tx, p.ty, p.tu32, p.u32, rhs, p.n,
        nullptr, 0, nullptr, nullptr, nullptr, err); count_launches(); }
  else
    { k_pipe_residual<2><<<row_blocks(p), 32 * kRWarps, kRSmem, ctx->stream>>>(
        p.nn, ctx->row_ptr, ctx->col, ctx->aff, p.xyff, p.tx, p.ty, p.by32, nullptr, rhs, p.n,
        nullptr, 0, nullptr, nullptr, nullptr, err); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_targets(tlr_ctx *ctx, Pipe &p, double sr, double si, double2 *x, float2 *rhs,
                 int correct) {
  { k_pipe_targets<<<node_blocks(p), kThreads, 0, ctx->stream>>>(
      p.n, correct, ctx->B, p.B32, make_double2(sr, si), x, p.xyff, p.b, p.tx, p.ty, rhs, p.by32,
      p.u32, p.tu32); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

int pipe_accept(tlr_ctx *ctx, Pipe &p, double *out, int *err) {
  { k_pipe_residual<1><<<row_blocks(p), 32 * kRWarps, kRSmem, ctx->stream>>>(
      p.nn, ctx->row_ptr, ctx->col, ctx->aff, p.xyff, p.tx, p.ty, p.by32, nullptr, nullptr, p.n,
      p.rpart, shift_blocks(p), p.bpart, p.arrived, out, err); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  return TLR_OK;
}

}  // namespace tlr
