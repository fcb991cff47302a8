// tlr_bc.cu -- wall and characteristic far-field rows (K4).
//
// Reference: BoundaryConditions.cpp:353-548.  A_bc = -L and B_bc = M_Gamma
// are copied on the device; the wall (xi plane i = 0) keeps its continuity
// row and gets Dirichlet rows for u, v, w, T; each far-field node (i = Ny-1)
// gets rows R^-1[m,:] on its own columns for incoming modes and
// P[m,:] (-L rows), P[m,:] M rows otherwise, with P = R^-1 Gamma^-1.
//
// The reference obtains the normal eigensystem (n_y B_c + n_z C_c) r =
// s Gamma r from LAPACK zggev, whose eigenvector scaling and order are
// implementation details.  The inviscid blocks of LNSCoefficients.cpp:
// 303-356 give it in closed form -- speeds u_n (three times) and u_n +- c
// with c = sqrt(T)/M -- so each far-field node builds R analytically
// (acoustic, entropy, streamwise and tangential waves) and inverts it with
// the same pivoted Gauss-Jordan step as the reference (92-140).  The
// replaced rows span the reference's rows node by node (they differ by an
// invertible 5x5 left factor), which leaves the pencil's spectrum unchanged.
#include <algorithm>
#include <cfloat>

#include "tlr_internal.h"

namespace tlr {
namespace {

constexpr double kEps = DBL_EPSILON;

// A = -L, and the per-CTA sums of |a|^2 over the block rows that the boundary
// kernels leave alone (part).  CTA = whole block rows: both the copy and the
// sum stream L once; as passes of their own the sum cost as much again (the
// FP64 pipe: two FMAs per entry).
__global__ void __launch_bounds__(256)
    k_negate_copy(int nn, int ny, int row_entries, const double2 *__restrict__ L,
                  double2 *__restrict__ A, double *__restrict__ part) {
  __shared__ double sh[8];
  double s = 0.0;
  for (int row = blockIdx.x; row < nn; row += gridDim.x) {
    const int i = row % ny;
    const bool inner = i != 0 && i != ny - 1;
    const double2 *l = L + (long long)row * row_entries;
    double2 *a = A + (long long)row * row_entries;
    for (int x0 = threadIdx.x; x0 < row_entries; x0 += 4 * 256) {
      double2 v[4];  // four loads in flight
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[u] = x0 + 256 * u < row_entries ? __ldcs(l + x0 + 256 * u) : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (x0 + 256 * u < row_entries) __stcs(a + x0 + 256 * u, make_double2(-v[u].x, -v[u].y));
        if (inner) s = fma(v[u].x, v[u].x, fma(v[u].y, v[u].y, s));
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += sh[w];
    part[blockIdx.x] = t;
  }
}

// part[blockIdx.x] = the sum of |a|^2 of boundary block row blockIdx.x (wall
// rows first, then far-field rows); the last CTA adds all nparts partial sums
// from `all` on, in order, and writes the norm
__global__ void __launch_bounds__(256)
    k_boundary_norm(int ny, int nz, int row_entries, const double2 *__restrict__ A,
                    double *__restrict__ part, const double *__restrict__ all, int nparts,
                    double *__restrict__ out, int *__restrict__ ctr) {
  __shared__ double sh[8];
  __shared__ bool last;
  const int j = blockIdx.x % nz;
  const long long row = (long long)j * ny + (blockIdx.x < nz ? 0 : ny - 1);
  const double2 *a = A + row * row_entries;
  double s = 0.0;
  for (int x = threadIdx.x; x < row_entries; x += 256) {
    const double2 v = a[x];
    s = fma(v.x, v.x, fma(v.y, v.y, s));
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += sh[w];
    part[blockIdx.x] = t;
    __threadfence();
    last = atomicAdd(ctr, 1) == (int)gridDim.x - 1;
    if (last) *ctr = 0;
    __threadfence();
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  double t = 0.0;
  for (int b = threadIdx.x; b < nparts; b += 32) t += __ldcg(all + b);
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (threadIdx.x == 0) *out = sqrt(t);
}

// Wall: rows 1..4 of block row j*ny become e_row (A) and zero (B).
__global__ void k_wall(int ny, int nz, int S, const int *__restrict__ col,
                       double2 *__restrict__ A, double2 *__restrict__ B) {
  const long long total = (long long)nz * S * 20;
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < (long long)nz * 20) {
    const int j = (int)(x / 20), e = 5 + (int)(x % 20);
    B[(long long)(j * ny) * 25 + e] = make_double2(0.0, 0.0);
  }
  if (x >= total) return;
  const int j = (int)(x / (S * 20));
  const int rem = (int)(x % (S * 20));
  const int k = rem / 20, e = 5 + rem % 20;
  const int node = j * ny;
  const long long blk = (long long)node * S + k;
  const int r = e / 5, c = e % 5;
  const bool diag = col[blk] == node && r == c;
  A[blk * 25 + e] = make_double2(diag ? 1.0 : 0.0, 0.0);
}

struct Char {
  double Rinv[25];
  double P[25];
  int incoming[5];
  int ok;  // 0 success, else characteristic status
  int n_in, n_neutral;
  double cond;
};

// The 5 x 5 work of a far-field node by one warp, lane 5 r + c holding entry
// (r, c): serial on one thread it was a chain of a thousand dependent FP64
// operations (104 us).  Every entry takes the serial code's operations in its
// order, so the rows are bitwise the same.
struct CharWork {
  double R[25], m[25], Ginv[25], cond[2][5];
};

// inv = a^-1 by the reference's pivoted Gauss-Jordan; m: work
__device__ bool invert5(const double *a, double *m, double *inv) {
  const int lane = threadIdx.x & 31, r = lane / 5, c = lane % 5;
  const bool on = lane < 25;
  if (on) {
    m[lane] = a[lane];
    inv[lane] = (lane % 6 == 0) ? 1.0 : 0.0;
  }
  __syncwarp();
  for (int pc = 0; pc < 5; ++pc) {
    int pr = pc;
    double mag = fabs(m[pr * 5 + pc]);
    for (int q = pc + 1; q < 5; ++q)
      if (fabs(m[q * 5 + pc]) > mag) { mag = fabs(m[q * 5 + pc]); pr = q; }
    if (!isfinite(mag) || mag <= 100.0 * kEps) return false;
    __syncwarp();
    if (pr != pc && lane < 5) {
      double t = m[pr * 5 + lane]; m[pr * 5 + lane] = m[pc * 5 + lane]; m[pc * 5 + lane] = t;
      t = inv[pr * 5 + lane]; inv[pr * 5 + lane] = inv[pc * 5 + lane]; inv[pc * 5 + lane] = t;
    }
    __syncwarp();
    const double piv = m[pc * 5 + pc];
    __syncwarp();
    if (lane < 5) {
      m[pc * 5 + lane] /= piv;
      inv[pc * 5 + lane] /= piv;
    }
    __syncwarp();
    const double f = on ? m[r * 5 + pc] : 0.0;
    __syncwarp();
    if (on && r != pc) {
      m[lane] -= f * m[pc * 5 + c];
      inv[lane] -= f * inv[pc * 5 + c];
    }
    __syncwarp();
  }
  return true;
}

// computeCharacteristics (BoundaryConditions.cpp:152-280), closed form.
// Called by a whole warp; every lane returns the status.
__device__ int characteristics(const double *state, const double *m10, double M, double gamma,
                               Char &ch, CharWork &wk) {
  const int lane = threadIdx.x & 31;
  const bool on = lane < 25;
  const double rho = state[0], V = state[2], W = state[3], T = state[4];
  if (!isfinite(rho) || !isfinite(V) || !isfinite(W) || !isfinite(T) ||
      !(rho > 0.0) || !(T > 0.0)) {
    return 1;  // InvalidInput
  }
  const double mag = sqrt(m10[0] * m10[0] + m10[1] * m10[1]);
  if (!isfinite(mag) || mag <= 100.0 * kEps) {
    return 2;  // SingularMetric
  }
  const double ny = m10[0] / mag, nz = m10[1] / mag;
  const double Pe = 1.0 / (gamma * M * M);
  const double g2 = 1.0 / ((gamma - 1.0) * M * M);
  const double c = sqrt(T) / M;
  const double un = ny * V + nz * W;
  const double speed[5] = {un - c, un, un, un, un + c};
  // R: columns -acoustic, entropy, streamwise, tangential, +acoustic
  const double th = (gamma - 1.0) * T / rho;
  const double cols[5][5] = {{1.0, 0.0, -c * ny / rho, -c * nz / rho, th},
                             {1.0, 0.0, 0.0, 0.0, -T / rho},
                             {0.0, 1.0, 0.0, 0.0, 0.0},
                             {0.0, 0.0, -nz, ny, 0.0},
                             {1.0, 0.0, c * ny / rho, c * nz / rho, th}};
  if (lane == 0)
    for (int r = 0; r < 5; ++r)
      for (int mm = 0; mm < 5; ++mm) wk.R[r * 5 + mm] = cols[mm][r];
  __syncwarp();
  if (!invert5(wk.R, wk.m, ch.Rinv)) return 6;  // SingularEigenvectors
  // Gamma (LNSCoefficients.cpp:141-146) is diag(1, rho, rho, rho, g44)
  // plus Gamma[4][0] = -Pe T; its inverse in closed form.
  const double g44 = rho * g2 - Pe * rho;
  if (!isfinite(g44) || fabs(g44) <= 100.0 * kEps) return 6;
  if (on) {
    double g = 0.0;
    if (lane == 0) g = 1.0;
    if (lane == 6 || lane == 12 || lane == 18) g = 1.0 / rho;
    if (lane == 24) g = 1.0 / g44;
    if (lane == 20) g = Pe * T / g44;
    wk.Ginv[lane] = g;
  }
  __syncwarp();
  // P = R^-1 Gamma^-1, and the self-check R R^-1 = I to rounding
  double worst = 0.0;
  if (on) {
    const int r = lane / 5, q = lane % 5;
    double s = 0.0;
    for (int k = 0; k < 5; ++k) s += ch.Rinv[r * 5 + k] * wk.Ginv[k * 5 + q];
    ch.P[lane] = s;
    s = 0.0;
    for (int k = 0; k < 5; ++k) s += wk.R[r * 5 + k] * ch.Rinv[k * 5 + q];
    worst = fmax(worst, fabs(s - (r == q ? 1.0 : 0.0)));
  }
  for (int o = 16; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
  if (!(worst <= 1e-10)) return 6;
  // condition number in the infinity norm: one lane per row and matrix
  if (lane < 10) {
    const double *a = (lane < 5 ? wk.R : ch.Rinv) + lane % 5 * 5;
    double s = 0.0;
    for (int c2 = 0; c2 < 5; ++c2) s += fabs(a[c2]);
    wk.cond[lane / 5][lane % 5] = s;
  }
  __syncwarp();
  double nr = 0.0, ni = 0.0;
  for (int r = 0; r < 5; ++r) {
    nr = fmax(nr, wk.cond[0][r]);
    ni = fmax(ni, wk.cond[1][r]);
  }
  const double cond = nr * ni;
  if (!isfinite(cond) || cond > 1.0e12) return 7;  // IllConditionedEigenvectors
  if (lane == 0) {
    ch.cond = cond;
    double smax = 1.0;
    for (int mm = 0; mm < 5; ++mm) smax = fmax(smax, fabs(speed[mm]));
    const double tol = 1000.0 * kEps * smax;
    ch.n_in = 0;
    ch.n_neutral = 0;
    for (int mm = 0; mm < 5; ++mm) {
      ch.incoming[mm] = speed[mm] < -tol;
      ch.n_in += ch.incoming[mm];
      ch.n_neutral += fabs(speed[mm]) <= tol;
    }
  }
  return 0;
}

// One CTA per far-field node j; its first warp finds the characteristics.
__global__ void k_farfield(int ny, int nz, int S, double M, double gamma,
                           const double *__restrict__ base,
                           const double *__restrict__ met,
                           const int *__restrict__ col, double2 *__restrict__ A,
                           double2 *__restrict__ B, int *modes, double *cond,
                           int *status) {
  __shared__ Char ch;
  __shared__ CharWork wk;
  const int j = blockIdx.x;
  const int nn = ny * nz;
  const int node = j * ny + ny - 1;
  if (threadIdx.x < 32) {
    double state[5], m10[10];
    for (int f = 0; f < 5; ++f) state[f] = base[f * (size_t)nn + node];
    for (int k = 0; k < 10; ++k) m10[k] = met[k * (size_t)nn + node];
    const int ok = characteristics(state, m10, M, gamma, ch, wk);
    if (threadIdx.x == 0) ch.ok = ok;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (ch.ok) atomicMax(status + ST_CHAR, ch.ok);
    modes[j * 2 + 0] = ch.ok ? 0 : ch.n_in;
    modes[j * 2 + 1] = ch.ok ? 0 : ch.n_neutral;
    cond[j] = ch.ok ? 0.0 : ch.cond;
  }
  __syncthreads();
  if (ch.ok) return;
  // A rows of the node: blocks k, columns c.
  for (int x = threadIdx.x; x < S * 5; x += blockDim.x) {
    const int k = x / 5, c = x % 5;
    const long long blk = (long long)node * S + k;
    double2 old[5];
    for (int s = 0; s < 5; ++s) old[s] = A[blk * 25 + s * 5 + c];
    const bool own = col[blk] == node;
    for (int mm = 0; mm < 5; ++mm) {
      double2 v = make_double2(0.0, 0.0);
      if (ch.incoming[mm]) {
        if (own) v.x = ch.Rinv[mm * 5 + c];
      } else {
        for (int s = 0; s < 5; ++s) {
          const double p = ch.P[mm * 5 + s];
          if (p == 0.0) continue;
          v.x += p * old[s].x;
          v.y += p * old[s].y;
        }
      }
      A[blk * 25 + mm * 5 + c] = v;
    }
  }
  if (threadIdx.x < 5) {
    const int c = threadIdx.x;
    double2 old[5];
    for (int s = 0; s < 5; ++s) old[s] = B[(long long)node * 25 + s * 5 + c];
    for (int mm = 0; mm < 5; ++mm) {
      double2 v = make_double2(0.0, 0.0);
      if (!ch.incoming[mm])
        for (int s = 0; s < 5; ++s) {
          const double p = ch.P[mm * 5 + s];
          if (p == 0.0) continue;
          v.x += p * old[s].x;
          v.y += p * old[s].y;
        }
      B[(long long)node * 25 + mm * 5 + c] = v;
    }
  }
}

}  // namespace

int run_bc(tlr_ctx *ctx, tlr_bc_diag *diag) {
  const long long nB = (long long)ctx->nn * 25;
  int rc = pinned_words(ctx);
  if (!rc) rc = arrival_counters(ctx, 1);
  if (rc) return rc;
  // partial sums of the interior and the boundary rows, in one array
  int sms = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int row_entries = ctx->S * 25, copy_ctas = std::min(ctx->nn, 8 * sms);
  if (!ctx->bc_part)
    TLR_CUDA(ctx, cudaMalloc(&ctx->bc_part, sizeof(double) * (copy_ctas + 2 * ctx->nz)));
  TLR_CUDA(ctx, cudaMemsetAsync(ctx->status, 0, sizeof(int) * ST_COUNT, ctx->stream));
  { k_negate_copy<<<copy_ctas, 256, 0, ctx->stream>>>(ctx->nn, ctx->ny, row_entries, ctx->L, ctx->A,
                                                      ctx->bc_part); count_launches(); }
  TLR_CUDA(ctx, cudaMemcpyAsync(ctx->B, ctx->M, sizeof(double2) * nB,
                                cudaMemcpyDeviceToDevice, ctx->stream));
  const long long wall = (long long)ctx->nz * ctx->S * 20;
  { k_wall<<<blocks_for(wall, 256), 256, 0, ctx->stream>>>(ctx->ny, ctx->nz, ctx->S,
                                                         ctx->col, ctx->A, ctx->B); count_launches(); }
  { k_farfield<<<ctx->nz, 64, 0, ctx->stream>>>(
      ctx->ny, ctx->nz, ctx->S, ctx->recipe.mach, ctx->recipe.gamma, ctx->base,
      ctx->metrics, ctx->col, ctx->A, ctx->B, ctx->bc_modes, ctx->bc_cond,
      ctx->status); count_launches(); }
  { k_boundary_norm<<<2 * ctx->nz, 256, 0, ctx->stream>>>(
      ctx->ny, ctx->nz, row_entries, ctx->A, ctx->bc_part + copy_ctas, ctx->bc_part,
      copy_ctas + 2 * ctx->nz, ctx->pin + PIN_NORMS, ctx->kv_ctr); count_launches(); }
  TLR_CUDA(ctx, cudaGetLastError());
  if ((rc = frobenius_async(ctx, ctx->B, nB, ctx->pin + PIN_NORMS + 1))) return rc;
  int st[ST_COUNT];
  std::vector<int> modes(ctx->nz * 2);
  std::vector<double> cond(ctx->nz);
  TLR_CUDA(ctx, cudaMemcpyAsync(st, ctx->status, sizeof(st), cudaMemcpyDeviceToHost,
                                ctx->stream));
  TLR_CUDA(ctx, cudaMemcpyAsync(modes.data(), ctx->bc_modes, sizeof(int) * ctx->nz * 2,
                                cudaMemcpyDeviceToHost, ctx->stream));
  TLR_CUDA(ctx, cudaMemcpyAsync(cond.data(), ctx->bc_cond, sizeof(double) * ctx->nz,
                                cudaMemcpyDeviceToHost, ctx->stream));
  TLR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (st[ST_CHAR]) {
    char buf[128];
    snprintf(buf, sizeof(buf),
             "Far-field characteristic decomposition failed (status %d)", st[ST_CHAR]);
    return fail(ctx, TLR_ERR_CHARACTERISTIC, buf);
  }
  tlr_bc_diag d{};
  d.wall_nodes = ctx->nz;
  d.farfield_nodes = ctx->nz;
  d.min_incoming_per_node = 5;
  for (int j = 0; j < ctx->nz; ++j) {
    d.incoming_modes += modes[j * 2];
    d.neutral_modes += modes[j * 2 + 1];
    d.min_incoming_per_node = std::min(d.min_incoming_per_node, modes[j * 2]);
    d.max_incoming_per_node = std::max(d.max_incoming_per_node, modes[j * 2]);
    d.max_eigenvector_condition = std::max(d.max_eigenvector_condition, cond[j]);
  }
  d.max_characteristic_imaginary = 0.0;
  d.eigen_frobenius_norm = ctx->pin[PIN_NORMS];
  d.eigen_mass_frobenius_norm = ctx->pin[PIN_NORMS + 1];
  if (diag) *diag = d;
  return TLR_OK;
}

}  // namespace tlr
