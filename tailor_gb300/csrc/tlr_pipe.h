// tlr_pipe.h -- pipelined refined operator applications of the mixed form.
//
// Shift-and-invert Arnoldi needs x = OP v_j, OP = K^-1 B, to a residual of
// 1e-12 from a factor that contracts an error by 1e-5 or so per triangular
// solve: three dependent solves per application when each starts from
// nothing.  The applications are not independent, though: v_{j+1} is a
// combination of OP v_j and the basis, so OP v_{j+1} is one of OP^2 v_j and
// the (known) images of the basis.  The driver therefore carries
//   x ~ OP v_j,  y ~ OP^2 v_j,  u ~ OP^3 v_j
// and every triangular solve takes three right-hand sides at once -- the
// residuals of x and of y, and B y -- reading the factor once.  When x is
// accepted and v_{j+1} known, the same combination that made v_{j+1} out of
// x makes the next x out of y and the next y out of u; the new x usually
// needs one correction only.  x is accepted on the same residual as before
// (||B v - K x|| <= 1e-12 ||B v||, A x in float-float), so a poor guess
// costs another round and no accuracy; and not before it is as good as three
// corrections from nothing are (Solver::pipe_tol), which are mostly far better
// than that limit: accepted at the limit alone, eigenvalues of pencils of a few
// rows lost up to two digits for 1 to 3% of the time (60 x 32: 108.9 against 112.1
// ms, 300 x 192: 898 against 910 ms).  A step's second and later rounds refine
// u too (against B y + sigma B u in FP32), which makes the next step's y better:
// 192 -> 175 rounds at 300 x 192, 196 -> 175 at 200 x 128, 353 -> 348 at 60 x 32.
// Measured rounds per application: 1.17 (60 x 32), 1.21 (100 x 50), 1.32 (300 x
// 192) and 1.34 (200 x 128, complex target; its factor contracts by 3e-5 only),
// against three dependent solves.  A pass of a point with these applications
// alone, before and after: 221 -> 161 ms at 60 x 32, 227 -> 173 ms at 100 x 50,
// 643 -> 594 ms at 200 x 128, 1465 -> 1231 ms at 300 x 192; refining u took
// another 30 of 495 ms at 200 x 128 and 50 of 1048 ms at 300 x 192.
#pragma once

#include "tlr_internal.h"

namespace tlr {

struct Pipe {
  long long n = 0;        // scalar unknowns, 5 nn
  int nn = 0, ncv = 0, ldh = 0, sms = 1;
  float4 *vff = nullptr;  // the basis as FP32 hi/lo pairs, (ncv + 1) x n
  // x (held in FP64 too, by the caller) and y the same way, interleaved [n][2]
  float4 *xyff = nullptr;
  float2 *B32 = nullptr;  // B in FP32
  double2 *b = nullptr, *tx = nullptr, *ty = nullptr;
  float2 *by32 = nullptr; // B y, the right-hand side of u
  float2 *u32 = nullptr, *tu32 = nullptr;  // u and its target B y + sigma B u
  double2 *H = nullptr;   // (ncv + 1) x ncv projected matrix, ld ldh
  float4 *g = nullptr;    // combination coefficients, 2 x ldh
  double *bpart = nullptr, *rpart = nullptr;  // per-CTA partial sums of squares
  int *arrived = nullptr; // CTAs done with the acceptance residual
  double2 *hup = nullptr; // pinned stage of H
};

// all buffers, or none and TLR_ERR_NOMEM
int pipe_alloc(tlr_ctx *ctx, Pipe &p, int ncv);
void pipe_free(Pipe &p);
// Begin with v (= basis vector 0): x = y = u = 0.
int pipe_start(tlr_ctx *ctx, Pipe &p, const double2 *v, double2 *x);
// basis columns 0 .. nk-1 into p.vff (after a restart)
int pipe_split_basis(tlr_ctx *ctx, Pipe &p, const double2 *V, int nk);
// upload the leading l columns of the restarted projected matrix
int pipe_upload_h(tlr_ctx *ctx, Pipe &p, int l);
// x (holding the orthogonalised w) -> v_{j+1} = w / beta and the next x, y,
// targets and right-hand side; rhs: 3 x n, its third vector holds u
int pipe_shift(tlr_ctx *ctx, Pipe &p, int j, const double *beta, double sr, double si,
               double2 *x, double2 *vnew, const float2 *rhs);
// rhs = the residuals of x and y, and B y or (refine_u, in a step's second and
// later rounds) the residual of u; err: set when a bounded wait of the kernel
// ran out
int pipe_residuals(tlr_ctx *ctx, Pipe &p, float2 *rhs, bool refine_u, int *err);
// x += rhs(0), y += rhs(1), u = rhs(2) (correct 1) or u += rhs(2) (correct 2,
// rhs(2) then holds u), and the targets of the new iterates; correct 0: the
// targets only
int pipe_targets(tlr_ctx *ctx, Pipe &p, double sr, double si, double2 *x, float2 *rhs,
                 int correct);
// out[0] = ||B v - K x||, out[1] = ||B v|| (out: pinned host memory)
int pipe_accept(tlr_ctx *ctx, Pipe &p, double *out, int *err);

}  // namespace tlr
