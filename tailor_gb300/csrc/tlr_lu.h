// tlr_lu.h -- device multifrontal factorisation of K = A_bc - sigma B_bc.
#pragma once

#include <vector>

#include "tlr_internal.h"
#include "tlr_symbolic.h"

namespace tlr {

struct DevFront {
  long long off, toff, cmap_off;
  int p, m, parent, node_off;
};

// What a complex128 solve step needs of a front, in the levels' order.
struct StepFront {
  long long off, toff, inv;  // pool, work and diagonal-block offsets
  int p, m, node_off, pad;
};


constexpr int kOzPanel = 32;  // panel columns of the sliced FP64 Schur update

// One 32-column pass of a product of the complex128 rewrite, column-major:
// kind 0 L' (A in the pool, B in linv), 1 U' (A in uinv, B in the pool).
struct OzJob {
  long long a, b, c;
  int lda, ldb, ldc, rows, cols, kw, kind, pad;
};

constexpr int kOzPasses = 4;  // 128-row diagonal blocks, 32 columns per pass

// A batch of such passes, ordered by pass; pass[q]: its first output tile
struct OzBatch {
  int job_off = 0, jobs = 0, prefix_off = 0, atiles = 0, btiles = 0;
  int max_len = 0;  // longest side of a product
  int pass[kOzPasses + 1] = {};
};

// Default of Factor::cluster_rows (the automatic cluster-panel choice).
constexpr int kClusterPanelRows = 256;

// One tensor-core product C(rows, cols) -= F(rows, K) F(K, cols) inside a
// front (m x m at off in the pool): rows [r0, r1), columns [c0, c1), inner
// range [k0, k0 + kw).
struct TcJob {
  long long off;
  int m, k0, kw, r0, r1, c0, c1, pad;
};

// A batch of such products run by one launch: offsets of its jobs and of
// the per-job prefixes (jobs + 1 each) of its output tiles and of the
// operand tiles.
struct TcBatch {
  int job_off = 0, jobs = 0, prefix_off = 0, pa_off = 0, pb_off = 0;
  int tiles = 0, atiles = 0, btiles = 0;
};

// Work item of the inverse-form solves (tlr_inv.cu): up to 32 rows of a
// front times a range of columns.
struct SvItem {
  long long a;     // pool offset of the item's first entry
  int ld, rows, cols;
  int vec;         // work index of the first vector entry
  int piv;         // leading columns whose vector entries are pivot rows' values
  int out;         // work index of the first row
  int tile;        // row tile of the launch (partial sums and counter)
  int split, nsplit;
  int kind;        // 0 forward pivot rows, 1 forward border rows, 2 backward
};

struct Step {  // one panel step of one level
  int nf, max_m, max_b, max_ext, prefix_off, tiles;
  // complex64: per-front prefixes (nf + 1 each, in the schedule) of the
  // step's 128-row L21 tiles and 64-column U12 tiles, and their totals
  // (complex128 in 32-column panels: 128-row and 32-column tiles of the
  // sliced update, with the prefix of its 128 x 32 output tiles)
  int pa_off = 0, pb_off = 0, atiles = 0, btiles = 0;
  int oz_prefix_off = 0, oz_tiles = 0;
};

struct Level {
  int nfronts = 0, fronts_off = 0, max_m = 0;
  int sf_off = 0;  // first entry of the level in Factor::d_sfronts
  int pmax = 0, bmax = 0, nck_b = 1;  // backward border GEMV chunks
  int kids[2] = {0, 0}, kids_off[2] = {0, 0}, kids_maxb[2] = {0, 0};
  long long entry_begin = 0, entry_end = 0, pool_begin = 0, pool_end = 0;
  std::vector<Step> steps;
  std::vector<int> blk_nf;    // blk_nf[b]: fronts of the level with p > b sw
  std::vector<int> fwd_rows;  // rows below block b, largest over those fronts
  // dependency-driven solve of the level (levels with two or more blocks):
  // forward and backward 32-row tiles in dependency order, and their
  // counters (4 + nfronts * maxblk each)
  bool wave = false;
  int maxblk = 0;
  long long wf_off = 0, wb_off = 0;
  int wf_n = 0, wb_n = 0;
  long long wcf_off = 0, wcb_off = 0;
  int wctr_n = 0;
  // inverse-form solve: items of the forward and of the backward launch
  int if_off = 0, if_n = 0, ib_off = 0, ib_n = 0;
  bool if_small = false, ib_small = false;  // launch-bound (tlr_inv.cu)
};

// One phase of the persistent solve: a kind of work item over a level's
// fronts (fl_off into the level schedule), block b, and an nx x ny x nz
// item grid (the CTA grid of the equivalent separate launch).
struct Phase {
  int type, fl_off, b, nx, ny, nz, nck, pmax;
};

struct Factor {
  Symbolic sym;
  int prec = 0;  // 0: complex128 fronts, 1: complex64 fronts
  // Schur updates on the tensor cores: tcgen05 (3xTF32) for complex64
  // fronts, DMMA (FP64 mma.sync) for complex128 fronts; else CUDA cores
  bool tensor_cores = true;
  // panel steps with at least this many fully summed rows left run over an
  // 8-CTA cluster (INT_MAX: never)
  int cluster_rows = kClusterPanelRows;
  int *d_tc_err = nullptr;   // set by a tensor-core kernel whose wait timed out
  // complex64 Schur updates: operand plane images of one panel step, read
  // by bulk copies (tc_bulk), else staged by every tile's own threads
  bool tc_bulk = true;
  // bulk kernel: 2 persistent warp-specialised (default), 0 one tile per CTA
  // with three stages / two CTAs per SM, 1 two stages / three CTAs per SM
  int tc_variant = 2;
  // scratch, also of the inversion and of the sliced products
  unsigned char *tc_planes = nullptr;
  size_t planes_bytes = 0;
  // at least `bytes` of tc_planes (contents are lost); TLR_ERR_NOMEM
  int reserve_planes(tlr_ctx *ctx, size_t bytes);
  // complex128 Schur updates by exact integer slices on the tensor cores
  // (tlr_oz.cu), with 32-column panels
  bool sliced = false;
  // its products of the factor rewrite, in batches
  std::vector<OzBatch> oz_batches;
  std::vector<OzJob> oz_jobs;
  std::vector<int> oz_prefix;
  OzJob *d_oz_jobs = nullptr;
  int *d_oz_prefix = nullptr;
  size_t oz_bytes = 0;      // operand images of the largest launch
  int oz_fronts = 1;        // products of the largest launch
  // whether the buffers of the slices exist; or there is no memory
  // for them: CUDA cores then
  bool oz_ok = false, oz_failed = false;
  int build_oz(tlr_ctx *ctx);
  StepFront *d_sfronts = nullptr;  // complex128: fronts of every level in order
  int *d_rowexp = nullptr;
  int w = 32;    // panel width
  int sw = 128;  // rows of a diagonal block of the solves (128 or 256)
  int ring_slack = kRingSlackDefault;  // nested-dissection ring slack, percent
  std::vector<Level> levels;
  void *pool = nullptr, *work = nullptr, *work2 = nullptr, *vec_a = nullptr;
  DevFront *d_fronts = nullptr;
  AsmEntry *d_entries = nullptr;
  int *d_cmap = nullptr, *d_nodes = nullptr, *d_ipiv = nullptr, *d_perm = nullptr;
  int *d_sched = nullptr, *d_pert = nullptr;
  int2 *d_cinv = nullptr;  // child border rows mapped onto each front row
  // sw x sw diagonal blocks of every pivot block: inv(L_bb), inv(U_bb)
  // (scratch of the factor rewrite) and D_b = inv(U_bb) inv(L_bb)
  void *linv = nullptr, *uinv = nullptr, *dmat = nullptr;
  long long *d_inv_off = nullptr;
  int2 *d_inv_blocks = nullptr;
  int4 *d_ltiles = nullptr, *d_utiles = nullptr;
  // the same rewrite on the tensor cores (complex64, 256-row blocks, when
  // the Schur updates run there too): 128-row L tiles, 64-column U tiles
  int4 *d_ltiles_tc = nullptr, *d_utiles_tc = nullptr;
  long long n_ltiles_tc = 0, n_utiles_tc = 0;
  int n_inv_blocks = 0;
  // Inverse form (complex64, 256-row blocks, tensor cores): the pivot
  // blocks are inverted past the diagonal blocks, so a front needs one
  // product each way (tlr_inv.cu) instead of one step per diagonal block.
  bool inverse = false;            // the form of the present factor
  // whether the structures of the form exist (made by the first factorisation
  // that uses them), or there is no memory for them: block steps then
  bool inverse_ok = false, inverse_failed = false;
  std::vector<TcBatch> inv_batches;
  TcJob *d_inv_jobs = nullptr;
  int *d_inv_prefix = nullptr;
  int4 *d_gtiles = nullptr;        // 64-column tiles of the D_b row scaling
  long long n_gtiles = 0;
  SvItem *d_items = nullptr;
  int item_cols = 0;               // largest column range of an item
  int *d_uidx = nullptr;           // unknown of every front row (border: ancestors')
  int *d_gsrc = nullptr;           // right-hand side entry of every pivot row
  int max_split_tiles = 0, max_split = 1;
  float2 *split_part = nullptr;    // partial sums of split row tiles
  int *split_ctr = nullptr;
  bool use_inverse() const {
    return prec == 1 && sw == 256 && tensor_cores && !persistent && !inverse_failed;
  }
  int build_inverse(tlr_ctx *ctx);
  void free_inverse();
  int invert_pivots(tlr_ctx *ctx);
  template <int NR> int solve_inverse(tlr_ctx *ctx, float2 *x, float2 *W, float2 *W2);
  long long inv_elems = 0, n_ltiles = 0, n_utiles = 0;
  // sliced rewrite: leading L and U tiles that stay in FP64 (the D_b, blocks of
  // fewer than 32 columns)
  long long n_ltiles64 = 0, n_utiles64 = 0;
  cudaGraphExec_t graph_exec = nullptr;  // captured solve, replayed per call
  // persistent solve: one cooperative launch per solve over a phase table
  bool persistent = false;
  int persist_grid = 0;                  // CTAs (0: two per SM, capped by occupancy)
  Phase *d_phases = nullptr;
  int nphases = 0;
  unsigned *d_barrier = nullptr;
  int *d_solve_err = nullptr;
  long long graph_kernels = 0;           // kernel nodes of graph_exec
  // levels with several diagonal blocks per front solved by one dependency-
  // driven launch each way (false, the default: one launch per block step)
  bool wave = false;
  int4 *d_wave_tiles = nullptr;
  int *d_wave_ctr = nullptr;
  int wave_grid = 0;                     // CTAs of a wave launch (at most)
  double2 *d_partial = nullptr;
  int perturbed = 0;
  // CUDA events around every replayed solve graph (device time of the
  // triangular solves); collected and reset by take_solve_time()
  std::vector<cudaEvent_t> ev_pool;
  size_t ev_used = 0;
  double take_solve_time(int *count);
  bool factored = false;
  double sigma_re = 0.0, sigma_im = 0.0;

  // Multi-RHS solves (complex64 factors): nr vectors at once, every factor
  // tile read once for all of them.  Buffers sized for multi_cap vectors,
  // allocated on first use; one captured graph per vector count.
  static constexpr int kMaxRhs = 8;
  int multi_cap = 0;
  long long partial_stride = 0;   // border partial sums of one vector
  void *work_m = nullptr, *work2_m = nullptr, *vec_m = nullptr;
  double2 *partial_m = nullptr;
  cudaGraphExec_t graph_m[kMaxRhs + 1] = {};
  long long graph_m_kernels[kMaxRhs + 1] = {};
  // In-place x <- K^-1 x for nr vectors at x + r * 5 nn (complex64 only,
  // 2 <= nr <= kMaxRhs; events a/b, when given, bracket the triangular
  // solve and mark a capture into the caller's graph: no graph of our own).
  int solve_multi(tlr_ctx *ctx, void *x, int nr, cudaEvent_t a = nullptr,
                  cudaEvent_t b = nullptr, bool capture = false);
  // allocate the multi-vector buffers (outside any stream capture)
  int solve_multi_prepare(tlr_ctx *ctx);
  // Enqueue the solve of the nr right-hand sides in vec_m, in place, for
  // capture into a caller's graph (solve_multi_prepare first).  Block steps
  // with the dependency-driven level launches (wave) take one vector at a
  // time; the bits are the same.
  int enqueue_multi(tlr_ctx *ctx, int nr, cudaEvent_t a, cudaEvent_t b);
  template <int SW, int NR> int solve_impl_m(tlr_ctx *ctx);
  int solve_impl_m_dispatch(tlr_ctx *ctx, int nr);

  int setup(tlr_ctx *ctx, int precision, int leaf, int solve_block = 0, int panel_width = 0,
            int ring_slack_percent = 0);
  void release();
  // What only some forms of the factor need, on the first factorisation in that
  // form; without the memory for it the factor takes the form that does without.
  // (factor() does this itself, but not outside a caller's timing.)
  int prepare(tlr_ctx *ctx);
  int factor(tlr_ctx *ctx, double sr, double si, double tiny);
  // In-place x <- K^-1 x on a device vector in the factor's precision.
  int solve(tlr_ctx *ctx, void *x);
  // Enqueue one solve's kernels on the context stream without a graph
  // (for capture into a caller's graph); events a/b, when given, bracket
  // the triangular solve.
  int enqueue_solve(tlr_ctx *ctx, void *x, cudaEvent_t a, cudaEvent_t b);

  template <class C> int factor_impl(tlr_ctx *ctx, double sr, double si, double tiny);
  template <class C, int SW> int solve_impl(tlr_ctx *ctx, void *x);
  template <class C, int SW> int rewrite_factors(tlr_ctx *ctx);
  template <class C, int SW> int solve_persistent(tlr_ctx *ctx);
  int build_phases(tlr_ctx *ctx);
  // error raised inside a persistent solve since the last call (a grid
  // barrier that gave up); resets the flag
  int take_solve_error(tlr_ctx *ctx);
};

}  // namespace tlr
