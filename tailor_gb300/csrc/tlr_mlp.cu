// tlr_mlp.cu -- the learned shift / start-vector proposal: a small MLP
// (inputs -> depth x width SiLU hidden layers -> outputs) trained and
// evaluated on the GPU by the kernels in this file.  No reference
// counterpart: the reference always starts Krylov-Schur from SLEPc's
// random vector at the configured target (EigenSolver.cpp:46-72).
//
// Parameters are FP32, flat: for each layer l, W_l [out][in] row-major then
// b_l [out].  Training: mean-squared error, full forward/backward per
// minibatch, Adam.  Inference: FP32 or BF16 weights/activations with FP32
// accumulation.
#include <cuda_bf16.h>

#include <cmath>
#include <vector>

#include "tlr_internal.h"

struct tlr_mlp {
  int n_in = 0, width = 0, depth = 0, n_out = 0, n_layers = 0;
  std::vector<int> fan_in, fan_out;
  std::vector<long long> w_off, b_off;
  long long n_params = 0;
  float *params = nullptr, *grads = nullptr, *m1 = nullptr, *m2 = nullptr;
  __nv_bfloat16 *params16 = nullptr;
  float *act = nullptr, *pre = nullptr, *dact = nullptr;  // [layers+1][batch][maxw]
  int cap = 0, maxw = 0;
  float *xbuf = nullptr, *ybuf = nullptr, *loss = nullptr;
  float *wpart = nullptr;  // row-split partial parameter gradients: max_split x n_params
  int max_split = 1;
  float *lpart = nullptr;  // per-CTA partial losses
  int *lctr = nullptr;     // CTAs done with the loss
  long long adam_t = 0;
  int sms = 1;
  cudaStream_t stream = nullptr;
};

namespace tlr {
namespace {

constexpr int kT = 32;

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = 1.f / (1.f + __expf(-z));
  return s * (1.f + z * (1.f - s));
}

constexpr int kMaxSplit = 16;   // row ranges of a weight gradient
constexpr int kLossCtas = 64;

template <int N>
struct __align__(4 * N) Vec {
  float v[N];
};

// The three products of a layer in FP32 over kG x kG tiles: 256 threads of (kG /
// 16)^2 results, inner chunks of 1024 / kG in shared memory (inner index leading),
// the next chunk's loads in flight during the present one's FMAs.  32 x 32 tiles with a
// result per thread were bound by shared-memory reads (two per FMA), and a weight
// gradient by its 64 CTAs of 2048 serial rows.  64 x 64 ones are bound by the latency
// of a chunk on one CTA per SM (2048 rows: 23 us, shared memory 42% and FMAs 22%
// busy, half of the stalls for global loads).  Small batches are bound by the latency of the chunks, so they take
// smaller tiles and longer chunks (layer_tile).  Every result is the sum over the
// inner index in order, whatever the tile.
//   kFwd:    Y[r][c] = act(sum_k X[r][k] W[c][k] + b[c]), Z the pre-activation
//   kData:   dX[r][c] = sum_k dZ[r][k] W[k][c] (times silu'(Z[r][c]) with Z)
//   kWeight: dW[r][c] = sum_k dZ[k][r] X[k][c], db[r] = sum_k dZ[k][r] over the
//            rows k of range blockIdx.z
enum LayerProduct { kFwd, kData, kWeight };
constexpr int kGK(int g) { return 1024 / g; }  // four elements of each operand per thread

template <int MODE, int kG>
__global__ void __launch_bounds__(256)
    k_layer(int M, int N, int K, const float *__restrict__ A, int lda,
            const float *__restrict__ B, int ldb, const float *__restrict__ bias,
            float *__restrict__ Z, float *__restrict__ C, int ldc, int act, int krange,
            long long zstride, float *__restrict__ db) {
  constexpr int kK = kGK(kG), kR = kG / 16;  // inner chunk, results per thread and side
  constexpr int kQ = kK / 4, kL = kG / 4;    // groups of four along the inner index, of lines
  __shared__ __align__(16) float as[kK][kG + 4], bs[kK][kG + 4];
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int r0 = blockIdx.y * kG, c0 = blockIdx.x * kG;
  const int ka = MODE == kWeight ? blockIdx.z * krange : 0;
  const int kb = MODE == kWeight ? min(K, ka + krange) : K;
  // element (line, k) of an operand whose inner index is contiguous (thread:
  // one line, four k) or whose lines are (one k, four lines)
  constexpr bool aInner = MODE != kWeight, bInner = MODE == kFwd;
  float ra[4], rb[4];
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int la = aInner ? tid / kQ : tid % kL * 4 + q;
      const int k1 = k0 + (aInner ? tid % kQ * 4 + q : tid / kL);
      ra[q] = r0 + la < M && k1 < kb
                  ? A[aInner ? (long long)(r0 + la) * lda + k1 : (long long)k1 * lda + r0 + la]
                  : 0.f;
      const int lb = bInner ? tid / kQ : tid % kL * 4 + q;
      const int k2 = k0 + (bInner ? tid % kQ * 4 + q : tid / kL);
      rb[q] = c0 + lb < N && k2 < kb
                  ? B[bInner ? (long long)(c0 + lb) * ldb + k2 : (long long)k2 * ldb + c0 + lb]
                  : 0.f;
    }
  };
  float acc[kR][kR] = {};
  float sb = 0.f;  // kWeight: this thread's share of db (a thread per row, first column)
  load(ka);
  for (int k0 = ka; k0 < kb; k0 += kK) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (aInner) as[tid % kQ * 4 + q][tid / kQ] = ra[q];
      else as[tid / kL][tid % kL * 4 + q] = ra[q];
      if (bInner) bs[tid % kQ * 4 + q][tid / kQ] = rb[q];
      else bs[tid / kL][tid % kL * 4 + q] = rb[q];
    }
    __syncthreads();
    if (k0 + kK < kb) load(k0 + kK);
#pragma unroll
    for (int k = 0; k < kK; ++k) {
      const auto a = *reinterpret_cast<const Vec<kR> *>(&as[k][ty * kR]);
      const auto b = *reinterpret_cast<const Vec<kR> *>(&bs[k][tx * kR]);
#pragma unroll
      for (int i = 0; i < kR; ++i)
#pragma unroll
        for (int j = 0; j < kR; ++j) acc[i][j] = fmaf(a.v[i], b.v[j], acc[i][j]);
    }
    if (MODE == kWeight && blockIdx.x == 0 && tid < kG)
#pragma unroll
      for (int k = 0; k < kK; ++k) sb += as[k][tid];
    __syncthreads();
  }
  if (MODE == kWeight) {
    C += blockIdx.z * zstride;
    if (blockIdx.x == 0 && tid < kG && r0 + tid < M) db[blockIdx.z * zstride + r0 + tid] = sb;
  }
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    const int r = r0 + ty * kR + i;
    if (r >= M) break;
#pragma unroll
    for (int j = 0; j < kR; ++j) {
      const int c = c0 + tx * kR + j;
      if (c >= N) break;
      const long long o = (long long)r * ldc + c;
      float v = acc[i][j];
      if (MODE == kFwd) {
        v += bias[c];
        if (Z) Z[o] = v;
        if (act) v = silu(v);
      } else if (MODE == kData && Z) {
        v *= silu_grad(Z[o]);
      }
      C[o] = v;
    }
  }
}

// The tile of a product with m x n results in z ranges: the largest of 64, 32 and 16
// that gives every other SM a CTA.  Gradients of the 256-wide network, in ms, for
// batches of 24, 192, 512 and 2048 rows: 0.148, 0.188, 0.198, 0.302, against 0.229,
// 0.295, 0.286, 0.312 with 64 x 64 tiles everywhere, 0.159, 0.187, 0.198, 0.341 with 32 x
// 32 and 0.146, 0.188, 0.274, 0.635 with 16 x 16.
int layer_tile(int m, int n, int z, int sms) {
  for (int g = 64; g > 16; g /= 2)
    if (2LL * blocks_for(m, g) * blocks_for(n, g) * z >= sms) return g;
  return 16;
}

template <int MODE>
void launch_layer(const tlr_mlp *m, int M, int N, int K, const float *A, int lda, const float *B,
                  int ldb, const float *bias, float *Z, float *C, int ldc, int act, int nz = 1,
                  int krange = 0, float *db = nullptr) {
  auto go = [&](auto *kernel, int g) {
    kernel<<<dim3(blocks_for(N, g), blocks_for(M, g), nz), 256, 0, m->stream>>>(
        M, N, K, A, lda, B, ldb, bias, Z, C, ldc, act, krange, m->n_params, db);
    count_launches();
  };
  const int g = layer_tile(M, N, nz, m->sms);
  if (g == 64) go(k_layer<MODE, 64>, 64);
  else if (g == 32) go(k_layer<MODE, 32>, 32);
  else go(k_layer<MODE, 16>, 16);
}

// g[x] = the partial gradients of all row ranges, in order
__global__ void k_sum_splits(long long count, int splits, const float *__restrict__ part,
                             float *__restrict__ g) {
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= count) return;
  float s = 0.f;
  for (int z = 0; z < splits; ++z) s += part[z * count + x];
  g[x] = s;
}

// BF16 inference layer: weights and activations in bf16, FP32 accumulate.
__global__ void k_lin_fwd16(int n, int in, int out, const __nv_bfloat16 *__restrict__ X,
                            const __nv_bfloat16 *__restrict__ W, const __nv_bfloat16 *__restrict__ b,
                            __nv_bfloat16 *__restrict__ Y16, float *__restrict__ Y32, int act) {
  __shared__ float xs[kT][kT + 1], ws[kT][kT + 1];
  const int row = blockIdx.y * kT + threadIdx.y, col = blockIdx.x * kT + threadIdx.x;
  float acc = 0.f;
  for (int k0 = 0; k0 < in; k0 += kT) {
    xs[threadIdx.y][threadIdx.x] = (row < n && k0 + threadIdx.x < in)
                                       ? __bfloat162float(X[(long long)row * in + k0 + threadIdx.x])
                                       : 0.f;
    const int wr = blockIdx.x * kT + threadIdx.y;
    ws[threadIdx.y][threadIdx.x] = (wr < out && k0 + threadIdx.x < in)
                                       ? __bfloat162float(W[(long long)wr * in + k0 + threadIdx.x])
                                       : 0.f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kT; ++k) acc = fmaf(xs[threadIdx.y][k], ws[threadIdx.x][k], acc);
    __syncthreads();
  }
  if (row < n && col < out) {
    const float z = acc + __bfloat162float(b[col]);
    const float y = act ? silu(z) : z;
    if (Y16) Y16[(long long)row * out + col] = __float2bfloat16(y);
    if (Y32) Y32[(long long)row * out + col] = y;
  }
}

// loss = mean((Y - T)^2) over n*o; dY = 2 (Y - T) / (n o).  The CTAs' partial
// sums are added in CTA order by the CTA that finishes last.
__global__ void __launch_bounds__(256)
    k_mse(int n, int o, int ld, const float *__restrict__ Y, const float *__restrict__ T,
          float *__restrict__ dY, float *__restrict__ loss, float *__restrict__ part,
          int *__restrict__ ctr) {
  __shared__ float sh[256];
  __shared__ bool last;
  float s = 0.f;
  const long long total = (long long)n * o;
  const float scale = 2.f / (float)total;
  for (long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x; x < total;
       x += (long long)gridDim.x * blockDim.x) {
    const long long r = x / o, c = x % o;
    const float d = Y[r * ld + c] - T[x];
    s += d * d;
    dY[r * ld + c] = scale * d;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) sh[threadIdx.x] += sh[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[blockIdx.x] = sh[0];
    __threadfence();
    last = atomicAdd(ctr, 1) == (int)gridDim.x - 1;
    if (last) {
      *ctr = 0;
      __threadfence();
      float t = 0.f;
      for (int b = 0; b < (int)gridDim.x; ++b) t += __ldcg(part + b);
      *loss = t / (float)total;
    }
  }
}

__global__ void k_adam(long long count, float *__restrict__ p, const float *__restrict__ g,
                       float *__restrict__ m, float *__restrict__ v, float lr, float b1, float b2,
                       float c1, float c2, float eps) {
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= count) return;
  const float gi = g[x];
  m[x] = b1 * m[x] + (1.f - b1) * gi;
  v[x] = b2 * v[x] + (1.f - b2) * gi * gi;
  p[x] -= lr * (m[x] / c1) / (sqrtf(v[x] / c2) + eps);
}

__global__ void k_to_bf16(long long count, const float *__restrict__ a, __nv_bfloat16 *__restrict__ b) {
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < count) b[x] = __float2bfloat16(a[x]);
}

int ensure_capacity(tlr_mlp *m, int n) {
  if (n <= m->cap) return TLR_OK;
  cudaFree(m->act); cudaFree(m->pre); cudaFree(m->dact); cudaFree(m->xbuf); cudaFree(m->ybuf);
  const size_t plane = (size_t)n * m->maxw;
  if (cudaMalloc(&m->act, sizeof(float) * plane * (m->n_layers + 1)) ||
      cudaMalloc(&m->pre, sizeof(float) * plane * (m->n_layers + 1)) ||
      cudaMalloc(&m->dact, sizeof(float) * plane * (m->n_layers + 1)) ||
      cudaMalloc(&m->xbuf, sizeof(float) * (size_t)n * m->n_in) ||
      cudaMalloc(&m->ybuf, sizeof(float) * (size_t)n * m->n_out))
    return TLR_ERR_NOMEM;
  m->cap = n;
  return TLR_OK;
}

// forward of a batch already in xbuf; activations in act planes
void forward(tlr_mlp *m, int n) {
  const size_t plane = (size_t)m->cap * m->maxw;
  const float *X = m->xbuf;
  int ldx = m->n_in;
  for (int l = 0; l < m->n_layers; ++l) {
    const int in = m->fan_in[l], out = m->fan_out[l];
    float *Z = m->pre + plane * (l + 1), *Y = m->act + plane * (l + 1);
    launch_layer<kFwd>(m, n, out, in, X, ldx, m->params + m->w_off[l], in, m->params + m->b_off[l],
                       Z, Y, m->maxw, l + 1 < m->n_layers);
    X = Y;
    ldx = m->maxw;
  }
}

// loss and dY of the batch in act[last] / ybuf
void loss_gradient(tlr_mlp *m, int n) {
  const size_t plane = (size_t)m->cap * m->maxw;
  const int ctas = std::min(kLossCtas, blocks_for((long long)n * m->n_out, 1024));
  { k_mse<<<ctas, 256, 0, m->stream>>>(n, m->n_out, m->maxw, m->act + plane * m->n_layers, m->ybuf,
                                       m->dact + plane * m->n_layers, m->loss, m->lpart,
                                       m->lctr); count_launches(); }
}

// backward from dact[last] (dY) into grads.  The rows of a weight gradient are
// split into ranges of 128 (up to kMaxSplit), so that the 16 tiles of a 256 x
// 256 layer fill the SMs; one launch adds the ranges of all layers.
void backward(tlr_mlp *m, int n) {
  const size_t plane = (size_t)m->cap * m->maxw;
  const int splits = std::min(m->max_split, std::max(1, n / 128));
  const int krange = ((n + splits - 1) / splits + 15) / 16 * 16;
  const int nz = (n + krange - 1) / krange;
  float *dst = nz > 1 ? m->wpart : m->grads;
  for (int l = m->n_layers - 1; l >= 0; --l) {
    const int in = m->fan_in[l], out = m->fan_out[l];
    const float *dZ = m->dact + plane * (l + 1);
    const float *X = l == 0 ? m->xbuf : m->act + plane * l;
    const int ldx = l == 0 ? m->n_in : m->maxw;
    launch_layer<kWeight>(m, out, in, n, dZ, m->maxw, X, ldx, nullptr, nullptr, dst + m->w_off[l],
                          in, 0, nz, krange, dst + m->b_off[l]);
    if (l > 0)  // times silu' of the layer below: dZ of that layer
      launch_layer<kData>(m, n, in, out, dZ, m->maxw, m->params + m->w_off[l], in, nullptr,
                          m->pre + plane * l, m->dact + plane * l, m->maxw, 0);
  }
  if (nz > 1)
    { k_sum_splits<<<blocks_for(m->n_params, 256), 256, 0, m->stream>>>(m->n_params, nz, m->wpart,
                                                                       m->grads); count_launches(); }
}

}  // namespace
}  // namespace tlr

using namespace tlr;

extern "C" {

int tlr_mlp_tile(int rows, int cols, int ranges, int sms) {
  return layer_tile(rows, cols, ranges, sms);
}

int tlr_mlp_create(int n_in, int width, int depth, int n_out, unsigned long long seed,
                   tlr_mlp **out) {
  if (!out || n_in < 1 || width < 1 || depth < 1 || n_out < 1) return TLR_ERR_ARG;
  tlr_mlp *m = new tlr_mlp();
  m->n_in = n_in; m->width = width; m->depth = depth; m->n_out = n_out;
  m->n_layers = depth + 1;
  m->maxw = std::max(width, std::max(n_out, n_in));
  long long off = 0;
  for (int l = 0; l < m->n_layers; ++l) {
    const int in = l == 0 ? n_in : width, o = l + 1 == m->n_layers ? n_out : width;
    m->fan_in.push_back(in);
    m->fan_out.push_back(o);
    m->w_off.push_back(off);
    off += (long long)in * o;
    m->b_off.push_back(off);
    off += o;
  }
  m->n_params = off;
  // He-style initialisation from a deterministic generator
  std::vector<float> h(off, 0.f);
  unsigned long long s = seed ? seed : 0x243F6A8885A308D3ull;
  auto next = [&]() {
    s ^= s >> 12; s ^= s << 25; s ^= s >> 27;
    return (double)((s * 2685821657736338717ull) >> 11) * (1.0 / 9007199254740992.0);
  };
  for (int l = 0; l < m->n_layers; ++l) {
    const double a = std::sqrt(6.0 / m->fan_in[l]) * (l + 1 == m->n_layers ? 0.5 : 1.0);
    for (long long k = 0; k < (long long)m->fan_in[l] * m->fan_out[l]; ++k)
      h[m->w_off[l] + k] = (float)((2.0 * next() - 1.0) * a);
  }
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, dev);
  // at most 256 MB of partial gradients
  m->max_split = (int)std::max(1LL, std::min<long long>(kMaxSplit, (64LL << 20) / off));
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) ||
      cudaMalloc(&m->params, sizeof(float) * off) || cudaMalloc(&m->grads, sizeof(float) * off) ||
      cudaMalloc(&m->m1, sizeof(float) * off) || cudaMalloc(&m->m2, sizeof(float) * off) ||
      cudaMalloc(&m->params16, sizeof(__nv_bfloat16) * off) ||
      cudaMalloc(&m->loss, sizeof(float)) ||
      (m->max_split > 1 && cudaMalloc(&m->wpart, sizeof(float) * m->max_split * off)) ||
      cudaMalloc(&m->lpart, sizeof(float) * kLossCtas) || cudaMalloc(&m->lctr, sizeof(int)) ||
      cudaMemset(m->lctr, 0, sizeof(int)) ||
      cudaMemcpy(m->params, h.data(), sizeof(float) * off, cudaMemcpyHostToDevice) ||
      cudaMemset(m->m1, 0, sizeof(float) * off) || cudaMemset(m->m2, 0, sizeof(float) * off)) {
    tlr_mlp_destroy(m);
    return TLR_ERR_NOMEM;
  }
  *out = m;
  return TLR_OK;
}

void tlr_mlp_destroy(tlr_mlp *m) {
  if (!m) return;
  if (m->stream) cudaStreamSynchronize(m->stream);
  cudaFree(m->params); cudaFree(m->grads); cudaFree(m->m1); cudaFree(m->m2);
  cudaFree(m->params16); cudaFree(m->act); cudaFree(m->pre); cudaFree(m->dact);
  cudaFree(m->xbuf); cudaFree(m->ybuf); cudaFree(m->loss);
  cudaFree(m->wpart); cudaFree(m->lpart); cudaFree(m->lctr);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
}

long long tlr_mlp_num_params(const tlr_mlp *m) { return m ? m->n_params : 0; }

int tlr_mlp_params(tlr_mlp *m, float *host, int set) {
  if (!m || !host) return TLR_ERR_ARG;
  const size_t bytes = sizeof(float) * m->n_params;
  cudaError_t e = set ? cudaMemcpy(m->params, host, bytes, cudaMemcpyHostToDevice)
                      : cudaMemcpy(host, m->params, bytes, cudaMemcpyDeviceToHost);
  if (set) m->adam_t = 0;
  return e == cudaSuccess ? TLR_OK : TLR_ERR_CUDA;
}

// Loss and parameter gradients of one batch (host arrays), without update.
int tlr_mlp_gradients(tlr_mlp *m, const float *X, const float *Y, int n, float *grads,
                      float *loss) {
  if (!m || !X || !Y || n < 1) return TLR_ERR_ARG;
  int rc = ensure_capacity(m, n);
  if (rc) return rc;
  cudaMemcpyAsync(m->xbuf, X, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream);
  cudaMemcpyAsync(m->ybuf, Y, sizeof(float) * n * m->n_out, cudaMemcpyHostToDevice, m->stream);
  forward(m, n);
  loss_gradient(m, n);
  backward(m, n);
  if (grads)
    cudaMemcpyAsync(grads, m->grads, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost,
                    m->stream);
  if (loss) cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  return cudaStreamSynchronize(m->stream) == cudaSuccess ? TLR_OK : TLR_ERR_CUDA;
}

// Adam training over (X, Y) for `epochs`, minibatches of `batch` rows in a
// fixed cyclic order; loss_history[epoch] = mean minibatch loss (optional).
int tlr_mlp_train(tlr_mlp *m, const float *X, const float *Y, int n, int epochs, int batch,
                  float lr, float *loss_history) {
  if (!m || !X || !Y || n < 1 || epochs < 1 || batch < 1) return TLR_ERR_ARG;
  batch = std::min(batch, n);
  int rc = ensure_capacity(m, batch);
  if (rc) return rc;
  float *dX = nullptr, *dY = nullptr;
  if (cudaMalloc(&dX, sizeof(float) * (size_t)n * m->n_in) ||
      cudaMalloc(&dY, sizeof(float) * (size_t)n * m->n_out)) {
    cudaFree(dX);
    return TLR_ERR_NOMEM;
  }
  cudaMemcpy(dX, X, sizeof(float) * (size_t)n * m->n_in, cudaMemcpyHostToDevice);
  cudaMemcpy(dY, Y, sizeof(float) * (size_t)n * m->n_out, cudaMemcpyHostToDevice);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  std::vector<float> hl;
  for (int ep = 0; ep < epochs; ++ep) {
    double acc = 0.0;
    int nb = 0;
    for (int r0 = 0; r0 < n; r0 += batch) {
      const int nr = std::min(batch, n - r0);
      cudaMemcpyAsync(m->xbuf, dX + (size_t)r0 * m->n_in, sizeof(float) * nr * m->n_in,
                      cudaMemcpyDeviceToDevice, m->stream);
      cudaMemcpyAsync(m->ybuf, dY + (size_t)r0 * m->n_out, sizeof(float) * nr * m->n_out,
                      cudaMemcpyDeviceToDevice, m->stream);
      forward(m, nr);
      loss_gradient(m, nr);
      backward(m, nr);
      ++m->adam_t;
      const float c1 = 1.f - std::pow(b1, (float)m->adam_t), c2 = 1.f - std::pow(b2, (float)m->adam_t);
      { k_adam<<<blocks_for(m->n_params, 256), 256, 0, m->stream>>>(m->n_params, m->params, m->grads,
                                                                  m->m1, m->m2, lr, b1, b2, c1, c2,
                                                                  eps); count_launches(); }
      if (loss_history) {
        float l = 0.f;
        cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
        cudaStreamSynchronize(m->stream);
        acc += l;
        ++nb;
      }
    }
    if (loss_history) loss_history[ep] = (float)(acc / std::max(nb, 1));
  }
  cudaFree(dX);
  cudaFree(dY);
  return cudaStreamSynchronize(m->stream) == cudaSuccess ? TLR_OK : TLR_ERR_CUDA;
}

// Inference: Y [n][n_out] from X [n][n_in] (host arrays); bf16 != 0 runs the
// BF16 path (weights and activations rounded to bf16, FP32 accumulation).
int tlr_mlp_forward(tlr_mlp *m, const float *X, int n, float *Y, int bf16) {
  if (!m || !X || !Y || n < 1) return TLR_ERR_ARG;
  int rc = ensure_capacity(m, n);
  if (rc) return rc;
  cudaMemcpyAsync(m->xbuf, X, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream);
  const size_t plane = (size_t)m->cap * m->maxw;
  if (!bf16) {
    forward(m, n);
    // output plane has leading dimension maxw
    cudaMemcpy2DAsync(Y, sizeof(float) * m->n_out, m->act + plane * m->n_layers,
                      sizeof(float) * m->maxw, sizeof(float) * m->n_out, n,
                      cudaMemcpyDeviceToHost, m->stream);
  } else {
    { k_to_bf16<<<blocks_for(m->n_params, 256), 256, 0, m->stream>>>(m->n_params, m->params,
                                                                   m->params16); count_launches(); }
    __nv_bfloat16 *a = reinterpret_cast<__nv_bfloat16 *>(m->act);
    __nv_bfloat16 *bb = reinterpret_cast<__nv_bfloat16 *>(m->pre);
    { k_to_bf16<<<blocks_for((long long)n * m->n_in, 256), 256, 0, m->stream>>>(
        (long long)n * m->n_in, m->xbuf, a); count_launches(); }
    for (int l = 0; l < m->n_layers; ++l) {
      const int in = m->fan_in[l], o = m->fan_out[l];
      const bool last = l + 1 == m->n_layers;
      dim3 g((o + kT - 1) / kT, (n + kT - 1) / kT), b(kT, kT);
      { k_lin_fwd16<<<g, b, 0, m->stream>>>(n, in, o, a, m->params16 + m->w_off[l],
                                          m->params16 + m->b_off[l], last ? nullptr : bb,
                                          last ? m->dact : nullptr, !last); count_launches(); }
      std::swap(a, bb);
    }
    cudaMemcpyAsync(Y, m->dact, sizeof(float) * n * m->n_out, cudaMemcpyDeviceToHost, m->stream);
  }
  return cudaStreamSynchronize(m->stream) == cudaSuccess ? TLR_OK : TLR_ERR_CUDA;
}

}  // extern "C"
