/*
 * gd_mlp.cu -- forward, backward and Adam kernels of the energy surrogate (gd_mlp.cuh).
 *
 * Every matrix product of training runs on the fifth-generation tensor cores through
 * umma_gemm (gd_umma.cu: TMA-staged BF16 operands, FP32 accumulator in tensor memory), with
 * the elementwise step that follows it fused into its epilogue:
 *   forward        Z = X W + b, A = bf16(SiLU(Z))         (X K-major, W MN-major)
 *   input grad     dZ' = bf16((dZ W^T) SiLU'(Z'))         (dZ K-major, W K-major)
 *   weight grad    dW = A^T dZ over chunks of 256 rows    (both MN-major, split-K partials)
 * The 256 -> 1 output layer with the loss and its gradient (out_loss), the column sums it needs,
 * the embedding gradient (atomic scatter) and Adam are kernels of their own. Batch reductions
 * add per-chunk partials in a fixed order, all in one launch at the end (reduce_batch). Master
 * parameters, gradients and Adam moments are FP32; W1..W3 are mirrored in BF16 (row-major, and
 * in MMA-fragment order for the one-kernel forward) after every update.
 */
#include <algorithm>
#include <climits>
#include <cmath>

#include "gd_mlp.cuh"
#include "gd_mlp_fwd.cuh"
#include "gd_numerics.h"
#include "gd_umma.cuh"

namespace gd {

using bf16 = __nv_bfloat16;

namespace {

__device__ __forceinline__ float silu(float z) { return mlp_silu(z); }
__device__ __forceinline__ float silu_grad(float z) { return mlp_silu_grad(z); }

/* y[r] = A3[r] . w4 + b4, one warp per row */
__global__ void out_layer(const bf16 *__restrict__ A3, const float *__restrict__ w4,
                          const float *__restrict__ b4, float *__restrict__ y, int rows, int h) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= rows) return;
  float s = 0.0f;
  for (int j = lane; j < h; j += 32) s += __bfloat162float(A3[(size_t)r * h + j]) * w4[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) y[r] = s + b4[0];
}

/* The output layer, the loss and what they send back, one warp per row of M:
 *   y = A3 . w4 + b4, dy = 2 (y - t) / rows, e2 = (y - t)^2, D = bf16((dy w4^T) SiLU'(Z3)).
 * Rows past `rows` (padding) get dy = 0 and D = 0. Four kernels and two clears did this, at
 * 8,192 rows of 256 about 30 us; the row's A3 and Z3 are read once either way, so what goes is
 * the launches and the passes over y and dy. */
__global__ void __launch_bounds__(256) out_loss(const bf16 *__restrict__ A3,
                                                const float *__restrict__ Z3,
                                                const float *__restrict__ w4,
                                                const float *__restrict__ b4,
                                                const float *__restrict__ t, int rows, int M, int h,
                                                float *__restrict__ y, float *__restrict__ dy,
                                                float *__restrict__ e2, bf16 *__restrict__ D) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= M) return;
  const size_t r0 = (size_t)r * h;
  if (r >= rows) {
    if (lane == 0) dy[r] = 0.0f;
    for (int j = lane; j < h; j += 32) D[r0 + j] = __float2bfloat16_rn(0.0f);
    return;
  }
  float s = 0.0f;
#pragma unroll 8
  for (int j = lane; j < h; j += 32) s += __bfloat162float(A3[r0 + j]) * w4[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  const float yr = __shfl_sync(0xffffffffu, s + b4[0], 0);
  const float d = yr - t[r], g = 2.0f * d / (float)rows;
  if (lane == 0) {
    y[r] = yr;
    dy[r] = g;
    e2[r] = d * d;
  }
#pragma unroll 8
  for (int j = lane; j < h; j += 32)
    D[r0 + j] = __float2bfloat16_rn(g * w4[j] * silu_grad(Z3[r0 + j]));
}

/* Reductions over the batch are split into chunks of SPLIT_ROWS rows: each chunk writes a
 * partial result, reduce_partials adds the chunks in a fixed order (deterministic). */
constexpr int SPLIT_ROWS = 256;
constexpr size_t PARTS_MAX = (size_t)256 << 20; /* bytes */

/* Partial column sums of the output layer's two [rows][n] BF16 matrices, one per grid z:
 *   z = 0  A3 weighted per row by dy, with an extra column n that holds sum_r dy[r]
 *   z = 1  dZ3
 * Block: 32 columns x 8 row lanes; grid (columns / 32, chunks, 2). part_z[chunk][ncol]. A chain of
 * dependent additions over 32 rows a lane: the loads are issued eight at a time ahead of it (one
 * at a time, in two launches: 14.5 and 17.7 us at 8,192 rows of 256). */
__global__ void __launch_bounds__(256) colsum_split(const bf16 *__restrict__ A3,
                                                    const float *__restrict__ dy,
                                                    const bf16 *__restrict__ D, int rows, int n,
                                                    float *__restrict__ part0,
                                                    float *__restrict__ part1) {
  __shared__ float sh[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + cx, chunk = blockIdx.y;
  const bool weighted = blockIdx.z == 0;
  const int ncol = n + (weighted ? 1 : 0);
  const int r0 = chunk * SPLIT_ROWS, r1 = min(rows, r0 + SPLIT_ROWS);
  float s = 0.0f;
  if (col < ncol) {
    if (weighted) {
#pragma unroll 8
      for (int r = r0 + ry; r < r1; r += 8) {
        const float a = col < n ? __bfloat162float(A3[(size_t)r * n + col]) : 1.0f;
        s += a * dy[r];
      }
    } else {
#pragma unroll 8
      for (int r = r0 + ry; r < r1; r += 8) s += __bfloat162float(D[(size_t)r * n + col]);
    }
  }
  sh[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && col < ncol) {
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += sh[k][cx];
    (weighted ? part0 : part1)[(size_t)chunk * ncol + col] = t;
  }
}

/* One job per parameter tensor: out[i] = sum_c part[c * count + i] in the order of the chunks, by
 * blocks [first, next job's first); the last block is the loss, the mean of e2 (if given). One
 * launch at the end for the seven sums and the loss (launches of their own between the GEMMs: 6 us
 * each). */
struct ReduceJobs {
  static constexpr int N = 7;
  struct {
    const float *part;
    float *out;
    int chunks, count, first;
  } job[N];
};

__global__ void __launch_bounds__(256) reduce_batch(const ReduceJobs jobs,
                                                    const float *__restrict__ e2, int rows,
                                                    float *__restrict__ loss) {
  if (e2 && blockIdx.x == gridDim.x - 1) {
    __shared__ double sh[256];
    double s = 0.0;
#pragma unroll 8
    for (int i = threadIdx.x; i < rows; i += 256) s += e2[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) loss[0] = (float)(sh[0] / (double)rows);
    return;
  }
  int k = 0;
#pragma unroll
  for (int q = 1; q < ReduceJobs::N; ++q)
    if ((int)blockIdx.x >= jobs.job[q].first) k = q;
  const int i = ((int)blockIdx.x - jobs.job[k].first) * 256 + threadIdx.x;
  const int count = jobs.job[k].count, chunks = jobs.job[k].chunks;
  if (i >= count) return;
  const float *__restrict__ p = jobs.job[k].part + i;
  float s = 0.0f;
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) s += p[(size_t)c * count];
  jobs.job[k].out[i] = 0.0f + s;
}

/* embedding gradient: columns [7, 39) of dX1 scattered to the rows' conformer entries */
__global__ void emb_grad(const float *__restrict__ dX, const int *__restrict__ conf, int rows,
                         float *__restrict__ gemb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * GD_MLP_EMB) return;
  const int r = i / GD_MLP_EMB, c = i - r * GD_MLP_EMB;
  const int e = conf[r];
  if (e >= 0) atomicAdd(gemb + (size_t)e * GD_MLP_EMB + c, dX[(size_t)r * GD_MLP_IN + GD_MLP_EMB_OFF + c]);
}

/* embedding columns of X from theta (rows with conf < 0 keep their columns) */
__global__ void emb_fill(bf16 *__restrict__ X, const float *__restrict__ emb,
                         const int *__restrict__ conf, int rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * GD_MLP_EMB) return;
  const int r = i / GD_MLP_EMB, c = i - r * GD_MLP_EMB;
  const int e = conf[r];
  if (e >= 0)
    X[(size_t)r * GD_MLP_IN + GD_MLP_EMB_OFF + c] = __float2bfloat16_rn(emb[(size_t)e * GD_MLP_EMB + c]);
}

__global__ void adam_kernel(float *__restrict__ th, const float *__restrict__ g,
                            float *__restrict__ m, float *__restrict__ v, size_t n, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  th[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

/* the Adam step with its bias corrections read from c[0], c[1] (device) */
__global__ void adam_dev_kernel(float *__restrict__ th, const float *__restrict__ g,
                                float *__restrict__ m, float *__restrict__ v, size_t n, float lr,
                                float b1, float b2, float eps, const float *__restrict__ c) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float c1 = c[0], c2 = c[1];
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  th[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

/* advances the device step count t = st[0] and writes 1 - b1^t, 1 - b2^t as floats at st[1..2] */
__global__ void adam_tick(int *st, float b1, float b2) {
  const int t = st[0] + 1;
  st[0] = t;
  float *c = reinterpret_cast<float *>(st + 1);
  c[0] = 1.0f - powf(b1, (float)t);
  c[1] = 1.0f - powf(b2, (float)t);
}

__global__ void to_bf16(const float *__restrict__ a, bf16 *__restrict__ b, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = __float2bfloat16_rn(a[i]);
}

/* Fragment-ordered BF16 copy of W1, W2, W3 for the fused forward (H = 128 or 256, W = H / 16
 * warps): in each layer block, element (((ks W + w) 32 + lane) 2 + j) 4 + q holds W[k][n] with
 * k = 16 ks + 2 (lane % 4) + (q % 2) + 8 (q / 2) and n = 8 (2 w + j) + lane / 4, the
 * m16n8k16 B-operand fragment {b0, b1, b2, b3} of lane `lane` for 8-column tile j of warp w at
 * k-step ks, so that a lane's fragments of one k-step are 16 contiguous bytes. */
__global__ void to_frag(const float *__restrict__ theta, MlpLayout L, bf16 *__restrict__ wf) {
  const size_t H = L.hidden, n1 = (size_t)GD_MLP_IN * H, i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n1 + 2 * H * H) return;
  size_t e = i;
  const float *W = theta + L.w1;
  if (e >= n1 + H * H) {
    e -= n1 + H * H;
    W = theta + L.w3;
  } else if (e >= n1) {
    e -= n1;
    W = theta + L.w2;
  }
  const int warps = (int)(H / 16);
  const int q = (int)(e & 3), j = (int)((e >> 2) & 1), lane = (int)((e >> 3) & 31);
  const size_t t = e >> 8, ks = t / warps;
  const int w = (int)(t - ks * warps);
  const size_t k = 16 * ks + 2 * (lane & 3) + (q & 1) + 8 * (q >> 1);
  const size_t n = 8 * (2 * w + j) + (lane >> 2);
  wf[i] = __float2bfloat16_rn(W[k * H + n]);
}

/* FP32 rows to BF16 rows of X, eight columns a thread, with the embedding columns of rows with
 * conf >= 0 from the table in place of the row's own */
__global__ void __launch_bounds__(256) rows_to_x(const float4 *__restrict__ x,
                                                 const int *__restrict__ conf,
                                                 const float *__restrict__ emb, int rows,
                                                 uint4 *__restrict__ X) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  const int r = i / (GD_MLP_IN / 8), c0 = (i - r * (GD_MLP_IN / 8)) * 8;
  if (r >= rows) return;
  const float4 a = x[2 * (size_t)i], b = x[2 * (size_t)i + 1];
  float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  const int e = emb ? conf[r] : -1;
  if (e >= 0) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = c0 + k - GD_MLP_EMB_OFF;
      if (c >= 0 && c < GD_MLP_EMB) v[k] = emb[(size_t)e * GD_MLP_EMB + c];
    }
  }
  __align__(16) __nv_bfloat162 o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) o[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
  X[i] = *reinterpret_cast<const uint4 *>(o);
}

/* uniform(-scale, scale) from Philox, keyed by (seed, tensor id) */
__global__ void init_uniform(float *p, size_t n, float scale, uint32_t tensor, uint64_t seed) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const gd_u32x4 r = gd_philox4x32_10((uint32_t)i, tensor, 0x5EEDu, 7u, (uint32_t)seed,
                                      (uint32_t)(seed >> 32));
  p[i] = scale * gd_sym11(r.v[0]);
}

/* The whole forward pass of fwd::FR rows in one CTA (gd_mlp_fwd.cuh). */
template <int NT>
__global__ void __launch_bounds__(fwd::Dims<NT>::THREADS) fused_forward(const bf16 *__restrict__ X,
                                                     const int *__restrict__ conf,
                                                     const float *__restrict__ theta,
                                                     const bf16 *__restrict__ wf, MlpLayout L,
                                                     int rows, float *__restrict__ y) {
  using D = fwd::Dims<NT>;
  constexpr int FR = fwd::FR;
  extern __shared__ __align__(128) unsigned char fsm[];
  __shared__ int cf[FR];
  __shared__ float ys[FR];
  const fwd::Smem<NT> sm(fsm);
  bf16 *xs = sm.xs;
  const int tid = threadIdx.x;
  const int row0 = blockIdx.x * FR;
  fwd::Ring ring;
  fwd::prefetch_first<NT>(ring, wf, tid);
  fwd::stage_params<NT>(sm, theta, L, tid);
  for (int i = tid; i < FR * 8; i += D::THREADS) {
    const int r = i >> 3, c = i & 7;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row0 + r < rows) v = reinterpret_cast<const uint4 *>(X + (size_t)(row0 + r) * GD_MLP_IN)[c];
    *reinterpret_cast<uint4 *>(xs + r * D::LDX + c * 8) = v;
  }
  if (tid < FR) cf[tid] = row0 + tid < rows ? conf[row0 + tid] : -1;
  __syncthreads();
  fwd::fill_embedding<NT>(xs, cf, theta, L, tid);
  __syncthreads();
  fwd::rows_forward<NT>(sm, ring, wf, ys, tid);
  if (tid < FR && row0 + tid < rows) y[row0 + tid] = ys[tid];
}

constexpr int FR = fwd::FR;
template <int NT>
using FusedDims = fwd::Dims<NT>;

inline int blocks(size_t n, int t = 256) { return (int)((n + t - 1) / t); }

}  // namespace

int mlp_refresh_bf16(Mlp &n, cudaStream_t s) {
  const size_t nw = n.L.b4; /* W1..w4 region; biases converted too, unused */
  to_bf16<<<blocks(nw), 256, 0, s>>>(n.theta, n.wh, nw);
  if (n.wf) {
    const size_t H = n.L.hidden;
    to_frag<<<blocks((size_t)GD_MLP_IN * H + 2 * H * H), 256, 0, s>>>(n.theta, n.L, n.wf);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_create(Mlp &n, int hidden, int n_emb, uint64_t seed, cudaStream_t s) {
  if (hidden % 16 || hidden < 16 || hidden > 256) return -1;
  n.L.set(hidden, n_emb);
  const size_t T = n.L.total;
  if (cudaMalloc(&n.theta, T * 4) || cudaMalloc(&n.grad, T * 4) || cudaMalloc(&n.m, T * 4) ||
      cudaMalloc(&n.v, T * 4) || cudaMalloc(&n.wh, n.L.b4 * 2) || cudaMalloc(&n.loss, 16) ||
      cudaMalloc(&n.err, sizeof(int)) || cudaMalloc(&n.adam_dev, 3 * sizeof(int)))
    return -3;
  cudaMemsetAsync(n.err, 0, sizeof(int), s);
  if ((hidden == 128 || hidden == 256) &&
      cudaMalloc(&n.wf, ((size_t)GD_MLP_IN * hidden + 2 * (size_t)hidden * hidden) * 2))
    return -3;
  cudaMemsetAsync(n.theta, 0, T * 4, s);
  cudaMemsetAsync(n.m, 0, T * 4, s);
  cudaMemsetAsync(n.v, 0, T * 4, s);
  const int H = hidden;
  init_uniform<<<blocks((size_t)GD_MLP_IN * H), 256, 0, s>>>(n.theta + n.L.w1, (size_t)GD_MLP_IN * H,
                                                             1.0f / sqrtf((float)GD_MLP_IN), 1, seed);
  init_uniform<<<blocks((size_t)H * H), 256, 0, s>>>(n.theta + n.L.w2, (size_t)H * H,
                                                     1.0f / sqrtf((float)H), 2, seed);
  init_uniform<<<blocks((size_t)H * H), 256, 0, s>>>(n.theta + n.L.w3, (size_t)H * H,
                                                     1.0f / sqrtf((float)H), 3, seed);
  init_uniform<<<blocks(H), 256, 0, s>>>(n.theta + n.L.w4, H, 1.0f / sqrtf((float)H), 4, seed);
  if (n_emb)
    init_uniform<<<blocks((size_t)n_emb * GD_MLP_EMB), 256, 0, s>>>(
        n.theta + n.L.emb, (size_t)n_emb * GD_MLP_EMB, 0.3f, 5, seed);
  n.adam_t = 0;
  if (cudaFuncSetAttribute(fused_forward<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)FusedDims<1>::smem) != cudaSuccess ||
      cudaFuncSetAttribute(fused_forward<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)FusedDims<2>::smem) != cudaSuccess)
    return -2;
  return mlp_refresh_bf16(n, s);
}

void mlp_destroy(Mlp &n) {
  void *ps[] = {n.theta, n.grad, n.m, n.v, n.wh, n.wf, n.loss, n.err, n.adam_dev, n.work, n.P};
  for (void *p : ps)
    if (p) cudaFree(p);
  n = Mlp();
}

int mlp_reserve(Mlp &n, int rows) {
  rows = (rows + 15) & ~15;
  if (rows <= n.cap) return 0;
  const size_t H = n.L.hidden, R = rows, C = H > GD_MLP_IN ? H : GD_MLP_IN;
  /* one block, each array at a 256-byte boundary (TMA wants 16) */
  size_t used = 0;
  auto take = [&](size_t bytes) {
    const size_t at = used;
    used += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t oX = take(R * GD_MLP_IN * 2), oA1 = take(R * H * 2), oA2 = take(R * H * 2),
               oA3 = take(R * H * 2), oD = take(R * H * 2), oD2 = take(R * H * 2),
               oZ1 = take(R * H * 4), oZ2 = take(R * H * 4), oZ3 = take(R * H * 4),
               oC = take(R * C * 4), oy = take(R * 4), ody = take(R * 4), oconf = take(R * 4);
  if (n.work) cudaFree(n.work);
  n.work = nullptr;
  n.cap = 0;
  if (cudaMalloc(&n.work, used) != cudaSuccess) return -3;
  auto h = [&](size_t at) { return reinterpret_cast<bf16 *>(n.work + at); };
  auto f = [&](size_t at) { return reinterpret_cast<float *>(n.work + at); };
  n.X = h(oX), n.A1 = h(oA1), n.A2 = h(oA2), n.A3 = h(oA3), n.D = h(oD), n.D2 = h(oD2);
  n.Z1 = f(oZ1), n.Z2 = f(oZ2), n.Z3 = f(oZ3), n.C = f(oC), n.y = f(oy), n.dy = f(ody);
  n.conf = reinterpret_cast<int *>(n.work + oconf);
  cudaMemset(n.X, 0, R * GD_MLP_IN * 2);
  cudaMemset(n.conf, 0xff, R * 4);
  /* the network's stream does not wait for the default stream */
  if (cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) return -2;
  n.cap = (int)R;
  return 0;
}

int mlp_set_rows(Mlp &n, const float *x, int rows, cudaStream_t s) {
  if (rows > n.cap) return -4;
  rows_to_x<<<blocks((size_t)rows * (GD_MLP_IN / 8)), 256, 0, s>>>(
      reinterpret_cast<const float4 *>(x), n.conf, n.L.n_emb ? n.theta + n.L.emb : nullptr, rows,
      reinterpret_cast<uint4 *>(n.X));
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_embed(Mlp &n, int rows, cudaStream_t s) {
  if (!n.L.n_emb) return 0;
  emb_fill<<<blocks((size_t)rows * GD_MLP_EMB), 256, 0, s>>>(n.X, n.theta + n.L.emb, n.conf, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

/* the hidden layers over `rows` rows of n.X; keeps Z1..Z3 when `keep` for the backward pass */
static int hidden_forward(Mlp &n, int rows, bool keep, cudaStream_t s) {
  const int M = (rows + 15) & ~15, H = n.L.hidden;
  if (M > n.cap) return -4;
  /* Z_l = A_{l-1} W_l + b_l, A_l = bf16(SiLU(Z_l)) in one tensor-core kernel per layer */
  auto layer = [&](const bf16 *Ain, int K, size_t w, size_t b, float *Z, bf16 *Aout) {
    const UmmaOperand a{Ain, M, K, 0}, wt{n.wh + w, K, H, 1};
    UmmaEpilogue e{};
    e.kind = UMMA_FWD;
    e.bias = n.theta + b;
    e.Z = keep ? Z : nullptr;
    e.Ob = Aout;
    e.ldo = H;
    return umma_gemm(a, wt, M, H, K, 1, e, n.err, s);
  };
  int rc;
  if ((rc = layer(n.X, GD_MLP_IN, n.L.w1, n.L.b1, n.Z1, n.A1)) ||
      (rc = layer(n.A1, H, n.L.w2, n.L.b2, n.Z2, n.A2)) ||
      (rc = layer(n.A2, H, n.L.w3, n.L.b3, n.Z3, n.A3)))
    return rc;
  return 0;
}

int mlp_forward(Mlp &n, int rows, cudaStream_t s) {
  const int H = n.L.hidden;
  if (rows > n.cap) return -4;
  if (rows < 1) return 0;
  if (H == 128) {
    fused_forward<1><<<(rows + FR - 1) / FR, FusedDims<1>::THREADS, FusedDims<1>::smem, s>>>(
        n.X, n.conf, n.theta, n.wf, n.L, rows, n.y);
  } else if (H == 256) {
    fused_forward<2><<<(rows + FR - 1) / FR, FusedDims<2>::THREADS, FusedDims<2>::smem, s>>>(
        n.X, n.conf, n.theta, n.wf, n.L, rows, n.y);
  } else {
    int rc = mlp_embed(n, rows, s);
    if (rc || (rc = hidden_forward(n, rows, false, s))) return rc;
    out_layer<<<blocks((size_t)rows * 32), 256, 0, s>>>(n.A3, n.theta + n.L.w4, n.theta + n.L.b4,
                                                        n.y, rows, H);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_loss_backward(Mlp &n, int rows, const float *t, cudaStream_t s) {
  const int M = (rows + 15) & ~15, H = n.L.hidden;
  int rc = hidden_forward(n, rows, true, s);
  if (rc) return rc;
  /* batch reductions in chunks of SPLIT_ROWS rows and tiles of 128, whose partials are added in a
   * fixed order: a part of P for each, all added at the end, while they take at most PARTS_MAX
   * together (112,000 rows at H = 256); past that one after the other in a buffer that holds the
   * largest, so that the memory per row of a large batch is less than half. The six launches more
   * are 1 % of such a pass. */
  const int S = (M + SPLIT_ROWS - 1) / SPLIT_ROWS, T = (M + 127) / 128;
  size_t need = 0, largest = 0;
  auto part = [&](size_t count, bool beside = false) {
    const size_t at = need, size = (count + 63) & ~(size_t)63;
    need += size;
    largest = beside ? largest + size : std::max(largest, size);
    return at;
  };
  size_t p_w4 = part((size_t)S * (H + 1)), p_b3 = part((size_t)S * H, true),
         p_w1 = part((size_t)S * GD_MLP_IN * H), p_w2 = part((size_t)S * H * H),
         p_w3 = part((size_t)S * H * H), p_b2 = part((size_t)T * H), p_b1 = part((size_t)T * H);
  const bool together = need * sizeof(float) <= PARTS_MAX;
  if (!together) {
    need = largest; /* w4 and b3 come from one launch, side by side */
    p_w1 = p_w2 = p_w3 = p_b1 = p_b2 = 0;
  }
  if (need > n.p_cap) {
    if (n.P) cudaFree(n.P);
    n.P = nullptr;
    n.p_cap = 0;
    if (cudaMalloc(&n.P, need * sizeof(float)) != cudaSuccess) return -3;
    n.p_cap = need;
  }
  ReduceJobs jobs;
  int n_jobs = 0, red_blocks = 0;
  auto reduce = [&](size_t at, int chunks, int count, float *out) {
    jobs.job[n_jobs++] = {n.P + at, out, chunks, count, red_blocks};
    red_blocks += blocks(count);
  };
  float *e2 = n.C;
  /* adds up the jobs so far; the last time with the loss */
  auto add_up = [&](bool last) {
    for (int q = n_jobs; q < ReduceJobs::N; ++q) jobs.job[q].first = INT_MAX;
    reduce_batch<<<red_blocks + (last ? 1 : 0), 256, 0, s>>>(jobs, last ? e2 : nullptr, rows,
                                                             n.loss);
    n_jobs = red_blocks = 0;
  };
  auto stage_done = [&] {
    if (!together) add_up(false);
  };
  /* the embedding's gradient is scattered, b4 is padded to four; the rest is written whole */
  cudaMemsetAsync(n.grad + n.L.b4, 0, (n.L.total - n.L.b4) * 4, s);
  /* dW[i][j] = sum_r Aprev[r][i] dZ[r][j] in chunks of SPLIT_ROWS rows (both operands
   * MN-major, the rows are the reduction); W1 (64 rows) is computed as dW1^T = dZ1^T X so that
   * the 128-row MMA tile runs along the hidden dimension, and stored transposed */
  auto weight_grad = [&](const bf16 *Aprev, int K, const bf16 *D, size_t at, float *g) {
    UmmaEpilogue e{};
    e.kind = UMMA_F32;
    e.Of = n.P + at;
    e.ldo = H;
    e.split_stride = (size_t)K * H;
    reduce(at, S, K * H, g);
    if (K == H)
      return umma_gemm(UmmaOperand{Aprev, M, K, 1}, UmmaOperand{D, M, H, 1}, K, H, SPLIT_ROWS, S,
                       e, n.err, s);
    e.trans = 1;
    return umma_gemm(UmmaOperand{D, M, H, 1}, UmmaOperand{Aprev, M, K, 1}, H, K, SPLIT_ROWS, S, e,
                     n.err, s);
  };
  /* dZ_{l-1} = bf16((dZ_l W_l^T) SiLU'(Z_{l-1})), and its column sums (db_{l-1}) per 128-row
   * tile, added in tile order */
  auto input_grad = [&](const bf16 *D, size_t w, const float *Zprev, bf16 *Dout, size_t at,
                        float *gb) {
    UmmaEpilogue e{};
    e.kind = UMMA_DGRAD;
    e.Zin = Zprev;
    e.Ob = Dout;
    e.colsum = n.P + at;
    e.ldo = H;
    reduce(at, T, H, gb);
    return umma_gemm(UmmaOperand{D, M, H, 0}, UmmaOperand{n.wh + w, H, H, 0}, M, H, H, 1, e, n.err,
                     s);
  };
  bf16 *Dc = n.D, *Dn = n.D2;
  /* output layer and loss: dZ3, dw4 = A3^T dy, db4 = sum dy (b4 follows w4 in theta), db3 */
  out_loss<<<blocks((size_t)M * 32), 256, 0, s>>>(n.A3, n.Z3, n.theta + n.L.w4, n.theta + n.L.b4, t,
                                                  rows, M, H, n.y, n.dy, e2, Dc);
  colsum_split<<<dim3((H + 32) / 32, S, 2), 256, 0, s>>>(n.A3, n.dy, Dc, M, H, n.P + p_w4,
                                                         n.P + p_b3);
  reduce(p_w4, S, H + 1, n.grad + n.L.w4);
  reduce(p_b3, S, H, n.grad + n.L.b3);
  stage_done();
  /* layer 3: dW3 = A2^T dZ3, dZ2 with db2 */
  if ((rc = weight_grad(n.A2, H, Dc, p_w3, n.grad + n.L.w3))) return rc;
  stage_done();
  if ((rc = input_grad(Dc, n.L.w3, n.Z2, Dn, p_b2, n.grad + n.L.b2))) return rc;
  stage_done();
  std::swap(Dc, Dn);
  /* layer 2: dW2, dZ1 with db1 */
  if ((rc = weight_grad(n.A1, H, Dc, p_w2, n.grad + n.L.w2))) return rc;
  stage_done();
  if ((rc = input_grad(Dc, n.L.w2, n.Z1, Dn, p_b1, n.grad + n.L.b1))) return rc;
  stage_done();
  std::swap(Dc, Dn);
  /* layer 1: dW1 = X^T dZ1 (64 x H); dX = dZ1 W1^T (FP32) for the embedding */
  if ((rc = weight_grad(n.X, GD_MLP_IN, Dc, p_w1, n.grad + n.L.w1))) return rc;
  add_up(true);
  if (n.L.n_emb) {
    UmmaEpilogue e{};
    e.kind = UMMA_F32;
    e.Of = n.C;
    e.ldo = GD_MLP_IN;
    if ((rc = umma_gemm(UmmaOperand{Dc, M, H, 0}, UmmaOperand{n.wh + n.L.w1, GD_MLP_IN, H, 0}, M,
                        GD_MLP_IN, H, 1, e, n.err, s)))
      return rc;
    emb_grad<<<blocks((size_t)rows * GD_MLP_EMB), 256, 0, s>>>(n.C, n.conf, rows,
                                                             n.grad + n.L.emb);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_status(Mlp &n) {
  int e = 0;
  if (cudaMemcpy(&e, n.err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -2;
  if (!e) return 0;
  cudaMemset(n.err, 0, sizeof(int));
  return -6;
}

int mlp_adam(Mlp &n, float lr, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  n.adam_t += 1;
  const float c1 = 1.0f - powf(b1, (float)n.adam_t), c2 = 1.0f - powf(b2, (float)n.adam_t);
  adam_kernel<<<blocks(n.L.total), 256, 0, s>>>(n.theta, n.grad, n.m, n.v, n.L.total, lr, b1, b2,
                                               eps, c1, c2);
  return mlp_refresh_bf16(n, s);
}

int mlp_adam_dev_sync(Mlp &n, cudaStream_t s) {
  return cudaMemcpyAsync(n.adam_dev, &n.adam_t, sizeof(int), cudaMemcpyHostToDevice, s) ==
                 cudaSuccess
             ? 0
             : -2;
}

int mlp_adam_dev(Mlp &n, float lr, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  adam_tick<<<1, 1, 0, s>>>(n.adam_dev, b1, b2);
  adam_dev_kernel<<<blocks(n.L.total), 256, 0, s>>>(
      n.theta, n.grad, n.m, n.v, n.L.total, lr, b1, b2, eps,
      reinterpret_cast<const float *>(n.adam_dev + 1));
  return mlp_refresh_bf16(n, s);
}

}  // namespace gd
