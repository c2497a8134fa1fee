// mlp.cu -- the fusion cost model's network: forward, backward and Adam on the
// GPU.
//
// Network: F input features -> 64 -> 64 -> 64 (ReLU) -> 1 (linear), FP32,
// trained on squared error of log2(kernel milliseconds).  There is nothing
// like it in the reference (its only optimisation is the gate-history
// peephole of qc_optimize, src/qcs.c:650-698).
//
// A training step is two kernels.  k_mlp_rows takes 8 rows a CTA forward and
// back (a batch of 256 rows is 32 CTAs) and leaves every layer's activations
// and errors; k_mlp_grad forms the weight gradients, 8 weight rows a CTA, and
// takes the Adam step in place.  A gradient is summed over the rows in slots
// of 64, each in row order, and over the slots in order, so it does not
// depend on how the work is cut.  Latency bounds both: 64 steps on 256 rows
// take 1.16 ms (1.32 when a kernel starts only after the end of the one before
// it), where one CTA per 64 rows for everything, a kernel for the sum of the
// slots and one for Adam took 21.7 ms.
#include <atomic>
#include <math.h>
#include <string.h>

#include <vector>

#include "common.cuh"
#include "costmodel.h"

namespace qcs {

constexpr int kMlpSlot = 64;         // rows of a gradient slot
constexpr int kMlpRows = 8;          // rows per CTA, forward and back
constexpr int kMlpRowThreads = 128;  // a row's 64 units on 16 threads, 4 each
constexpr int kMlpGradRows = 8;      // weight rows per CTA of k_mlp_grad
constexpr int kMlpGradThreads = 16 * kMlpGradRows;
constexpr int kMlpPitch = 68;        // floats per 64-wide row in shared memory
// Batches up to this size go through k_mlp_grad in one piece; larger ones are
// cut into slots, summed afterwards.
constexpr int kMlpDirectRows = 1024;
// The activations, 1.5 KB a row, are kept for this many rows at a time: 404 MB, and
// 4096 slots, where a grid's second dimension takes 65535.  Gradients of 1e6 rows 6.60
// ms; all rows at once 6.53, 2^16 at a time 6.88.
constexpr int kMlpPieceRows = 1 << 18;

struct MlpShape {
  int F;
  int off_w1, off_b1, off_w2, off_b2, off_w3, off_b3, off_w4, off_b4, count;
  __host__ __device__ MlpShape(int f) : F(f) {
    off_w1 = 0;
    off_b1 = off_w1 + F * kMlpHidden;
    off_w2 = off_b1 + kMlpHidden;
    off_b2 = off_w2 + kMlpHidden * kMlpHidden;
    off_w3 = off_b2 + kMlpHidden;
    off_b3 = off_w3 + kMlpHidden * kMlpHidden;
    off_w4 = off_b3 + kMlpHidden;
    off_b4 = off_w4 + kMlpHidden;
    count = off_b4 + 1;
  }
};

// What a row leaves for the gradients: h1, h2, h3, then dL/d(pre-activation)
// of layers 1, 2, 3 (64 each), then the output's error.
constexpr int kMlpActs = 6 * kMlpHidden + 1;
struct MlpActs {
  float *p;
  size_t rows;
  __host__ __device__ float *h(int l) const { return p + (size_t)l * rows * kMlpHidden; }
  __host__ __device__ float *g(int l) const { return p + (size_t)(3 + l) * rows * kMlpHidden; }
  __host__ __device__ float *d() const { return p + (size_t)6 * rows * kMlpHidden; }
};

// Asynchronous copies to shared memory (16 or 4 bytes): a CTA has its whole
// working set in flight at once, where loops of plain loads waited on one L2
// access after another (k_mlp_rows 25
// us instead of 8 on 256 rows, k_mlp_grad 34 instead of 11).
__device__ __forceinline__ void copy16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING));
}

// Four outputs j .. j+3 of one row: act(b[j] + sum_i in[i] * w[i][j]), the
// sum in the order of i.
__device__ __forceinline__ float4 mlp_layer(const float *in, int K, const float *w, int ldw,
                                            const float *b, int j, bool relu) {
  float4 acc = *reinterpret_cast<const float4 *>(b + j);
#pragma unroll 16
  for (int i = 0; i < K; i++) {
    const float x = in[i];
    const float4 v = *reinterpret_cast<const float4 *>(w + i * ldw + j);
    acc.x = fmaf(x, v.x, acc.x);
    acc.y = fmaf(x, v.y, acc.y);
    acc.z = fmaf(x, v.z, acc.z);
    acc.w = fmaf(x, v.w, acc.w);
  }
  if (relu) {
    acc.x = fmaxf(acc.x, 0.f);
    acc.y = fmaxf(acc.y, 0.f);
    acc.z = fmaxf(acc.z, 0.f);
    acc.w = fmaxf(acc.w, 0.f);
  }
  return acc;
}

// Rows [8 b, 8 b + 8) of a batch: forward; with Y the squared error and, with
// acts.p, back to every layer's pre-activations.
__global__ void __launch_bounds__(kMlpRowThreads)
    k_mlp_rows(const float *params, int F, const float *X, const float *Y, int n, float inv_n,
               MlpActs acts, double *loss_rows, float *pred) {
  extern __shared__ __align__(16) float sm[];
  constexpr int H = kMlpHidden, LD = kMlpPitch;
  const MlpShape S(F);
  float *w1 = sm;               // [F][LD]
  float *w2 = w1 + F * LD;      // [H][LD]
  float *w3 = w2 + H * LD;
  float *b1 = w3 + H * LD;      // [H] each
  float *b2 = b1 + H;
  float *b3 = b2 + H;
  float *w4 = b3 + H;
  float *x = w4 + H;            // [rows][F]
  float *h1 = x + kMlpRows * ((F + 3) & ~3);  // [rows][LD]
  float *h2 = h1 + kMlpRows * LD;
  float *h3 = h2 + kMlpRows * LD;
  float *g = h3 + kMlpRows * LD;
  __shared__ float err[kMlpRows];
  const int tid = threadIdx.x;
  const int r0 = blockIdx.x * kMlpRows;
  const int s = tid >> 4, j = 4 * (tid & 15), row = r0 + s;
  for (int e = tid; e < kMlpRows * F; e += kMlpRowThreads) {
    if (r0 + e / F < n) copy4(x + e, X + (size_t)r0 * F + e);
    else x[e] = 0.f;
  }
  const float yr = Y && row < n ? Y[row] : 0.f;
  grid_wait();  // the parameters are the kernel before's, the records are not
  for (int e = tid; e < (F + 2 * H) * (H / 4); e += kMlpRowThreads) {
    const int i = e / (H / 4), c = 4 * (e % (H / 4));  // rows of w1, w2, w3
    const int off = i < F ? S.off_w1 + i * H : i < F + H ? S.off_w2 + (i - F) * H
                                                         : S.off_w3 + (i - F - H) * H;
    copy16(w1 + i * LD + c, params + off + c);
  }
  for (int e = tid; e < 4 * H / 4; e += kMlpRowThreads) {  // b1, b2, b3, w4
    const int k = e / (H / 4), c = 4 * (e % (H / 4));
    const int off = k == 0 ? S.off_b1 : k == 1 ? S.off_b2 : k == 2 ? S.off_b3 : S.off_w4;
    copy16(b1 + k * H + c, params + off + c);
  }
  const float b4 = params[S.off_b4];
  copy_commit();
  copy_wait<0>();
  __syncthreads();
  auto put = [&](float *m, float4 v) { *reinterpret_cast<float4 *>(m + s * LD + j) = v; };
  put(h1, mlp_layer(x + s * F, F, w1, LD, b1, j, true));
  __syncthreads();
  put(h2, mlp_layer(h1 + s * LD, H, w2, LD, b2, j, true));
  __syncthreads();
  put(h3, mlp_layer(h2 + s * LD, H, w3, LD, b3, j, true));
  __syncthreads();
  if ((tid & 15) == 0) {
    float o = b4;
#pragma unroll 16
    for (int i = 0; i < H; i++) o = fmaf(h3[s * LD + i], w4[i], o);
    const bool in = row < n;
    if (pred && in) pred[row] = o;
    const float off = Y && in ? o - yr : 0.f;
    // dLoss/dout for loss = (1/n) sum (out - y)^2
    err[s] = 2.f * off * inv_n;
    if (loss_rows && in) loss_rows[row] = (double)off * off;
  }
  if (!acts.p) return;
  __syncthreads();
  const float d = err[s];
  const bool in = row < n;
  auto keep = [&](float *m, float4 v) {
    if (in) *reinterpret_cast<float4 *>(m + (size_t)row * H + j) = v;
  };
  auto at = [&](const float *m) { return *reinterpret_cast<const float4 *>(m + s * LD + j); };
  keep(acts.h(0), at(h1));
  keep(acts.h(1), at(h2));
  keep(acts.h(2), at(h3));
  if (in && (tid & 15) == 0) acts.d()[row] = d;
  {  // dL/d(pre-activation 3)
    const float4 h = at(h3);
    const float4 v = make_float4(h.x > 0.f ? d * w4[j] : 0.f, h.y > 0.f ? d * w4[j + 1] : 0.f,
                                 h.z > 0.f ? d * w4[j + 2] : 0.f, h.w > 0.f ? d * w4[j + 3] : 0.f);
    keep(acts.g(2), v);
    put(g, v);
  }
  __syncthreads();
  // back through w3, then w2: units u, u + 16, u + 32, u + 48 of the row below,
  // each a dot product with a row of the weights
  const int u = tid & 15;
  for (int L = 1; L >= 0; L--) {
    const float *w = L == 1 ? w3 : w2, *below = L == 1 ? h2 : h1;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int c = 0; c < H; c += 4) {
      const float4 e = *reinterpret_cast<const float4 *>(g + s * LD + c);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float4 v = *reinterpret_cast<const float4 *>(w + (u + 16 * k) * LD + c);
        acc[k] = fmaf(e.x, v.x, acc[k]);
        acc[k] = fmaf(e.y, v.y, acc[k]);
        acc[k] = fmaf(e.z, v.z, acc[k]);
        acc[k] = fmaf(e.w, v.w, acc[k]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = u + 16 * k;
      const float v = below[s * LD + i] > 0.f ? acc[k] : 0.f;
      g[s * LD + i] = v;
      if (in) acts.g(L)[(size_t)row * H + i] = v;
    }
    __syncthreads();
  }
}

struct MlpAdam {
  float *params, *m, *v;
  float lr, b1, b2, c1, c2;
};

// One Adam step of a parameter from its state (m, v, p).
__device__ __forceinline__ void adam_step(const MlpAdam &A, int i, float3 mvp, float gp) {
  const float mp = A.b1 * mvp.x + (1.f - A.b1) * gp;
  const float vp = A.b2 * mvp.y + (1.f - A.b2) * gp * gp;
  A.m[i] = mp;
  A.v[i] = vp;
  A.params[i] = mvp.z - A.lr * (mp / A.c1) / (sqrtf(vp / A.c2) + 1e-8f);
}
__device__ __forceinline__ float3 adam_state(const MlpAdam &A, int i) {
  return make_float3(A.m[i], A.v[i], A.params[i]);
}

// Gradients of 8 rows of one layer's weights, its bias being one row more
// whose input is 1: for weight row i, unit j the sum over the batch of
// in[s][i] * err[s][j].  blockIdx.x counts the CTAs of layers 1, 2, 3, then
// one for the output layer, whose weights are one row with the output's error
// for input and h3 for error.  Rows [64 blockIdx.y ..) with gridDim.y > 1,
// else all of them.  A gradient goes to out[blockIdx.y * count + p], or into
// an Adam step (adam.params).
struct MlpChunk {  // one slot of rows: errors, and inputs of 8 weight rows
  float err[kMlpSlot][kMlpHidden];
  float in[kMlpSlot][kMlpGradRows + 1];
};
constexpr int kMlpStages = 4;  // chunks in flight

__global__ void __launch_bounds__(kMlpGradThreads)
    k_mlp_grad(int F, const float *X, int n, MlpActs acts, float *out, MlpAdam adam) {
  constexpr int H = kMlpHidden;
  extern __shared__ __align__(16) float sm[];
  MlpChunk *ring = reinterpret_cast<MlpChunk *>(sm);
  const MlpShape S(F);
  const int tid = threadIdx.x, ti = tid >> 4, j = 4 * (tid & 15);
  int b = blockIdx.x, layer = 0, K = F;
  while (layer < 3 && b >= (K + kMlpGradRows) / kMlpGradRows) {
    b -= (K + kMlpGradRows) / kMlpGradRows;  // ceil((K + 1) / 8)
    layer++;
    K = H;
  }
  const int i0 = b * kMlpGradRows, i = i0 + ti;
  const bool last = layer == 3;  // the output layer: row 0 alone
  const float *src = layer == 0 ? X : last ? acts.d() : acts.h(layer - 1);
  const float *e = last ? acts.h(2) : acts.g(layer);
  const int r_begin = gridDim.y > 1 ? blockIdx.y * kMlpSlot : 0;
  const int r_end = gridDim.y > 1 && r_begin + kMlpSlot < n ? r_begin + kMlpSlot : n;
  const int chunks = (r_end - r_begin + kMlpSlot - 1) / kMlpSlot;
  auto load = [&](int c) {
    if (c < chunks) {
      MlpChunk &M = ring[c % kMlpStages];
      const int r = r_begin + c * kMlpSlot;
      const int rows = r_end - r < kMlpSlot ? r_end - r : kMlpSlot;
      for (int q = tid; q < kMlpSlot * H / 4; q += kMlpGradThreads) {
        const int s = q / (H / 4), u = 4 * (q % (H / 4));
        if (s < rows) copy16(&M.err[s][u], e + (size_t)(r + s) * H + u);
      }
      for (int q = tid; q < kMlpSlot * kMlpGradRows; q += kMlpGradThreads) {
        const int s = q / kMlpGradRows, k = q % kMlpGradRows;
        if (s >= rows) continue;
        if (last) {
          if (k == 0) copy4(&M.in[s][0], src + r + s);
          else M.in[s][k] = 0.f;
        } else if (i0 + k < K) {
          copy4(&M.in[s][k], src + (size_t)(r + s) * K + i0 + k);
        } else {
          M.in[s][k] = i0 + k == K ? 1.f : 0.f;
        }
      }
    }
    copy_commit();
  };
  grid_wait();
  for (int c = 0; c < kMlpStages - 1; c++) load(c);
  const int off_w = layer == 0 ? S.off_w1 : layer == 1 ? S.off_w2 : layer == 2 ? S.off_w3 : S.off_w4;
  const bool mine = last ? i == 0 : i <= K;  // a layer's bias follows its weights
  const bool mine4 = last && tid == 0;       // and the output bias
  const int p = off_w + i * H + j;
  float3 state[4], state4;  // Adam's state, in flight with the rows
  if (adam.params && mine)
#pragma unroll
    for (int k = 0; k < 4; k++) state[k] = adam_state(adam, p + k);
  if (adam.params && mine4) state4 = adam_state(adam, S.off_b4);
  float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
  float bias4 = 0.f;  // of the output layer
  for (int c = 0; c < chunks; c++) {
    copy_wait<kMlpStages - 2>();
    __syncthreads();  // chunk c is here, and the ring slot of chunk c - 1 is free
    load(c + kMlpStages - 1);
    const MlpChunk &M = ring[c % kMlpStages];
    const int left = r_end - r_begin - c * kMlpSlot;
    const int rows = left < kMlpSlot ? left : kMlpSlot;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int s = 0; s < rows; s++) {
      const float x = M.in[s][ti];
      const float4 v = *reinterpret_cast<const float4 *>(&M.err[s][j]);
      acc.x = fmaf(x, v.x, acc.x);
      acc.y = fmaf(x, v.y, acc.y);
      acc.z = fmaf(x, v.z, acc.z);
      acc.w = fmaf(x, v.w, acc.w);
    }
    total.x += acc.x;
    total.y += acc.y;
    total.z += acc.z;
    total.w += acc.w;
    if (mine4) {
      float a = 0.f;
      for (int s = 0; s < rows; s++) a += M.in[s][0];
      bias4 += a;
    }
  }
  if (mine) {
    const float g[4] = {total.x, total.y, total.z, total.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (adam.params) adam_step(adam, p + k, state[k], g[k]);
      else out[(size_t)blockIdx.y * S.count + p + k] = g[k];
    }
  }
  if (mine4) {
    if (adam.params) adam_step(adam, S.off_b4, state4, bias4);
    else out[(size_t)blockIdx.y * S.count + S.off_b4] = bias4;
  }
}

static int mlp_grad_blocks(int F) {
  return (F + kMlpGradRows) / kMlpGradRows + 2 * ((kMlpHidden + kMlpGradRows) / kMlpGradRows) + 1;
}

// Sum the slots of a large batch in order.
__global__ void k_mlp_reduce(const float *slots, int nslots, int count, float *grad) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= count) return;
  float a = 0.f;
  for (int k = 0; k < nslots; k++) a += slots[(size_t)k * count + p];
  grad[p] = a;
}

// Sum of the rows' squared errors, in a fixed order.
__global__ void __launch_bounds__(256) k_mlp_loss(const double *loss_rows, int n, double *loss) {
  __shared__ double part[8];
  double a = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) a += loss_rows[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; k++) a += part[k];
    *loss = a;
  }
}

__global__ void k_adam(const float *grad, int count, MlpAdam adam) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < count) adam_step(adam, p, adam_state(adam, p), grad[p]);
}

}  // namespace qcs

struct qcs_cuda_costmodel {
  int F;
  int count;
  float *d_params, *d_grad, *d_m, *d_v;
  double *d_loss_rows, *d_loss;
  float *d_x, *d_y, *d_pred;
  int cap_rows;
  float *d_acts, *d_slots;  // for gradients of up to cap_grad rows
  int cap_grad;
  int step;
  std::vector<float> host_params;  // mirror for planning on the host
  unsigned long long generation;   // bumped whenever host_params change
  bool host_only;                  // no device: host planning only
  cudaStream_t stream;
};

namespace qcs {

static size_t mlp_smem(int F) {
  return sizeof(float) * ((size_t)(F + 2 * kMlpHidden + 4 * kMlpRows) * kMlpPitch +
                          4 * kMlpHidden + (size_t)kMlpRows * ((F + 3) & ~3));
}

static int cm_reserve(qcs_cuda_costmodel *m, int rows) {
  if (rows <= m->cap_rows) return QCS_CUDA_OK;
  cudaFree(m->d_x);
  cudaFree(m->d_y);
  cudaFree(m->d_pred);
  cudaFree(m->d_loss_rows);
  m->d_x = m->d_y = m->d_pred = nullptr;
  m->d_loss_rows = nullptr;
  m->cap_rows = 0;
  int rc = check_cuda(cudaMalloc((void **)&m->d_x, (size_t)rows * m->F * sizeof(float)), "cudaMalloc(mlp)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_y, (size_t)rows * sizeof(float)), "cudaMalloc(mlp)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_pred, (size_t)rows * sizeof(float)), "cudaMalloc(mlp)");
  if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_loss_rows, (size_t)rows * sizeof(double)), "cudaMalloc(mlp)");
  if (!rc) m->cap_rows = rows;
  return rc;
}

static int cm_reserve_grad(qcs_cuda_costmodel *m, int rows) {
  if (rows <= m->cap_grad) return QCS_CUDA_OK;
  cudaFree(m->d_acts);
  cudaFree(m->d_slots);
  m->d_acts = m->d_slots = nullptr;
  m->cap_grad = 0;
  const size_t nslots = rows > kMlpDirectRows ? ((size_t)rows + kMlpSlot - 1) / kMlpSlot : 0;
  const size_t kept = rows < kMlpPieceRows ? rows : kMlpPieceRows;
  int rc = check_cuda(cudaMalloc((void **)&m->d_acts, kept * kMlpActs * sizeof(float)), "cudaMalloc(mlp)");
  if (!rc && nslots)
    rc = check_cuda(cudaMalloc((void **)&m->d_slots, nslots * m->count * sizeof(float)), "cudaMalloc(mlp)");
  if (!rc) m->cap_grad = rows;
  return rc;
}

// Forward over rows [0, n) of the device arrays x/y, keeping the rows' squared
// errors, and the gradient of their mean: into d_grad, or into an Adam step.
static int cm_grad_device(qcs_cuda_costmodel *m, const float *x, const float *y, int n,
                          const MlpAdam *adam) {
  MlpActs acts;
  acts.p = m->d_acts;
  acts.rows = (size_t)(m->cap_grad < kMlpPieceRows ? m->cap_grad : kMlpPieceRows);
  MlpAdam none;
  memset(&none, 0, sizeof(none));
  auto rows_pass = [&](i64 r, int rows) {
    launch_next(true, k_mlp_rows, (rows + kMlpRows - 1) / kMlpRows, kMlpRowThreads, mlp_smem(m->F),
                m->stream, m->d_params, m->F, x + r * m->F, y + r, rows, 1.f / n, acts,
                m->d_loss_rows + r, (float *)nullptr);
    return check_launch("cost model rows");
  };
  if (n <= kMlpDirectRows) {
    int rc = rows_pass(0, n);
    if (rc) return rc;
    launch_next(true, k_mlp_grad, mlp_grad_blocks(m->F), kMlpGradThreads,
                kMlpStages * sizeof(MlpChunk), m->stream, m->F, x, n, acts, m->d_grad,
                adam ? *adam : none);
    return check_launch("cost model gradient");
  }
  int rc = QCS_CUDA_OK;
  for (i64 r = 0; !rc && r < n; r += kMlpPieceRows) {
    const int rows = (int)(n - r < kMlpPieceRows ? n - r : kMlpPieceRows);
    rc = rows_pass(r, rows);
    if (rc) return rc;
    k_mlp_grad<<<dim3(mlp_grad_blocks(m->F), (rows + kMlpSlot - 1) / kMlpSlot), kMlpGradThreads,
                 kMlpStages * sizeof(MlpChunk), m->stream>>>(
        m->F, x + r * m->F, rows, acts, m->d_slots + r / kMlpSlot * m->count, none);
    rc = check_launch("cost model gradient");
  }
  if (rc) return rc;
  const int nslots = (int)(((i64)n + kMlpSlot - 1) / kMlpSlot);
  k_mlp_reduce<<<(m->count + 255) / 256, 256, 0, m->stream>>>(m->d_slots, nslots, m->count,
                                                              m->d_grad);
  rc = check_launch("cost model gradient sum");
  if (rc || !adam) return rc;
  k_adam<<<(m->count + 255) / 256, 256, 0, m->stream>>>(m->d_grad, m->count, *adam);
  return check_launch("adam");
}

// Mean squared error over rows already on the device.
static int cm_loss(qcs_cuda_costmodel *m, int n, double *loss) {
  k_mlp_loss<<<1, 256, 0, m->stream>>>(m->d_loss_rows, n, m->d_loss);
  int rc = check_launch("cost model loss");
  double l = 0.0;
  if (!rc) rc = check_cuda(cudaMemcpyAsync(&l, m->d_loss, sizeof(double), cudaMemcpyDeviceToHost, m->stream), "loss");
  if (!rc) rc = check_cuda(cudaStreamSynchronize(m->stream), "sync");
  if (!rc && loss) *loss = l / n;
  return rc;
}

static int cm_upload(qcs_cuda_costmodel *m, const float *x, const float *y, int n) {
  int rc = cm_reserve(m, n);
  if (!rc) rc = check_cuda(cudaMemcpyAsync(m->d_x, x, (size_t)n * m->F * 4, cudaMemcpyHostToDevice, m->stream), "upload");
  if (!rc && y) rc = check_cuda(cudaMemcpyAsync(m->d_y, y, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream), "upload");
  return rc;
}

// Forward only: predictions, or (with y) the rows' squared errors.
static int cm_forward(qcs_cuda_costmodel *m, const float *x, const float *y, int n) {
  MlpActs none = {nullptr, 0};
  k_mlp_rows<<<(n + kMlpRows - 1) / kMlpRows, kMlpRowThreads, mlp_smem(m->F), m->stream>>>(
      m->d_params, m->F, x, y, n, 1.f / n, none, y ? m->d_loss_rows : nullptr,
      y ? nullptr : m->d_pred);
  return check_launch("cost model forward");
}

// Generations are unique across models, so a plan kept for a destroyed model
// never matches a new model that happens to reuse its address.
static std::atomic<unsigned long long> g_cm_generation{0};

static int cm_sync_host(qcs_cuda_costmodel *m) {
  m->generation = ++g_cm_generation;
  m->host_params.resize(m->count);
  int rc = check_cuda(cudaMemcpyAsync(m->host_params.data(), m->d_params, m->count * sizeof(float),
                                      cudaMemcpyDeviceToHost, m->stream),
                      "cost model params");
  return rc ? rc : check_cuda(cudaStreamSynchronize(m->stream), "cost model sync");
}

// Host forward pass (used while planning), FP32 like the device: every
// output sums its inputs in index order, as the row-major loops below do
// with the input index outermost.
float costmodel_predict_host(const qcs_cuda_costmodel *m, const float *x) {
  const MlpShape S(m->F);
  const float *w = m->host_params.data();
  float h[kMlpHidden], t[kMlpHidden];
  memcpy(h, w + S.off_b1, sizeof(h));
  for (int i = 0; i < m->F; i++) {
    const float xi = x[i];
    if (xi == 0.f) continue;  // one-hot and flag features are mostly zero
    const float *row = w + S.off_w1 + i * kMlpHidden;
    for (int j = 0; j < kMlpHidden; j++) h[j] += xi * row[j];
  }
  for (int j = 0; j < kMlpHidden; j++) h[j] = h[j] > 0.f ? h[j] : 0.f;
  const int wo[2] = {S.off_w2, S.off_w3}, bo[2] = {S.off_b2, S.off_b3};
  for (int L = 0; L < 2; L++) {
    memcpy(t, w + bo[L], sizeof(t));
    for (int i = 0; i < kMlpHidden; i++) {
      const float hi = h[i];
      if (hi == 0.f) continue;  // ReLU zeros
      const float *row = w + wo[L] + i * kMlpHidden;
      for (int j = 0; j < kMlpHidden; j++) t[j] += hi * row[j];
    }
    for (int j = 0; j < kMlpHidden; j++) h[j] = t[j] > 0.f ? t[j] : 0.f;
  }
  float o = w[S.off_b4];
  for (int i = 0; i < kMlpHidden; i++) o += h[i] * w[S.off_w4 + i];
  return o;
}

unsigned long long costmodel_generation(const qcs_cuda_costmodel *m) { return m->generation; }

bool costmodel_ready(const qcs_cuda_costmodel *m) { return m && !m->host_params.empty(); }
int costmodel_features(const qcs_cuda_costmodel *m) { return m->F; }

}  // namespace qcs

using namespace qcs;

extern "C" {

int qcs_cuda_costmodel_create(int num_features, unsigned long long seed, qcs_cuda_costmodel **out) {
  if (!out || num_features < 1 || num_features > 64)
    return set_error(QCS_CUDA_EINVAL, "cost model: 1..64 features");
  *out = nullptr;
  int ndev = 0;
  const bool host_only = cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0;
  if (host_only) cudaGetLastError();
  qcs_cuda_costmodel *m = new qcs_cuda_costmodel();
  m->F = num_features;
  m->count = MlpShape(num_features).count;
  m->host_only = host_only;
  int rc = QCS_CUDA_OK;
  if (!host_only) {
    rc = check_cuda(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    const size_t pb = (size_t)m->count * sizeof(float);
    if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_params, pb), "cudaMalloc(mlp)");
    if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_grad, pb), "cudaMalloc(mlp)");
    if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_m, pb), "cudaMalloc(mlp)");
    if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_v, pb), "cudaMalloc(mlp)");
    if (!rc) rc = check_cuda(cudaMalloc((void **)&m->d_loss, sizeof(double)), "cudaMalloc(mlp)");
    if (!rc)
      rc = check_cuda(cudaFuncSetAttribute(k_mlp_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)mlp_smem(64)),
                      "cudaFuncSetAttribute(mlp)");
    if (!rc)
      rc = check_cuda(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(kMlpStages * sizeof(MlpChunk))),
                      "cudaFuncSetAttribute(mlp)");
    if (rc) {
      qcs_cuda_costmodel_destroy(m);
      return rc;
    }
  }
  // He initialisation from a splitmix64 stream (host), biases zero
  std::vector<float> p(m->count, 0.f);
  const MlpShape S(num_features);
  unsigned long long st = seed;
  auto unif = [&]() {
    st += 0x9E3779B97F4A7C15ULL;
    unsigned long long z = st;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  auto normal = [&]() {
    double u1 = unif(), u2 = unif();
    if (u1 < 1e-300) u1 = 1e-300;
    return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
  };
  const int fan[4] = {num_features, kMlpHidden, kMlpHidden, kMlpHidden};
  const int off[4] = {S.off_w1, S.off_w2, S.off_w3, S.off_w4};
  const int cnt[4] = {num_features * kMlpHidden, kMlpHidden * kMlpHidden, kMlpHidden * kMlpHidden,
                      kMlpHidden};
  for (int L = 0; L < 4; L++) {
    const double sd = sqrt(2.0 / fan[L]);
    for (int i = 0; i < cnt[L]; i++) p[off[L] + i] = (float)(sd * normal());
  }
  rc = qcs_cuda_costmodel_set_params(m, p.data(), m->count);
  if (rc) {
    qcs_cuda_costmodel_destroy(m);
    return rc;
  }
  *out = m;
  return QCS_CUDA_OK;
}

int qcs_cuda_costmodel_destroy(qcs_cuda_costmodel *m) {
  if (!m) return set_error(QCS_CUDA_EINVAL, "null model");
  if (m->host_only) {
    delete m;
    return QCS_CUDA_OK;
  }
  if (m->stream) cudaStreamSynchronize(m->stream);
  cudaFree(m->d_params);
  cudaFree(m->d_grad);
  cudaFree(m->d_m);
  cudaFree(m->d_v);
  cudaFree(m->d_loss);
  cudaFree(m->d_x);
  cudaFree(m->d_y);
  cudaFree(m->d_pred);
  cudaFree(m->d_acts);
  cudaFree(m->d_slots);
  cudaFree(m->d_loss_rows);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
  return QCS_CUDA_OK;
}

int qcs_cuda_costmodel_num_params(qcs_cuda_costmodel *m, int *count) {
  if (!m || !count) return set_error(QCS_CUDA_EINVAL, "null argument");
  *count = m->count;
  return QCS_CUDA_OK;
}

int qcs_cuda_costmodel_get_params(qcs_cuda_costmodel *m, float *out) {
  if (!m || !out) return set_error(QCS_CUDA_EINVAL, "null argument");
  int rc = m->host_only ? QCS_CUDA_OK : cm_sync_host(m);
  if (!rc) memcpy(out, m->host_params.data(), m->count * sizeof(float));
  return rc;
}

int qcs_cuda_costmodel_set_params(qcs_cuda_costmodel *m, const float *in, int count) {
  if (!m || !in || count != m->count) return set_error(QCS_CUDA_EINVAL, "bad parameter vector");
  if (m->host_only) {
    m->host_params.assign(in, in + count);
    m->generation = ++g_cm_generation;
    return QCS_CUDA_OK;
  }
  int rc = check_cuda(cudaMemcpyAsync(m->d_params, in, count * sizeof(float), cudaMemcpyHostToDevice,
                                      m->stream),
                      "cost model params");
  if (!rc) rc = check_cuda(cudaMemsetAsync(m->d_m, 0, count * sizeof(float), m->stream), "adam");
  if (!rc) rc = check_cuda(cudaMemsetAsync(m->d_v, 0, count * sizeof(float), m->stream), "adam");
  m->step = 0;
  return rc ? rc : cm_sync_host(m);
}

int qcs_cuda_costmodel_loss_grad(qcs_cuda_costmodel *m, const float *x, const float *y, int n,
                                 double *loss, float *grad) {
  if (!m || !x || !y || n < 1) return set_error(QCS_CUDA_EINVAL, "bad arguments");
  if (m->host_only) return set_error(QCS_CUDA_ENODEV, "cost model without a device: planning only");
  int rc = cm_upload(m, x, y, n);
  if (!rc && !grad) rc = cm_forward(m, m->d_x, m->d_y, n);
  if (!rc && grad) {
    rc = cm_reserve_grad(m, n);
    if (!rc) rc = cm_grad_device(m, m->d_x, m->d_y, n, nullptr);
    if (!rc)
      rc = check_cuda(cudaMemcpyAsync(grad, m->d_grad, m->count * sizeof(float), cudaMemcpyDeviceToHost, m->stream), "grad");
  }
  return rc ? rc : cm_loss(m, n, loss);
}

int qcs_cuda_costmodel_train(qcs_cuda_costmodel *m, const float *x, const float *y, int n,
                             int epochs, int batch, float lr, double *final_loss) {
  if (!m || !x || !y || n < 1 || epochs < 1 || batch < 1) return set_error(QCS_CUDA_EINVAL, "bad arguments");
  if (m->host_only) return set_error(QCS_CUDA_ENODEV, "cost model without a device: planning only");
  if (batch > n) batch = n;
  int rc = cm_upload(m, x, y, n);
  if (!rc) rc = cm_reserve_grad(m, batch);
  MlpAdam adam;
  adam.params = m->d_params;
  adam.m = m->d_m;
  adam.v = m->d_v;
  adam.lr = lr;
  adam.b1 = 0.9f;
  adam.b2 = 0.999f;
  for (int e = 0; !rc && e < epochs; e++) {
    for (int r = 0; !rc && r < n; r += batch) {
      const int rows = n - r < batch ? n - r : batch;
      m->step++;
      adam.c1 = 1.f - powf(adam.b1, (float)m->step);
      adam.c2 = 1.f - powf(adam.b2, (float)m->step);
      rc = cm_grad_device(m, m->d_x + (size_t)r * m->F, m->d_y + r, rows, &adam);
    }
  }
  if (!rc && final_loss) {
    rc = cm_forward(m, m->d_x, m->d_y, n);
    if (!rc) rc = cm_loss(m, n, final_loss);
  }
  if (!rc) rc = cm_sync_host(m);
  return rc;
}

int qcs_cuda_costmodel_predict(qcs_cuda_costmodel *m, const float *x, int n, float *out) {
  if (!m || !x || !out || n < 1) return set_error(QCS_CUDA_EINVAL, "bad arguments");
  if (m->host_only) return set_error(QCS_CUDA_ENODEV, "cost model without a device: planning only");
  int rc = cm_upload(m, x, nullptr, n);
  if (!rc) rc = cm_forward(m, m->d_x, nullptr, n);
  if (!rc) rc = check_cuda(cudaMemcpyAsync(out, m->d_pred, (size_t)n * 4, cudaMemcpyDeviceToHost, m->stream), "predict");
  return rc ? rc : check_cuda(cudaStreamSynchronize(m->stream), "sync");
}

int qcs_cuda_costmodel_predict_host(qcs_cuda_costmodel *m, const float *x, int n, float *out) {
  if (!m || !x || !out || n < 1) return set_error(QCS_CUDA_EINVAL, "bad arguments");
  for (int i = 0; i < n; i++) out[i] = costmodel_predict_host(m, x + (size_t)i * m->F);
  return QCS_CUDA_OK;
}

}  // extern "C"
