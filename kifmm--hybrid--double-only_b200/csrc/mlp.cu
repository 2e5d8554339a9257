// Cost-model network: a 3-layer perceptron (FP32) trained and evaluated on the
// GPU by the kernels below (no counterpart in the reference, which takes its
// leaf size from the command line).
//
//   H1 = relu(X W1 + b1)   X: B x F,  W1: F x H
//   H2 = relu(H1 W2 + b2)  W2: H x H
//   Y  = H2 W3 + b3        W3: H x O
//   loss = mean over B x O of (Y - T)^2
//
// Parameters are one packed float array [W1 | b1 | W2 | b2 | W3 | b3], each
// weight matrix row-major (input index major).  Gradients use the same
// layout.  Training is full-batch Adam (beta1 0.9, beta2 0.999, eps 1e-8).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "host.h"

namespace kfmm {
namespace {

constexpr int kMlpThreads = 256;

struct Layout {
  int F, H, O;
  size_t w1, b1, w2, b2, w3, b3, total;
  Layout(int f, int h, int o) : F(f), H(h), O(o) {
    w1 = 0;
    b1 = w1 + (size_t)F * H;
    w2 = b1 + H;
    b2 = w2 + (size_t)H * H;
    w3 = b2 + H;
    b3 = w3 + (size_t)H * O;
    total = b3 + O;
  }
};

// The layers' products are C[m, n] = sum_k A[m, k] B[k, n] in FP32, tiles of 64 x 64
// outputs per block of 256 threads (4 x 4 outputs a thread), 16-deep slices of A
// and B staged in shared memory, the next slice loaded into registers meanwhile.
// At the cost model's sizes (B 19,200, F 73, H 64, O 5) a product is 0.1 to 0.2
// GFLOP and launch latency bounds it; the point of the tiles is that every
// product fills the device, the weight gradients (short outputs, sums over the
// whole batch) by splitting the batch.
// Ten training steps at those sizes, host copies included: 48 ms with a thread per
// output (the weight gradients serial over the batch), 2.1 to 2.7 ms now.
constexpr int kTile = 64, kTileK = 16;

struct __align__(16) TileSmem {  // read as float4
  float a[kTileK][kTile + 4];
  float b[kTileK][kTile + 4];
};

// One tile's outputs over k in [k0, k1): av(k, m) and bv(k, n) give the tile's
// elements (0 outside the matrices); bsum, where not null, also receives sum_k
// bv(k, n) of column n = threadIdx.x < kTile.
// kARow, kBRow: whether consecutive k (rather than consecutive m or n) are
// consecutive in memory, so that a warp's loads are.
template <bool kARow, bool kBRow, class FA, class FB>
__device__ __forceinline__ void tile_product(TileSmem& s, int k0, int k1, FA av, FB bv,
                                             float (&acc)[4][4], float* bsum) {
  const int tid = threadIdx.x, tm = (tid >> 4) * 4, tn = (tid & 15) * 4;
  constexpr int kPer = kTile * kTileK / kMlpThreads;
  float ra[kPer], rb[kPer], colsum = 0.f;
  auto at = [&](bool row, int q, int& k, int& i) {
    if (row) {
      k = q % kTileK;
      i = q / kTileK;
    } else {
      k = q / kTile;
      i = q % kTile;
    }
  };
  auto fetch = [&](int kb) {
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
      int k, i;
      at(kARow, tid + r * kMlpThreads, k, i);
      ra[r] = kb + k < k1 ? av(kb + k, i) : 0.f;
      at(kBRow, tid + r * kMlpThreads, k, i);
      rb[r] = kb + k < k1 ? bv(kb + k, i) : 0.f;
    }
  };
  if (k0 < k1) fetch(k0);
  for (int kb = k0; kb < k1; kb += kTileK) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
      int k, i;
      at(kARow, tid + r * kMlpThreads, k, i);
      s.a[k][i] = ra[r];
      at(kBRow, tid + r * kMlpThreads, k, i);
      s.b[k][i] = rb[r];
    }
    __syncthreads();
    if (kb + kTileK < k1) fetch(kb + kTileK);
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      const float4 a = *(const float4*)&s.a[k][tm], b = *(const float4*)&s.b[k][tn];
      const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
      if (bsum && tid < kTile) colsum += s.b[k][tid];
    }
  }
  if (bsum) *bsum = colsum;
}

// Y = X W + bias, X: B x I, W: I x O; relu optional.  The output layer of a
// training step (T given) also writes dY = 2 (Y - T) / (B O) and the block's
// part of the sum of (Y - T)^2.
__global__ void __launch_bounds__(kMlpThreads)
dense_forward(int B, int I, int O, const float* X, const float* W, const float* bias, float* Y,
              int relu, const float* T, float* dY, float* sq) {
  __shared__ TileSmem s;
  __shared__ float red[kMlpThreads];
  const int b0 = blockIdx.x * kTile, o0 = blockIdx.y * kTile;
  const int tm = (threadIdx.x >> 4) * 4, tn = (threadIdx.x & 15) * 4;
  float acc[4][4] = {};
  tile_product<true, false>(
      s, 0, I, [&](int k, int m) { return b0 + m < B ? X[(size_t)(b0 + m) * I + k] : 0.f; },
      [&](int k, int n) { return o0 + n < O ? W[(size_t)k * O + o0 + n] : 0.f; }, acc, nullptr);
  const float scale = 2.f / ((float)B * (float)O);
  float mine = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = b0 + tm + i, o = o0 + tn + j;
      if (b >= B || o >= O) continue;
      const size_t q = (size_t)b * O + o;
      const float v = acc[i][j] + bias[o];
      Y[q] = relu ? fmaxf(v, 0.f) : v;
      if (T) {
        const float d = v - T[q];
        dY[q] = scale * d;
        mine = fmaf(d, d, mine);
      }
    }
  if (!T) return;
  red[threadIdx.x] = mine;
  __syncthreads();
  for (int w = kMlpThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) sq[blockIdx.y * gridDim.x + blockIdx.x] = red[0];
}

// dX[b, i] = (sum_o dY[b, o] W[i, o]) * (H[b, i] > 0), H the layer's relu output
__global__ void __launch_bounds__(kMlpThreads)
dense_input_grad(int B, int I, int O, const float* dY, const float* W, const float* H, float* dX) {
  __shared__ TileSmem s;
  const int b0 = blockIdx.x * kTile, i0 = blockIdx.y * kTile;
  const int tm = (threadIdx.x >> 4) * 4, tn = (threadIdx.x & 15) * 4;
  float acc[4][4] = {};
  tile_product<true, true>(
      s, 0, O, [&](int k, int m) { return b0 + m < B ? dY[(size_t)(b0 + m) * O + k] : 0.f; },
      [&](int k, int n) { return i0 + n < I ? W[(size_t)(i0 + n) * O + k] : 0.f; }, acc, nullptr);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = b0 + tm + i, n = i0 + tn + j;
      if (b < B && n < I) {
        const size_t q = (size_t)b * I + n;
        dX[q] = H[q] > 0.f ? acc[i][j] : 0.f;
      }
    }
}

// dW[i, o] = sum_b X[b, i] dY[b, o] and dbias[o] = sum_b dY[b, o] of the three
// layers in one launch: blockIdx.x walks the layers' tiles, blockIdx.y is one of
// the batch's ranges of `rows`, whose sums go to part[blockIdx.y][parameter].
struct WeightGradLayer {
  const float *X, *dY;
  int I, O;
  size_t w, b;  // the layer's weights and biases in the packed parameters
  int tile0, tiles_o;
};
struct WeightGradParams {
  WeightGradLayer layer[3];
  int B, rows;
  size_t total;
  float* part;
};

__global__ void __launch_bounds__(kMlpThreads) dense_weight_grad(WeightGradParams p) {
  __shared__ TileSmem s;
  const int tile = blockIdx.x;
  const WeightGradLayer L =
      p.layer[tile >= p.layer[2].tile0 ? 2 : tile >= p.layer[1].tile0 ? 1 : 0];
  const int i0 = (tile - L.tile0) / L.tiles_o * kTile, o0 = (tile - L.tile0) % L.tiles_o * kTile;
  const int tm = (threadIdx.x >> 4) * 4, tn = (threadIdx.x & 15) * 4;
  const int k0 = min((long long)p.B, (long long)blockIdx.y * p.rows);
  const int k1 = min((long long)p.B, (long long)k0 + p.rows);
  float acc[4][4] = {}, bsum = 0.f;
  tile_product<false, false>(
      s, k0, k1, [&](int k, int m) { return i0 + m < L.I ? L.X[(size_t)k * L.I + i0 + m] : 0.f; },
      [&](int k, int n) { return o0 + n < L.O ? L.dY[(size_t)k * L.O + o0 + n] : 0.f; }, acc,
      &bsum);
  float* out = p.part + (size_t)blockIdx.y * p.total;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + tm + i < L.I && o0 + tn + j < L.O)
        out[L.w + (size_t)(i0 + tm + i) * L.O + o0 + tn + j] = acc[i][j];
  if (i0 == 0 && threadIdx.x < kTile && o0 + (int)threadIdx.x < L.O)
    out[L.b + o0 + threadIdx.x] = bsum;
}

// The gradient from the batch ranges' sums (in range order), the loss from the
// blocks' parts (block 0), and, with m given, the Adam step.
__global__ void __launch_bounds__(kMlpThreads)
finish_step(int n, int nparts, const float* part, float* g, int nsq, const float* sq, float count,
            float* loss, float* p, float* m, float* v, float lr, float c1, float c2) {
  __shared__ float red[kMlpThreads];
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    float s = 0.f;
#pragma unroll 8
    for (int r = 0; r < nparts; ++r) s += part[(size_t)r * n + q];
    if (!m) {
      g[q] = s;
      continue;
    }
    m[q] = 0.9f * m[q] + 0.1f * s;
    v[q] = 0.999f * v[q] + 0.001f * s * s;
    p[q] -= lr * (m[q] / c1) / (sqrtf(v[q] / c2) + 1e-8f);
  }
  if (blockIdx.x != 0) return;
  float s = 0.f;
  for (int q = threadIdx.x; q < nsq; q += blockDim.x) s += sq[q];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = red[0] / count;
}

inline int tiles(int n) { return (n + kTile - 1) / kTile; }

// The network's arrays on the device, in one allocation.
struct Net {
  Layout L;
  int B, steps;  // steps: losses kept
  float *p, *g, *X, *T, *H1, *H2, *Y, *dY, *dH2, *dH1, *sq, *loss, *m, *v, *part;
  int nparts = 0, rows = 0, nsq = 0;
  WeightGradParams wg{};
  void* mem = nullptr;
  Net(int f, int h, int o, int b, int nlosses = 1) : L(f, h, o), B(b), steps(nlosses) {}
  ~Net() {
    if (mem) cudaFree(mem);
  }
  cudaError_t init(bool train) {
    const size_t n = L.total, b = B;
    wg.layer[0].tile0 = 0;
    wg.layer[1].tile0 = tiles(L.F) * tiles(L.H);
    wg.layer[2].tile0 = wg.layer[1].tile0 + tiles(L.H) * tiles(L.H);
    const int ntiles = wg.layer[2].tile0 + tiles(L.H) * tiles(L.O);
    nsq = tiles(B) * tiles(L.O);
    // ranges of the batch for the weight gradients: about 512 blocks over the
    // layers' tiles, at least 4 slices of the batch each
    nparts = std::max(1, std::min(512 / ntiles, (B + 4 * kTileK - 1) / (4 * kTileK)));
    rows = ((B + nparts - 1) / nparts + kTileK - 1) / kTileK * kTileK;
    nparts = (B + rows - 1) / rows;
    struct Part {
      float** at;
      size_t n;
    };
    std::vector<Part> parts = {{&p, n}, {&X, b * L.F}, {&H1, b * L.H}, {&H2, b * L.H}, {&Y, b * L.O}};
    if (train)
      for (const Part& q : std::vector<Part>{{&m, n}, {&v, n}, {&g, n}, {&T, b * L.O}, {&dY, b * L.O},
                                             {&dH2, b * L.H}, {&dH1, b * L.H}, {&sq, (size_t)nsq},
                                             {&loss, (size_t)steps}, {&part, n * nparts}})
        parts.push_back(q);
    size_t total = 0;
    for (const Part& q : parts) total += (q.n + 63) / 64 * 64;  // 256-byte aligned
    cudaError_t e = cudaMalloc(&mem, total * sizeof(float));
    if (e != cudaSuccess) {
      mem = nullptr;
      return e;
    }
    size_t at = 0;
    for (const Part& q : parts) {
      *q.at = (float*)mem + at;
      at += (q.n + 63) / 64 * 64;
    }
    if (!train) return cudaSuccess;
    wg.B = B;
    wg.rows = rows;
    wg.total = n;
    wg.part = part;
    wg.layer[0] = {X, dH1, L.F, L.H, L.w1, L.b1, wg.layer[0].tile0, tiles(L.H)};
    wg.layer[1] = {H1, dH2, L.H, L.H, L.w2, L.b2, wg.layer[1].tile0, tiles(L.H)};
    wg.layer[2] = {H2, dY, L.H, L.O, L.w3, L.b3, wg.layer[2].tile0, tiles(L.O)};
    if ((e = cudaMemset(m, 0, n * sizeof(float)))) return e;
    return cudaMemset(v, 0, n * sizeof(float));
  }
  void forward(bool train) {
    dense_forward<<<dim3(tiles(B), tiles(L.H)), kMlpThreads>>>(B, L.F, L.H, X, p + L.w1, p + L.b1, H1,
                                                               1, nullptr, nullptr, nullptr);
    dense_forward<<<dim3(tiles(B), tiles(L.H)), kMlpThreads>>>(B, L.H, L.H, H1, p + L.w2, p + L.b2,
                                                               H2, 1, nullptr, nullptr, nullptr);
    dense_forward<<<dim3(tiles(B), tiles(L.O)), kMlpThreads>>>(
        B, L.H, L.O, H2, p + L.w3, p + L.b3, Y, 0, train ? T : nullptr, train ? dY : nullptr,
        train ? sq : nullptr);
  }
  // gradients (step 0) or the step's Adam update; the step's loss to loss[at]
  void backward(int at, int step, float lr) {
    dense_input_grad<<<dim3(tiles(B), tiles(L.H)), kMlpThreads>>>(B, L.H, L.O, dY, p + L.w3, H2, dH2);
    dense_input_grad<<<dim3(tiles(B), tiles(L.H)), kMlpThreads>>>(B, L.H, L.H, dH2, p + L.w2, H1, dH1);
    dense_weight_grad<<<dim3(wg.layer[2].tile0 + tiles(L.H) * tiles(L.O), nparts), kMlpThreads>>>(wg);
    const float c1 = 1.f - std::pow(0.9f, (float)step), c2 = 1.f - std::pow(0.999f, (float)step);
    const int n = (int)L.total;
    finish_step<<<std::min((n + kMlpThreads - 1) / kMlpThreads, 1024), kMlpThreads>>>(
        n, nparts, part, g, nsq, sq, (float)B * (float)L.O, loss + at, p, step ? m : nullptr, v, lr,
        c1, c2);
  }
};

#define MLP_CUDA(call)                                                                    \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess) {                                                              \
      set_error(std::string("mlp: ") + #call + ": " + cudaGetErrorString(e_));            \
      return KFMM_ERR_CUDA;                                                               \
    }                                                                                     \
  } while (0)

bool bad_shape(int F, int H, int O, int B) {
  return F < 1 || H < 1 || O < 1 || B < 1 || F > 4096 || H > 4096 || O > 4096;
}

}  // namespace
}  // namespace kfmm

using namespace kfmm;

extern "C" kfmm_status kfmm_mlp_param_count(int F, int H, int O, long long* count) {
  if (!count || bad_shape(F, H, O, 1)) {
    set_error("kfmm_mlp_param_count: bad shape");
    return KFMM_ERR_INVALID;
  }
  *count = (long long)Layout(F, H, O).total;
  return KFMM_OK;
}

extern "C" kfmm_status kfmm_mlp_forward(int F, int H, int O, const float* params, int B,
                                        const float* X, float* Y) {
  if (!params || !X || !Y || bad_shape(F, H, O, B)) {
    set_error("kfmm_mlp_forward: bad argument");
    return KFMM_ERR_INVALID;
  }
  Net net(F, H, O, B);
  MLP_CUDA(net.init(false));
  MLP_CUDA(cudaMemcpy(net.p, params, sizeof(float) * net.L.total, cudaMemcpyHostToDevice));
  MLP_CUDA(cudaMemcpy(net.X, X, sizeof(float) * (size_t)B * F, cudaMemcpyHostToDevice));
  net.forward(false);
  MLP_CUDA(cudaGetLastError());
  MLP_CUDA(cudaMemcpy(Y, net.Y, sizeof(float) * (size_t)B * O, cudaMemcpyDeviceToHost));
  return KFMM_OK;
}

extern "C" kfmm_status kfmm_mlp_gradients(int F, int H, int O, const float* params, int B,
                                          const float* X, const float* T, float* grads,
                                          float* loss) {
  if (!params || !X || !T || !grads || !loss || bad_shape(F, H, O, B)) {
    set_error("kfmm_mlp_gradients: bad argument");
    return KFMM_ERR_INVALID;
  }
  Net net(F, H, O, B);
  MLP_CUDA(net.init(true));
  MLP_CUDA(cudaMemcpy(net.p, params, sizeof(float) * net.L.total, cudaMemcpyHostToDevice));
  MLP_CUDA(cudaMemcpy(net.X, X, sizeof(float) * (size_t)B * F, cudaMemcpyHostToDevice));
  MLP_CUDA(cudaMemcpy(net.T, T, sizeof(float) * (size_t)B * O, cudaMemcpyHostToDevice));
  net.forward(true);
  net.backward(0, 0, 0.f);
  MLP_CUDA(cudaGetLastError());
  MLP_CUDA(cudaMemcpy(grads, net.g, sizeof(float) * net.L.total, cudaMemcpyDeviceToHost));
  MLP_CUDA(cudaMemcpy(loss, net.loss, sizeof(float), cudaMemcpyDeviceToHost));
  return KFMM_OK;
}

extern "C" kfmm_status kfmm_mlp_train(int F, int H, int O, float* params, int B, const float* X,
                                      const float* T, int steps, float lr, float* losses) {
  if (!params || !X || !T || steps < 1 || !(lr > 0.f) || bad_shape(F, H, O, B)) {
    set_error("kfmm_mlp_train: bad argument");
    return KFMM_ERR_INVALID;
  }
  Net net(F, H, O, B, losses ? steps : 1);
  MLP_CUDA(net.init(true));
  MLP_CUDA(cudaMemcpy(net.p, params, sizeof(float) * net.L.total, cudaMemcpyHostToDevice));
  MLP_CUDA(cudaMemcpy(net.X, X, sizeof(float) * (size_t)B * F, cudaMemcpyHostToDevice));
  MLP_CUDA(cudaMemcpy(net.T, T, sizeof(float) * (size_t)B * O, cudaMemcpyHostToDevice));
  for (int s = 1; s <= steps; ++s) {
    net.forward(true);
    net.backward(losses ? s - 1 : 0, s, lr);
  }
  MLP_CUDA(cudaGetLastError());
  if (losses)
    MLP_CUDA(cudaMemcpy(losses, net.loss, sizeof(float) * (size_t)steps, cudaMemcpyDeviceToHost));
  MLP_CUDA(cudaMemcpy(params, net.p, sizeof(float) * net.L.total, cudaMemcpyDeviceToHost));
  return KFMM_OK;
}
