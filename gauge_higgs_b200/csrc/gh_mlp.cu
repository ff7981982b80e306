// gh_mlp.cu -- the coupling-scan surrogate: an ensemble of small MLPs trained and
// evaluated by the kernels below (no library GEMMs).
//
// Network (per member): n_in -> H -> ... -> H -> n_out, SiLU between layers,
// FP32 weights and optimiser state, BF16 storage of hidden activations (the
// pre-activations z are kept in FP32 for the SiLU derivative), FP32 accumulation.
// Loss: mean squared error over the batch and the outputs.  Optimiser: Adam with
// bias correction.  All members train on the same minibatches from their own
// initialisation; prediction returns the ensemble mean and variance.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "gh_rng.cuh"
#include "../../include/gauge_higgs_b200.h"

namespace {

constexpr int MAXL = 8;      // layers (weight matrices)

struct StepInfo { int s0, B, slot; float c1, c2; };   // first sample, batch, loss slot (-1: none), Adam bias corrections
struct Net {
  int M = 0, nl = 0;
  int width[MAXL + 1] = {};
  long woff[MAXL] = {}, boff[MAXL] = {};
  long P = 0;                 // parameters per member
  float* p = nullptr;         // [M][P]
  float* g = nullptr;         // [M][P] gradients
  float* m1 = nullptr;        // Adam first moment
  float* m2 = nullptr;        // Adam second moment
  long t = 0;                 // Adam step
  int cap = 0;                // batch capacity of the activation buffers
  float* z[MAXL] = {};        // [M][width[l+1]][cap] pre-activations (FP32)
  __nv_bfloat16* a[MAXL] = {};  // [M][width[l+1]][cap] activations (BF16), last layer unused
  float* out = nullptr;       // [M][n_out][cap]
  float* gz[MAXL] = {};       // [M][width[l+1]][cap] gradients w.r.t. pre-activations
  float* loss = nullptr;      // [loss_cap][M]
  int loss_cap = 0;
  float *xd = nullptr, *yd = nullptr;   // training set [ns_cap][n_in], [ns_cap][n_out]
  long ns_cap = 0;
  int* idx = nullptr;         // sample order of the steps of one launch
  long idx_cap = 0;
  StepInfo* steps = nullptr;
  long step_cap = 0;
  std::string err;
};

thread_local std::string g_mlp_err;
int mfail(Net* n, int code, const std::string& m) { if (n) n->err = m; g_mlp_err = m; return code; }

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) { const float s = 1.f / (1.f + __expf(-z)); return s * (1.f + z * (1.f - s)); }

// ---------------------------------------------------------------------------
// One kernel runs whole optimiser steps (or one gradient, or a forward pass): a cluster of
// CL blocks per network, which meets at the cluster's hardware barrier between layers.  A
// step is seven dependent layers of a few hundred kFLOP, so its time is latency: as
// separate launches (13 per step and two blocking copies of the minibatch, each thread
// walking its rows or columns of the weights alone in global memory) a step of 5 networks
// 4-128-128-128-3 at batch 32 took 333 us; here 43 us.
// Each layer is one tile product out[row][col] = init[col] + sum_k W(col, k) X(row, k):
//   forward   row = sample, col = neuron j, k = input i:  z = b + W a
//   backward  row = sample, col = input i,  k = neuron j: gz' = (W^T gz) silu'(z')
//   weights   row = input i, col = neuron j, k = sample:  dW = gz^T a (then Adam in place)
// A block owns a slice of the columns, a warp one column, a lane up to RG / 32 rows; the sum
// runs over k in ascending order in one FP32 chain, whatever the tiling.  Activations and
// gradients lie with the samples contiguous, as the lanes read and write them.
// ---------------------------------------------------------------------------
constexpr int CL = 8;        // blocks per network (the portable cluster size)
constexpr int TW = 16;       // warps per block = columns per pass
constexpr int RG = 128;      // rows per pass
constexpr int KC = 128;      // terms staged in shared memory at a time
constexpr int XS = RG + 1, WS = KC + 4;   // shared-memory strides: transposed stores without bank conflicts, 16-byte rows
constexpr size_t STEP_SMEM = sizeof(float) * ((size_t)KC * XS + TW * WS + 4);
enum { FORWARD = 0, GRADIENT = 1, TRAIN = 2 };

struct StepArgs {
  int nl, M, mode, nsteps, rows;       // rows: samples per cluster in FORWARD (grid.y splits them)
  int width[MAXL + 1];
  long woff[MAXL], boff[MAXL], P, cap;
  float *p, *g, *m1, *m2;
  const float *x, *y;
  const int* idx;                      // sample order (null: as they lie)
  float* z[MAXL];
  __nv_bfloat16* a[MAXL];
  float* gz[MAXL];
  float* out;
  float* loss;                         // [slot][M]
  const StepInfo* steps;
  float lr, b1, b2, eps;
};

__device__ __forceinline__ void adam_update(float* p, float* m1, float* m2, float gv, float lr, float b1, float b2, float eps,
                                            float c1, float c2) {
  const float a = b1 * *m1 + (1.f - b1) * gv;
  const float v = b2 * *m2 + (1.f - b2) * gv * gv;
  *m1 = a;
  *m2 = v;
  *p -= lr * (a / c1) / (sqrtf(v / c2) + eps);
}

// BIAS: acc[NR] sums the column's terms alone (the bias gradient)
template <int NR, bool BIAS>
__device__ __forceinline__ void tile_fma(const float* sx, const float* sw, int kn, float* acc, float& bias) {
  int k = 0;
#pragma unroll 4
  for (; k + 4 <= kn; k += 4) {
    const float4 w = *reinterpret_cast<const float4*>(sw + k);
    const float wk[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int r = 0; r < NR; ++r) acc[r] = fmaf(wk[q], sx[(k + q) * XS + 32 * r], acc[r]);
      if (BIAS) bias = fmaf(wk[q], 1.f, bias);
    }
  }
  for (; k < kn; ++k) {
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = fmaf(sw[k], sx[k * XS + 32 * r], acc[r]);
    if (BIAS) bias = fmaf(sw[k], 1.f, bias);
  }
}

// An nf x ns tile from global to shared memory: the threads of a warp along the first
// index (the contiguous one in memory), eight loads in flight per thread.
template <typename L, typename S>
__device__ __forceinline__ void stage(int nf, int ns, L load, S store) {
  const int sh = nf <= 16 ? 4 : nf <= 32 ? 5 : nf <= 64 ? 6 : 7, step = (TW * 32) >> sh;
  const int f = threadIdx.x & ((1 << sh) - 1);
  if (f >= nf) return;
  for (int b = threadIdx.x >> sh; b < ns; b += 8 * step) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b + u * step < ns) v[u] = load(f, b + u * step);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b + u * step < ns) store(f, b + u * step, v[u]);
  }
}

// rows [0, nrow), columns [c0, c1), terms [0, nk).  XK: X is contiguous in k (else in the
// row), WK: W is contiguous in k (else in the column).  epi(c, first row, rows, acc, bias)
// gets a lane's rows first row + 32 r.
template <bool XK, bool WK, bool BIAS, typename FX, typename FW, typename FI, typename FE>
__device__ __forceinline__ void tile_product(float* sx, float* sw, int nrow, int c0, int c1, int nk, FX X, FW W, FI init, FE epi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int cb = c0; cb < c1; cb += TW) {
    const int c = cb + warp, nc = min(TW, c1 - cb);
    for (int rb = 0; rb < nrow; rb += RG) {
      const int nr = min(RG, nrow - rb), nv = (nr + 31) >> 5;
      float acc[RG / 32], bias = 0.f;
#pragma unroll
      for (int r = 0; r < RG / 32; ++r) acc[r] = c < c1 ? init(c) : 0.f;
      for (int kb = 0; kb < nk; kb += KC) {
        const int kn = min(KC, nk - kb);
        __syncthreads();                       // earlier readers of the tiles are done
        if (XK) stage(kn, nr, [&](int k, int r) { return X(rb + r, kb + k); }, [&](int k, int r, float v) { sx[k * XS + r] = v; });
        else stage(nr, kn, [&](int r, int k) { return X(rb + r, kb + k); }, [&](int r, int k, float v) { sx[k * XS + r] = v; });
        if (WK) stage(kn, nc, [&](int k, int q) { return W(cb + q, kb + k); }, [&](int k, int q, float v) { sw[q * WS + k] = v; });
        else stage(nc, kn, [&](int q, int k) { return W(cb + q, kb + k); }, [&](int q, int k, float v) { sw[q * WS + k] = v; });
        __syncthreads();
        if (c < c1) {
          const float* px = sx + lane;
          const float* pw = sw + warp * WS;
          if (nv == 1) tile_fma<1, BIAS>(px, pw, kn, acc, bias);
          else if (nv == 2) tile_fma<2, BIAS>(px, pw, kn, acc, bias);
          else tile_fma<4, BIAS>(px, pw, kn, acc, bias);
        }
      }
      if (c < c1) epi(c, rb + lane, nrow, acc, bias);
    }
  }
}

__device__ __forceinline__ void cluster_barrier() {   // all threads; orders global memory among the cluster's blocks
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(TW * 32) k_steps(const StepArgs t) {
  extern __shared__ float smem[];
  float* sw = smem;                            // [TW][WS], 16-byte rows
  float* sx = smem + TW * WS;                  // [KC][XS]
  const int rank = blockIdx.x % CL, m = blockIdx.x / CL, nl = t.nl;
  float* p = t.p + m * t.P;
  const long cap = t.cap;
  const auto slice = [&](int n, int& c0, int& c1) {
    const int per = (n + CL - 1) / CL;
    c0 = min(n, rank * per);
    c1 = min(n, c0 + per);
  };
  for (int st = 0; st < t.nsteps; ++st) {
    StepInfo si;
    if (t.mode == FORWARD) {
      si.s0 = blockIdx.y * t.rows;
      si.B = min(t.rows, t.steps[0].B - si.s0);
      si.slot = -1;
    } else {
      si = t.steps[st];
    }
    const int B = si.B;
    const long first = t.mode == FORWARD ? si.s0 : 0;    // row of the activation buffers of sample s0
    const auto sample = [&](int b) { return (long)(t.idx ? t.idx[si.s0 + b] : si.s0 + b); };
    for (int l = 0; l < nl; ++l) {
      const int nin = t.width[l], nout = t.width[l + 1];
      const bool last = l == nl - 1;
      // a short output layer is computed by every block (the same values), which saves a barrier
      const bool dup = last && nout <= TW && nl > 1;
      int c0 = 0, c1 = nout;
      if (!dup) slice(nout, c0, c1);
      const float* w = p + t.woff[l];
      const float* bias = p + t.boff[l];
      const __nv_bfloat16* in = l ? t.a[l - 1] + m * cap * nin + first : nullptr;
      const long ob = m * cap * nout + first;
      const auto X = [&](int b, int k) { return l ? __bfloat162float(in[k * cap + b]) : t.x[sample(b) * nin + k]; };
      const auto W = [&](int j, int k) { return w[(long)j * nin + k]; };
      const auto I = [&](int j) { return bias[j]; };
      const auto E = [&](int j, int b0, int nrow, const float* acc, float) {
#pragma unroll
        for (int r = 0; r < RG / 32; ++r) {
          const int b = b0 + 32 * r;
          if (b >= nrow) break;
          const float v = acc[r];
          const long o = ob + j * cap + b;
          if (!last) {
            t.z[l][o] = v;
            t.a[l][o] = __float2bfloat16(silu(v));
          } else {
            t.out[o] = v;
            if (t.mode != FORWARD) {
              const float d = v - t.y[sample(b) * nout + j];
              t.gz[l][o] = 2.f * d / (float)(B * nout);
            }
          }
        }
      };
      tile_product<false, true, false>(sx, sw, B, c0, c1, nin, X, W, I, E);
      if (dup) __syncthreads();
      else cluster_barrier();
    }
    if (t.mode == FORWARD) return;
    if (si.slot >= 0 && rank == 0) {           // loss: mean of (out - y)^2, 256 strided sums and a tree
      const int nout = t.width[nl];
      float* sh = sx;
      __syncthreads();
      if (threadIdx.x < 256) {
        float s = 0.f;
        for (int e = threadIdx.x; e < B * nout; e += 256) {
          const float d = t.out[(m * nout + e % nout) * cap + e / nout] - t.y[sample(e / nout) * nout + e % nout];
          s += d * d;
        }
        sh[threadIdx.x] = s;
      }
      __syncthreads();
      for (int q = 128; q > 0; q >>= 1) {
        if ((int)threadIdx.x < q) sh[threadIdx.x] += sh[threadIdx.x + q];
        __syncthreads();
      }
      if (threadIdx.x == 0) t.loss[(long)si.slot * t.M + m] = sh[0] / (float)(B * nout);
    }
    for (int l = nl - 1; l > 0; --l) {         // gradient through layer l and the SiLU before it
      const int nin = t.width[l], nout = t.width[l + 1];
      const float* w = p + t.woff[l];
      const float* gz = t.gz[l] + m * cap * nout;
      const float* zp = t.z[l - 1] + m * cap * nin;
      float* gp = t.gz[l - 1] + m * cap * nin;
      int c0, c1;
      slice(nin, c0, c1);
      tile_product<false, false, false>(
          sx, sw, B, c0, c1, nout, [&](int b, int k) { return gz[k * cap + b]; },
          [&](int i, int k) { return w[(long)k * nin + i]; }, [](int) { return 0.f; },
          [&](int i, int b0, int nrow, const float* acc, float) {
#pragma unroll
            for (int r = 0; r < RG / 32; ++r)
              if (b0 + 32 * r < nrow) gp[i * cap + b0 + 32 * r] = acc[r] * dsilu(zp[i * cap + b0 + 32 * r]);
          });
      cluster_barrier();
    }
    for (int l = 0; l < nl; ++l) {             // weight gradients of this block's neurons, and Adam on them
      const int nin = t.width[l], nout = t.width[l + 1];
      const float* gz = t.gz[l] + m * cap * nout;
      const __nv_bfloat16* in = l ? t.a[l - 1] + m * cap * nin : nullptr;
      int c0, c1;
      slice(nout, c0, c1);
      const auto update = [&](long o, float v) {
        t.g[o] = v;
        if (t.mode == TRAIN) adam_update(t.p + o, t.m1 + o, t.m2 + o, v, t.lr, t.b1, t.b2, t.eps, si.c1, si.c2);
      };
      tile_product<true, true, true>(
          sx, sw, nin, c0, c1, B,
          [&](int i, int b) { return l ? __bfloat162float(in[i * cap + b]) : t.x[sample(b) * nin + i]; },
          [&](int j, int b) { return gz[j * cap + b]; }, [](int) { return 0.f; },
          [&](int j, int i0, int nrow, const float* acc, float bias) {
            const long o = m * t.P + t.woff[l] + (long)j * nin + i0;
            if (t.mode == TRAIN) {             // all loads of the weights and moments before the first store
              float pv[RG / 32], a1[RG / 32], a2[RG / 32];
#pragma unroll
              for (int r = 0; r < RG / 32; ++r)
                if (i0 + 32 * r < nrow) { pv[r] = t.p[o + 32 * r]; a1[r] = t.m1[o + 32 * r]; a2[r] = t.m2[o + 32 * r]; }
#pragma unroll
              for (int r = 0; r < RG / 32; ++r)
                if (i0 + 32 * r < nrow) {
                  adam_update(pv + r, a1 + r, a2 + r, acc[r], t.lr, t.b1, t.b2, t.eps, si.c1, si.c2);
                  t.p[o + 32 * r] = pv[r]; t.m1[o + 32 * r] = a1[r]; t.m2[o + 32 * r] = a2[r];
                }
            }
#pragma unroll
            for (int r = 0; r < RG / 32; ++r)
              if (i0 + 32 * r < nrow) t.g[o + 32 * r] = acc[r];
            if (i0 == 0) update(m * t.P + t.boff[l] + j, bias);
          });
    }
    cluster_barrier();                         // the next step reads the new weights and reuses the buffers
  }
}

__global__ void k_adam(float* p, const float* g, float* m1, float* m2, long n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x)
    adam_update(p + e, m1 + e, m2 + e, g[e], lr, b1, b2, eps, c1, c2);
}

int ensure_cap(Net* n, int B) {
  if (B <= n->cap) return GH_OK;
  auto fr = [](void* q) { if (q) cudaFree(q); };
  fr(n->out);
  n->out = nullptr;
  n->cap = 0;
  for (int l = 0; l < n->nl; ++l) { fr(n->z[l]); fr(n->a[l]); fr(n->gz[l]); n->z[l] = n->gz[l] = nullptr; n->a[l] = nullptr; }
  const int cap = std::max(B, 256);
  cudaError_t e = cudaSuccess;
  e = e ? e : cudaMalloc(&n->out, sizeof(float) * n->M * cap * n->width[n->nl]);
  for (int l = 0; l < n->nl && !e; ++l) {
    e = cudaMalloc(&n->z[l], sizeof(float) * n->M * cap * n->width[l + 1]);
    if (!e) e = cudaMalloc(&n->a[l], sizeof(__nv_bfloat16) * n->M * cap * n->width[l + 1]);
    if (!e) e = cudaMalloc(&n->gz[l], sizeof(float) * n->M * cap * n->width[l + 1]);
  }
  if (e) { cudaGetLastError(); return mfail(n, GH_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e)); }
  n->cap = cap;
  return GH_OK;
}

// A device array that only grows (contents are not kept).
template <typename T> cudaError_t grow(T** p, long* cap, long n) {
  if (n <= *cap) return cudaSuccess;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  const cudaError_t e = cudaMalloc(p, sizeof(T) * n);
  if (e == cudaSuccess) *cap = n;
  return e;
}

// The samples on the device; y may be null (forward).
int upload_samples(Net* n, const float* x, const float* y, long ns) {
  const int nin = n->width[0], nout = n->width[n->nl];
  cudaError_t e = cudaSuccess;
  if (ns > n->ns_cap) {
    if (n->xd) cudaFree(n->xd);
    if (n->yd) cudaFree(n->yd);
    n->xd = n->yd = nullptr;
    n->ns_cap = 0;
    const long c = std::max<long>(ns, 256);
    e = cudaMalloc(&n->xd, sizeof(float) * c * nin);
    if (!e) e = cudaMalloc(&n->yd, sizeof(float) * c * nout);
    if (e) { cudaGetLastError(); return mfail(n, GH_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e)); }
    n->ns_cap = c;
  }
  if (cudaMemcpy(n->xd, x, sizeof(float) * ns * nin, cudaMemcpyHostToDevice) ||
      (y && cudaMemcpy(n->yd, y, sizeof(float) * ns * nout, cudaMemcpyHostToDevice)))
    return mfail(n, GH_ERR_CUDA, "copy");
  return GH_OK;
}

// Runs `steps` (one for FORWARD and GRADIENT) over the uploaded samples; order: sample
// index of every row of the steps, null for the order they lie in.
int run_steps(Net* n, int mode, const std::vector<StepInfo>& steps, const std::vector<int>* order, int slots, float lr) {
  long lc = (long)n->loss_cap * n->M;
  cudaError_t e = grow(&n->steps, &n->step_cap, (long)steps.size());
  if (!e && order) e = grow(&n->idx, &n->idx_cap, (long)order->size());
  if (!e) e = grow(&n->loss, &lc, (long)std::max(slots, 1) * n->M);
  n->loss_cap = (int)(lc / n->M);
  if (!e) e = cudaMemcpy(n->steps, steps.data(), sizeof(StepInfo) * steps.size(), cudaMemcpyHostToDevice);
  if (!e && order) e = cudaMemcpy(n->idx, order->data(), sizeof(int) * order->size(), cudaMemcpyHostToDevice);
  if (!e) e = cudaFuncSetAttribute(k_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STEP_SMEM);
  if (e) { cudaGetLastError(); return mfail(n, GH_ERR_CUDA, std::string("MLP steps: ") + cudaGetErrorString(e)); }
  StepArgs t{};
  t.nl = n->nl; t.M = n->M; t.mode = mode; t.nsteps = (int)steps.size();
  t.P = n->P; t.cap = n->cap;
  for (int l = 0; l <= n->nl; ++l) t.width[l] = n->width[l];
  for (int l = 0; l < n->nl; ++l) {
    t.woff[l] = n->woff[l]; t.boff[l] = n->boff[l];
    t.z[l] = n->z[l]; t.a[l] = n->a[l]; t.gz[l] = n->gz[l];
  }
  t.p = n->p; t.g = n->g; t.m1 = n->m1; t.m2 = n->m2;
  t.x = n->xd; t.y = n->yd; t.idx = order ? n->idx : nullptr;
  t.out = n->out; t.loss = n->loss; t.steps = n->steps;
  t.lr = lr; t.b1 = 0.9f; t.b2 = 0.999f; t.eps = 1e-8f;
  t.rows = 64;                                  // forward rows are independent: clusters of 64 samples
  const int gy = mode == FORWARD ? (steps[0].B + t.rows - 1) / t.rows : 1;
  k_steps<<<dim3(n->M * CL, gy), TW * 32, STEP_SMEM>>>(t);
  e = cudaGetLastError();
  if (e) return mfail(n, GH_ERR_CUDA, std::string("MLP kernel: ") + cudaGetErrorString(e));
  return GH_OK;
}

}  // namespace

struct gh_mlp : Net {};

extern "C" {

const char* gh_mlp_last_error(void) { return g_mlp_err.c_str(); }

int gh_mlp_create(int n_members, const int* widths, int n_layers, uint64_t seed, gh_mlp** out) {
  if (!out || !widths || n_members < 1 || n_layers < 1 || n_layers > MAXL) return mfail(nullptr, GH_ERR_ARG, "bad MLP shape");
  for (int l = 0; l <= n_layers; ++l)
    if (widths[l] < 1 || widths[l] > 1024) return mfail(nullptr, GH_ERR_ARG, "layer widths must be 1..1024");
  int dc = 0;
  if (cudaGetDeviceCount(&dc) != cudaSuccess || dc == 0) { cudaGetLastError(); return mfail(nullptr, GH_ERR_CUDA, "no CUDA device"); }
  gh_mlp* n = new gh_mlp();
  n->M = n_members;
  n->nl = n_layers;
  long off = 0;
  for (int l = 0; l <= n_layers; ++l) n->width[l] = widths[l];
  for (int l = 0; l < n_layers; ++l) {
    n->woff[l] = off; off += (long)widths[l + 1] * widths[l];
    n->boff[l] = off; off += widths[l + 1];
  }
  n->P = off;
  const long tot = n->P * n->M;
  // initialisation: W ~ U(-1/sqrt(fan_in), 1/sqrt(fan_in)), b = 0, from the project's counter RNG
  std::vector<float> h(tot, 0.f);
  for (int m = 0; m < n->M; ++m)
    for (int l = 0; l < n_layers; ++l) {
      const float a = 1.f / std::sqrt((float)widths[l]);
      for (long e = 0; e < (long)widths[l + 1] * widths[l]; ++e)
        h[m * n->P + n->woff[l] + e] = a * (float)(2.0 * ghrng::uniform(seed, ghrng::key(0x4D4C50, m, l, e)) - 1.0);
    }
  cudaError_t e = cudaSuccess;
  e = e ? e : cudaMalloc(&n->p, sizeof(float) * tot);
  e = e ? e : cudaMalloc(&n->g, sizeof(float) * tot);
  e = e ? e : cudaMalloc(&n->m1, sizeof(float) * tot);
  e = e ? e : cudaMalloc(&n->m2, sizeof(float) * tot);
  if (!e) e = cudaMemcpy(n->p, h.data(), sizeof(float) * tot, cudaMemcpyHostToDevice);
  if (!e) e = cudaMemset(n->m1, 0, sizeof(float) * tot);
  if (!e) e = cudaMemset(n->m2, 0, sizeof(float) * tot);
  if (e) { cudaGetLastError(); delete n; return mfail(nullptr, GH_ERR_CUDA, std::string("MLP allocation: ") + cudaGetErrorString(e)); }
  if (ensure_cap(n, 256)) { delete n; return GH_ERR_CUDA; }
  *out = n;
  return GH_OK;
}

int gh_mlp_destroy(gh_mlp* n) {
  if (!n) return GH_OK;
  cudaDeviceSynchronize();
  void* ps[] = {n->p, n->g, n->m1, n->m2, n->loss, n->xd, n->yd, n->idx, n->steps, n->out};
  for (void* q : ps) if (q) cudaFree(q);
  for (int l = 0; l < n->nl; ++l) {
    if (n->z[l]) cudaFree(n->z[l]);
    if (n->a[l]) cudaFree(n->a[l]);
    if (n->gz[l]) cudaFree(n->gz[l]);
  }
  delete n;
  return GH_OK;
}

int gh_mlp_num_params(const gh_mlp* n, long* per_member) {
  if (!n || !per_member) return mfail(nullptr, GH_ERR_ARG, "null argument");
  *per_member = n->P;
  return GH_OK;
}

int gh_mlp_get_params(gh_mlp* n, float* params) {
  if (!n || !params) return mfail(nullptr, GH_ERR_ARG, "null argument");
  if (cudaMemcpy(params, n->p, sizeof(float) * n->P * n->M, cudaMemcpyDeviceToHost)) return mfail(n, GH_ERR_CUDA, "copy");
  return GH_OK;
}

int gh_mlp_set_params(gh_mlp* n, const float* params) {
  if (!n || !params) return mfail(nullptr, GH_ERR_ARG, "null argument");
  if (cudaMemcpy(n->p, params, sizeof(float) * n->P * n->M, cudaMemcpyHostToDevice)) return mfail(n, GH_ERR_CUDA, "copy");
  return GH_OK;
}

// forward + loss + backward on one batch; gradients stay on the device (and are
// copied to grads if non-null: [M][P]); loss: [M].
static int grad_batch(gh_mlp* n, const float* xh, const float* yh, int B, float* grads, float* loss) {
  int rc = ensure_cap(n, B);
  if (rc || (rc = upload_samples(n, xh, yh, B))) return rc;
  if ((rc = run_steps(n, GRADIENT, {StepInfo{0, B, 0, 0.f, 0.f}}, nullptr, 1, 0.f))) return rc;
  if (grads && cudaMemcpy(grads, n->g, sizeof(float) * n->P * n->M, cudaMemcpyDeviceToHost)) return mfail(n, GH_ERR_CUDA, "copy");
  if (loss && cudaMemcpy(loss, n->loss, sizeof(float) * n->M, cudaMemcpyDeviceToHost)) return mfail(n, GH_ERR_CUDA, "copy");
  return GH_OK;
}

int gh_mlp_grad(gh_mlp* n, const float* x, const float* y, int B, float* grads, float* loss) {
  if (!n || !x || !y || B < 1) return mfail(n, GH_ERR_ARG, "bad arguments");
  return grad_batch(n, x, y, B, grads, loss);
}

int gh_mlp_adam_step(gh_mlp* n, float lr) {
  if (!n) return mfail(nullptr, GH_ERR_ARG, "null network");
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  n->t += 1;
  const float c1 = 1.f - std::pow(b1, (float)n->t), c2 = 1.f - std::pow(b2, (float)n->t);
  k_adam<<<296, 256>>>(n->p, n->g, n->m1, n->m2, n->P * n->M, lr, b1, b2, eps, c1, c2);
  cudaError_t e = cudaGetLastError();
  if (e) return mfail(n, GH_ERR_CUDA, std::string("adam: ") + cudaGetErrorString(e));
  return GH_OK;
}

// epochs over (x, y) in shuffled minibatches of `batch`; loss: mean loss of the last epoch per member
int gh_mlp_train(gh_mlp* n, const float* x, const float* y, int n_samples, int epochs, int batch, float lr, uint64_t seed,
                 float* loss) {
  if (!n || !x || !y || n_samples < 1 || epochs < 1 || batch < 1) return mfail(n, GH_ERR_ARG, "bad arguments");
  const int maxB = std::min(batch, n_samples);
  int rc = ensure_cap(n, maxB);
  if (rc || (rc = upload_samples(n, x, y, n_samples))) return rc;
  const float b1 = 0.9f, b2 = 0.999f;
  const int nb = (n_samples + batch - 1) / batch;
  // epochs per launch: a bounded table of steps and sample orders
  const int per = std::max(1, std::min(epochs, (int)(std::min<long>(4096 / std::max(nb, 1) + 1, (1L << 20) / n_samples + 1))));
  std::vector<int> idx(n_samples), order;
  std::vector<StepInfo> steps;
  for (int e0 = 0; e0 < epochs; e0 += per) {
    order.clear();
    steps.clear();
    for (int ep = e0; ep < std::min(epochs, e0 + per); ++ep) {
      for (int i = 0; i < n_samples; ++i) idx[i] = i;
      for (int i = n_samples - 1; i > 0; --i) {   // Fisher-Yates with the counter RNG
        const int j = (int)(ghrng::uniform(seed, ghrng::key(0x5348, ep, i)) * (i + 1));
        std::swap(idx[i], idx[std::min(j, i)]);
      }
      const int base = (int)order.size();
      order.insert(order.end(), idx.begin(), idx.end());
      for (int s0 = 0, k = 0; s0 < n_samples; s0 += batch, ++k) {
        n->t += 1;
        steps.push_back(StepInfo{base + s0, std::min(batch, n_samples - s0), ep == epochs - 1 ? k : -1,
                                 1.f - std::pow(b1, (float)n->t), 1.f - std::pow(b2, (float)n->t)});
      }
    }
    if ((rc = run_steps(n, TRAIN, steps, &order, nb, lr))) return rc;
  }
  if (loss) {
    std::vector<float> lb((size_t)nb * n->M);
    if (cudaMemcpy(lb.data(), n->loss, sizeof(float) * lb.size(), cudaMemcpyDeviceToHost)) return mfail(n, GH_ERR_CUDA, "copy");
    for (int m = 0; m < n->M; ++m) {
      float sum = 0.f;
      for (int k = 0; k < nb; ++k) sum += lb[(size_t)k * n->M + m];
      loss[m] = sum / nb;
    }
  }
  if (cudaDeviceSynchronize()) return mfail(n, GH_ERR_CUDA, "train sync");
  return GH_OK;
}

// predictions of every member: out [M][n][n_out] (may be null), and the ensemble
// mean / variance [n][n_out] (population variance over members)
int gh_mlp_predict(gh_mlp* n, const float* x, int B, float* per_member, float* mean, float* var) {
  if (!n || !x || B < 1) return mfail(n, GH_ERR_ARG, "bad arguments");
  int rc = ensure_cap(n, B);
  if (rc) return rc;
  const int nout = n->width[n->nl];
  if ((rc = upload_samples(n, x, nullptr, B)) || (rc = run_steps(n, FORWARD, {StepInfo{0, B, -1, 0.f, 0.f}}, nullptr, 0, 0.f))) return rc;
  std::vector<float> o((size_t)n->M * n->cap * nout);
  if (cudaMemcpy(o.data(), n->out, sizeof(float) * o.size(), cudaMemcpyDeviceToHost)) return mfail(n, GH_ERR_CUDA, "copy");
  for (int b = 0; b < B; ++b)
    for (int k = 0; k < nout; ++k) {
      double s = 0.0, s2 = 0.0;
      for (int m = 0; m < n->M; ++m) {
        const double v = o[((size_t)m * nout + k) * n->cap + b];
        if (per_member) per_member[((size_t)m * B + b) * nout + k] = (float)v;
        s += v;
        s2 += v * v;
      }
      if (mean) mean[(size_t)b * nout + k] = (float)(s / n->M);
      if (var) var[(size_t)b * nout + k] = (float)std::max(0.0, s2 / n->M - (s / n->M) * (s / n->M));
    }
  return GH_OK;
}

}  // extern "C"
