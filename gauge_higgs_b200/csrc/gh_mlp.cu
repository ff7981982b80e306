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
  float* out = nullptr;       // [M][cap][n_out]
  float* gz[MAXL] = {};       // [M][width[l+1]][cap] gradients w.r.t. pre-activations
  float* loss = nullptr;      // [loss_cap][M]
  int loss_cap = 0;
  float *xd = nullptr, *yd = nullptr;   // training set [ns_cap][n_in], [ns_cap][n_out]
  long ns_cap = 0;
  int* idx = nullptr;         // sample order of the steps of one launch
  long idx_cap = 0;
  StepInfo* steps = nullptr;
  long step_cap = 0;
  float *xs = nullptr, *ys = nullptr;   // a step's samples in its order (layer by layer)
  long xs_cap = 0, ys_cap = 0;
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
// separate launches (each thread walking its rows or columns of the weights alone in global
// memory) a step of 5 networks 4-128-128-128-3 at batch 32 takes 267 us; here 43 us.
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

__device__ __forceinline__ float as_float(float v) { return v; }
__device__ __forceinline__ float as_float(__nv_bfloat16 v) { return __bfloat162float(v); }
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

// all threads; orders global and shared memory among the cluster's blocks
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() {
  cluster_arrive();
  cluster_wait();
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
            t.out[(m * cap + first + b) * nout + j] = v;
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
          const float d = t.out[m * cap * nout + e] - t.y[sample(e / nout) * nout + e % nout];
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

// ---------------------------------------------------------------------------
// The same steps with everything a network needs in its cluster's shared memory: each block
// holds its neurons' weight rows, their moments, the columns of the next layer's weights
// that its neurons feed (for the gradient), and the whole batch's activations and
// gradients, which the blocks write into one another's memory (st.shared::cluster).  What
// is left of a step is its cluster barriers and the chains of multiply-adds between them;
// k_steps goes through L2 for every operand and its stores must drain before each barrier
// (2.4 us a layer whatever its size).  Five networks 4-128-128-128-3, batch 32, per step:
// 26 us against 43.  Taken whenever the layout fits 227 KB (hidden width 128: batch
// up to 64).  Bound: instruction issue of the short chains (40% of issue slots) and the waits
// at the barriers between them.  The sums run in the same order as there.
// ---------------------------------------------------------------------------
constexpr int RT = 512;      // threads
constexpr int RES_SMEM = 227 * 1024;   // all that a block may have
struct ResLayout {           // offsets in floats
  int Bp, RS, RH;            // batch rounded up to 32; row strides: floats RS (odd), halves RH (odd words)
  int dup;                   // the output layer is computed by every block
  int per[MAXL];             // neurons per block
  int A0[2], Y[2], ids[2], O;
  int A[MAXL], G[MAXL], Z[MAXL], Wf[MAXL], bf[MAXL], Wb[MAXL], m1[MAXL], m2[MAXL];
  int wfs[MAXL], wbs[MAXL];  // row strides of Wf and Wb
  int total;
};
struct ResArgs { StepArgs s; ResLayout L; };

__device__ __forceinline__ unsigned smem_addr(const void* q) { return (unsigned)__cvta_generic_to_shared(q); }
__device__ __forceinline__ unsigned peer_addr(unsigned local, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// This block's n16 16-byte words at `local` into the same place of every other block of the
// cluster (written by all threads after a __syncthreads).
__device__ __forceinline__ void push(const float* local, int n16, int rank) {
  const unsigned a = smem_addr(local);
  for (int e = threadIdx.x; e < n16 * (CL - 1); e += blockDim.x) {
    const int r = e / n16, v = e - r * n16;
    const float4 q = *reinterpret_cast<const float4*>(local + 4 * v);
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(peer_addr(a, (rank + 1 + r) % CL) + 16 * v), "f"(q.x),
                 "f"(q.y), "f"(q.z), "f"(q.w)
                 : "memory");
  }
}
__device__ __forceinline__ float4 ld_peer4(unsigned a) {
  float4 q;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w) : "r"(a) : "memory");
  return q;
}
__device__ __forceinline__ void copy4(float* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// Columns in pairs (shared memory delivers one operand row per cycle, so a pair's
// multiply-adds share each load of x) and rows in groups of 32, one unit per warp:
// init(c) + sum_k W[c][k] x[k][row], k ascending; epi(c, row, sum).
template <typename T, typename FI, typename FE>
__device__ __forceinline__ void columns(const T* x, int xs, const float* W, int ws, int nk, int nc, int B, FI init, FE epi) {
  const int lane = threadIdx.x & 31, rows = (B + 31) / 32, units = (nc + 1) / 2 * rows;
  for (int u = threadIdx.x >> 5; u < units; u += RT / 32) {
    const int c = u / rows * 2, row = (u - u / rows * rows) * 32 + lane, c2 = min(c + 1, nc - 1);
    const T* px = x + row;
    const float* w0 = W + c * ws;
    const float* w1 = W + c2 * ws;
    float a0 = init(c), a1 = init(c2);
    int k = 0;
    for (; k + 16 <= nk; k += 16) {
      float xv[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) xv[q] = as_float(px[(k + q) * xs]);
#pragma unroll
      for (int q = 0; q < 16; q += 4) {
        const float4 v0 = *reinterpret_cast<const float4*>(w0 + k + q), v1 = *reinterpret_cast<const float4*>(w1 + k + q);
        a0 = fmaf(v0.x, xv[q], a0); a1 = fmaf(v1.x, xv[q], a1);
        a0 = fmaf(v0.y, xv[q + 1], a0); a1 = fmaf(v1.y, xv[q + 1], a1);
        a0 = fmaf(v0.z, xv[q + 2], a0); a1 = fmaf(v1.z, xv[q + 2], a1);
        a0 = fmaf(v0.w, xv[q + 3], a0); a1 = fmaf(v1.w, xv[q + 3], a1);
      }
    }
    for (; k < nk; ++k) {
      const float xk = as_float(px[k * xs]);
      a0 = fmaf(w0[k], xk, a0);
      a1 = fmaf(w1[k], xk, a1);
    }
    if (row < B) {
      epi(c, row, a0);
      if (c2 > c) epi(c2, row, a1);
    }
  }
}
// Weight gradients of neurons in pairs, lanes along the inputs in groups of 64: sum_b G[c][b]
// x[i][b], b ascending; epi(c, i, sum) and, once per neuron, bias(c, sum_b G[c][b]).
template <typename T, typename FE, typename FB>
__device__ __forceinline__ void weight_sums(const T* x, int xs, const float* G, int gs, int B, int nin, int nc, FE epi, FB bias) {
  const int lane = threadIdx.x & 31, blocks = (nin + 63) / 64, units = (nc + 1) / 2 * blocks;
  for (int u = threadIdx.x >> 5; u < units; u += RT / 32) {
    const int c = u / blocks * 2, ib = (u - u / blocks * blocks) * 64, c2 = min(c + 1, nc - 1);
    const int i0 = min(ib + lane, nin - 1), i1 = min(ib + lane + 32, nin - 1);
    const T* x0 = x + i0 * xs;
    const T* x1 = x + i1 * xs;
    const float* g0 = G + c * gs;
    const float* g1 = G + c2 * gs;
    float a00 = 0.f, a01 = 0.f, a10 = 0.f, a11 = 0.f, b0 = 0.f, b1 = 0.f;
    int b = 0;
    for (; b + 8 <= B; b += 8) {
      float p[8], q[8], e[8], f[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) { p[k] = as_float(x0[b + k]); q[k] = as_float(x1[b + k]); e[k] = g0[b + k]; f[k] = g1[b + k]; }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        a00 = fmaf(e[k], p[k], a00); a01 = fmaf(e[k], q[k], a01); b0 = fmaf(e[k], 1.f, b0);
        a10 = fmaf(f[k], p[k], a10); a11 = fmaf(f[k], q[k], a11); b1 = fmaf(f[k], 1.f, b1);
      }
    }
    for (; b < B; ++b) {
      const float p = as_float(x0[b]), q = as_float(x1[b]), e = g0[b], f = g1[b];
      a00 = fmaf(e, p, a00); a01 = fmaf(e, q, a01); b0 = fmaf(e, 1.f, b0);
      a10 = fmaf(f, p, a10); a11 = fmaf(f, q, a11); b1 = fmaf(f, 1.f, b1);
    }
    const bool in0 = ib + lane < nin, in1 = ib + lane + 32 < nin;
    if (in0) epi(c, i0, a00);
    if (in1) epi(c, i1, a01);
    if (c2 > c && in0) epi(c2, i0, a10);
    if (c2 > c && in1) epi(c2, i1, a11);
    if (ib == 0 && lane == 0) {
      bias(c, b0);
      if (c2 > c) bias(c2, b1);
    }
  }
}

// BP: the batch rounded up to 32, 32 or 64 (row strides are then immediate offsets), or 0: any.
template <int BP>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(RT, 1) k_steps_resident(const __grid_constant__ ResArgs ar) {
  extern __shared__ float smem[];
  const StepArgs& t = ar.s;
  const ResLayout& L = ar.L;
  const int rank = blockIdx.x % CL, m = blockIdx.x / CL, nl = t.nl, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = RT / 32;
  const int RS = BP ? BP + 1 : L.RS, RH = BP ? BP + 2 : L.RH;
  const auto nc4 = [](int n) { return (n + 3) / 4 * 4; };
  const int n0 = t.width[0], no = t.width[nl];
  const auto owned = [&](int l, int& c0) {      // this block's neurons of layer l: the first and how many
    if (L.dup && l == nl - 1) { c0 = 0; return t.width[l + 1]; }
    c0 = min(t.width[l + 1], rank * L.per[l]);
    return min(L.per[l], t.width[l + 1] - c0);
  };
  // the weights and moments
  for (int l = 0; l < nl; ++l) {
    int c0;
    const int nc = owned(l, c0), nin = t.width[l];
    const long w = m * t.P + t.woff[l] + (long)c0 * nin, b = m * t.P + t.boff[l] + c0;
    for (int c = warp; c < nc; c += NW)
      for (int i = lane; i < nin; i += 32) {
        smem[L.Wf[l] + c * L.wfs[l] + i] = t.p[w + (long)c * nin + i];
        smem[L.m1[l] + c * (nin + 1) + i] = t.m1[w + (long)c * nin + i];
        smem[L.m2[l] + c * (nin + 1) + i] = t.m2[w + (long)c * nin + i];
      }
    for (int c = tid; c < nc; c += RT) {
      smem[L.bf[l] + c] = t.p[b + c];
      smem[L.m1[l] + c * (nin + 1) + nin] = t.m1[b + c];
      smem[L.m2[l] + c * (nin + 1) + nin] = t.m2[b + c];
    }
  }
  // columns of layer l's weights that this block's neurons of layer l - 1 feed, from the
  // blocks that hold the rows
  const auto pull = [&]() {
    for (int l = 1; l < nl; ++l) {
      int i0;
      const int ni = owned(l - 1, i0), q4 = (ni + 3) / 4, nout = t.width[l + 1];
      if (q4 == 0) continue;
      for (int e = tid; e < nout * q4; e += RT) {
        const int k = e / q4, i = 4 * (e - k * q4), own = L.dup && l == nl - 1 ? rank : k / L.per[l];
        const int row = L.dup && l == nl - 1 ? k : k - own * L.per[l];
        const float4 v = ld_peer4(peer_addr(smem_addr(smem + L.Wf[l] + row * L.wfs[l] + i0 + i), own));
        float* d = smem + L.Wb[l] + i * L.wbs[l] + k;
        d[0] = v.x;
        if (i + 1 < ni) d[L.wbs[l]] = v.y;
        if (i + 2 < ni) d[2 * L.wbs[l]] = v.z;
        if (i + 3 < ni) d[3 * L.wbs[l]] = v.w;
      }
    }
  };
  // a step's samples, in flight while the step before it runs
  const auto info = [&](int st) { return st < t.nsteps ? t.steps[st] : StepInfo{0, 0, -1, 0.f, 0.f}; };
  const auto fetch_ids = [&](int st, const StepInfo& q) {
    int* d = reinterpret_cast<int*>(smem + L.ids[st & 1]);
    for (int b = tid; b < q.B; b += RT) {
      if (t.idx) copy4(reinterpret_cast<float*>(d + b), t.idx + q.s0 + b);
      else d[b] = q.s0 + b;
    }
  };
  const auto fetch_samples = [&](int st, int B) {
    const int* id = reinterpret_cast<const int*>(smem + L.ids[st & 1]);
    for (int b = warp; b < B; b += NW) {
      const long q = id[b];
      for (int k = lane; k < n0; k += 32) copy4(smem + L.A0[st & 1] + k * RS + b, t.x + q * n0 + k);
      for (int k = lane; k < no; k += 32) copy4(smem + L.Y[st & 1] + k * RS + b, t.y + q * no + k);
    }
  };
  const auto landed = [&]() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  };
  StepInfo si = info(0), s1 = info(1), s2 = info(2);   // read ahead of their use
  fetch_ids(0, si);
  landed();
  fetch_samples(0, si.B);
  fetch_ids(1, s1);
  landed();
  cluster_barrier();                            // every block of the cluster runs: its memory may be written
  for (int st = 0; st < t.nsteps; ++st) {
    const StepInfo s3 = info(st + 3);
    const int B = si.B;
    const float* A0 = smem + L.A0[st & 1];
    const float* Y = smem + L.Y[st & 1];
    fetch_samples(st + 1, s1.B);
    fetch_ids(st + 2, s2);
    pull();                                     // before the first barrier of the step: Adam comes after it
    for (int l = 0; l < nl; ++l) {
      int c0;
      const int nc = owned(l, c0), nin = t.width[l];
      const bool last = l == nl - 1;
      const auto I = [&](int c) { return smem[L.bf[l] + c]; };
      const auto E = [&](int c, int b, float v) {
        const int o = (c0 + c) * RS + b;
        if (!last) {
          smem[L.Z[l] + c * RS + b] = v;
          reinterpret_cast<__nv_bfloat16*>(smem + L.A[l + 1])[(c0 + c) * RH + b] = __float2bfloat16(silu(v));
        } else {
          const float d = v - Y[o];
          smem[L.G[l] + o] = 2.f * d / (float)(B * no);
          smem[L.O + o] = v;
        }
      };
      if (l) columns(reinterpret_cast<const __nv_bfloat16*>(smem + L.A[l]), RH, smem + L.Wf[l], L.wfs[l], nin, nc, B, I, E);
      else columns(A0, RS, smem + L.Wf[l], L.wfs[l], nin, nc, B, I, E);
      __syncthreads();
      if (last && L.dup) break;
      if (!last) {
        push(smem + L.A[l + 1] + c0 * RH / 2, nc4(nc) * RH / 8, rank);
      } else {
        push(smem + L.G[l] + c0 * RS, nc4(nc) * RS / 4, rank);
        push(smem + L.O + c0 * RS, nc4(nc) * RS / 4, rank);
      }
      cluster_barrier();
    }
    for (int l = nl - 1; l > 0; --l) {          // gradient through layer l and the SiLU before it
      int i0;
      const int ni = owned(l - 1, i0);
      columns(smem + L.G[l], RS, smem + L.Wb[l], L.wbs[l], t.width[l + 1], ni, B, [](int) { return 0.f; },
              [&](int i, int b, float v) {
        smem[L.G[l - 1] + ((l == 1 ? 0 : i0) + i) * RS + b] = v * dsilu(smem[L.Z[l - 1] + i * RS + b]);
      });
      __syncthreads();
      if (l == 1) break;                        // only this block's weight gradients read G[0]
      push(smem + L.G[l - 1] + i0 * RS, nc4(ni) * RS / 4, rank);
      cluster_barrier();
    }
    if (si.slot >= 0 && rank == 0 && warp < 8) {  // loss: mean of (out - y)^2, 256 strided sums and a tree
      float* sh = smem + L.O + (no + 3) / 4 * 4 * RS;
      float sum = 0.f;
      for (int e = tid; e < B * no; e += 256) {
        const float d = smem[L.O + (e % no) * RS + e / no] - Y[(e % no) * RS + e / no];
        sum += d * d;
      }
      sh[tid] = sum;
      for (int q = 128; q > 0; q >>= 1) {
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (tid < q) sh[tid] += sh[tid + q];
      }
      if (tid == 0) t.loss[(long)si.slot * t.M + m] = sh[0] / (float)(B * no);
    }
    const bool keep = st == t.nsteps - 1;       // the gradients of the last step stay for gh_mlp_adam_step
    for (int l = 0; l < nl; ++l) {
      int c0;
      const int nc = owned(l, c0), nin = t.width[l];
      const bool out = keep && (rank == 0 || !(L.dup && l == nl - 1));
      const auto E = [&](int c, int i, float v) {
        if (out) t.g[m * t.P + t.woff[l] + (long)(c0 + c) * nin + i] = v;
        if (t.mode == TRAIN)
          adam_update(smem + L.Wf[l] + c * L.wfs[l] + i, smem + L.m1[l] + c * (nin + 1) + i, smem + L.m2[l] + c * (nin + 1) + i, v,
                      t.lr, t.b1, t.b2, t.eps, si.c1, si.c2);
      };
      const auto EB = [&](int c, float v) {
        if (out) t.g[m * t.P + t.boff[l] + c0 + c] = v;
        if (t.mode == TRAIN)
          adam_update(smem + L.bf[l] + c, smem + L.m1[l] + c * (nin + 1) + nin, smem + L.m2[l] + c * (nin + 1) + nin, v, t.lr, t.b1,
                      t.b2, t.eps, si.c1, si.c2);
      };
      // G[0] below other layers holds this block's rows only
      const float* g = smem + L.G[l] + (l || nl == 1 ? c0 : 0) * RS;
      if (l) weight_sums(reinterpret_cast<const __nv_bfloat16*>(smem + L.A[l]), RH, g, RS, B, nin, nc, E, EB);
      else weight_sums(A0, RS, g, RS, B, nin, nc, E, EB);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_barrier();                          // new weights and the next step's samples are in place
    si = s1;
    s1 = s2;
    s2 = s3;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (t.mode == TRAIN)
    for (int l = 0; l < nl; ++l) {
      int c0;
      const int nc = owned(l, c0), nin = t.width[l];
      if (L.dup && l == nl - 1 && rank != 0) break;
      const long w = m * t.P + t.woff[l] + (long)c0 * nin, b = m * t.P + t.boff[l] + c0;
      for (int c = warp; c < nc; c += NW)
        for (int i = lane; i < nin; i += 32) {
          t.p[w + (long)c * nin + i] = smem[L.Wf[l] + c * L.wfs[l] + i];
          t.m1[w + (long)c * nin + i] = smem[L.m1[l] + c * (nin + 1) + i];
          t.m2[w + (long)c * nin + i] = smem[L.m2[l] + c * (nin + 1) + i];
        }
      for (int c = tid; c < nc; c += RT) {
        t.p[b + c] = smem[L.bf[l] + c];
        t.m1[b + c] = smem[L.m1[l] + c * (nin + 1) + nin];
        t.m2[b + c] = smem[L.m2[l] + c * (nin + 1) + nin];
      }
    }
}

// The layout for batches of up to maxB samples; false if it does not fit a block.
bool res_layout(const Net& n, int maxB, ResLayout& L) {
  std::memset(&L, 0, sizeof(L));
  long at = 0;
  const auto take = [&](long f) {               // rows that are read as float4 start on 16 bytes
    const long o = at;
    at += (f + 3) / 4 * 4;
    return (int)std::min<long>(o, 1 << 28);
  };
  const auto up4 = [](int x) { return (x + 3) / 4 * 4; };
  L.Bp = (maxB + 31) / 32 * 32;
  L.RS = L.Bp + 1;
  L.RH = L.Bp + 2;
  const int nl = n.nl, no = n.width[nl];
  L.dup = no <= 16;
  for (int k = 0; k < 2; ++k) { L.A0[k] = take((long)n.width[0] * L.RS); L.Y[k] = take((long)no * L.RS); L.ids[k] = take(L.Bp); }
  L.O = take((long)up4(no) * L.RS + 256);
  for (int l = 0; l < nl; ++l) {
    const int nin = n.width[l], nout = n.width[l + 1];
    const bool dup = L.dup && l == nl - 1;
    L.per[l] = dup ? nout : up4((nout + CL - 1) / CL);   // fours: slices of A, G and W rows start on 16 bytes
    const long nc = L.per[l];
    if (l) L.A[l] = take((long)up4(nin) * L.RH / 2);
    L.G[l] = take((long)(l || nl == 1 ? up4(nout) : nc) * L.RS);
    if (l + 1 < nl) L.Z[l] = take(nc * L.RS);
    L.wfs[l] = up4(nin) + 4;
    L.Wf[l] = take(nc * L.wfs[l]);
    L.bf[l] = take(nc);
    if (l) { L.wbs[l] = up4(nout) + 4; L.Wb[l] = take((long)L.per[l - 1] * L.wbs[l]); }
    L.m1[l] = take(nc * (nin + 1));
    L.m2[l] = take(nc * (nin + 1));
  }
  L.total = (int)std::min<long>(at, 1 << 28);
  return at * sizeof(float) <= RES_SMEM;
}

__global__ void k_adam(float* p, const float* g, float* m1, float* m2, long n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x)
    adam_update(p + e, m1 + e, m2 + e, g[e], lr, b1, b2, eps, c1, c2);
}

// ---------------------------------------------------------------------------
// The same arithmetic with one launch per layer and product, over the whole GPU, for the calls
// whose work fills it: a cluster has 8 of its 148 SMs.  Which form a call takes: cluster_us and
// layers_us.  Activations and gradients lie [sample][neuron] here.  Sums in the order of k_steps.
// Bound: one thread's chain of multiply-adds in small calls (a neuron's weights, or the batch),
// the shared and L1 loads beside each multiply-add in large ones.
// ---------------------------------------------------------------------------
constexpr int BT = 16;       // samples per block (forward and input gradient)
struct LayerArgs {
  int B, nin, nout;
  long cap, P;                 // samples per network in the buffers; parameters per network
  const float *w, *bias;       // network 0's
  const float* x;              // layer 0: the step's samples, else null
  const __nv_bfloat16* in;     // other layers: activations
};

// a step's samples and targets in its order
__global__ void k_gather(const float* x, const float* y, const int* idx, int B, int nin, int nout, float* xs, float* ys) {
  const int row = nin + nout;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)B * row; e += (long)gridDim.x * blockDim.x) {
    const int b = (int)(e / row), k = (int)(e - (long)b * row);
    if (k < nin) xs[(long)b * nin + k] = x[(long)idx[b] * nin + k];
    else ys[(long)b * nout + k - nin] = y[(long)idx[b] * nout + k - nin];
  }
}

// z = b + W a, and the next layer's activations (a null: none); a thread per neuron
__global__ void __launch_bounds__(1024) k_dense_fwd(const LayerArgs t, float* z, __nv_bfloat16* a) {
  extern __shared__ float s_in[];   // [BT][nin]
  const int tiles = (t.B + BT - 1) / BT, m = blockIdx.x / tiles, b0 = (blockIdx.x - m * tiles) * BT, j = threadIdx.x;
  const int nin = t.nin, rows = min(BT, t.B - b0);
  const __nv_bfloat16* in = t.in + (m * t.cap + b0) * nin;
  for (int e = threadIdx.x; e < BT * nin; e += blockDim.x)
    s_in[e] = e >= rows * nin ? 0.f : t.x ? t.x[(long)b0 * nin + e] : __bfloat162float(in[e]);
  __syncthreads();
  if (j >= t.nout) return;
  const float* w = t.w + m * t.P + (long)j * nin;
  float acc[BT];
#pragma unroll
  for (int bb = 0; bb < BT; ++bb) acc[bb] = t.bias[m * t.P + j];
  for (int i = 0; i < nin; ++i) {
    const float wi = w[i];
#pragma unroll
    for (int bb = 0; bb < BT; ++bb) acc[bb] = fmaf(wi, s_in[bb * nin + i], acc[bb]);
  }
#pragma unroll
  for (int bb = 0; bb < BT; ++bb) {
    if (bb >= rows) break;
    const long o = (m * t.cap + b0 + bb) * t.nout + j;
    z[o] = acc[bb];
    if (a) a[o] = __float2bfloat16(silu(acc[bb]));
  }
}

// output gradient 2 (out - y) / (B n_out), and the loss where its slot is not null
__global__ void __launch_bounds__(256) k_mse(const LayerArgs t, const float* out, const float* y, float* gz, float* loss) {
  const int m = blockIdx.x, n = t.B * t.nout;
  out += m * t.cap * t.nout;
  gz += m * t.cap * t.nout;
  float s = 0.f;
  for (int e = threadIdx.x; e < n; e += 256) {
    const float d = out[e] - y[e];
    s += d * d;
    gz[e] = 2.f * d / (float)n;
  }
  __shared__ float sh[256];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0 && loss) loss[m] = sh[0] / (float)n;
}

// dW[j][i] = sum_b gz[b][j] in[b][i], db[j] = sum_b gz[b][j]; a block per neuron, threads over i
template <bool FIRST>
__global__ void __launch_bounds__(128) k_dense_wgrad(const LayerArgs t, const float* gz, float* g, long woff, long boff) {
  const int m = blockIdx.x, j = blockIdx.y, nin = t.nin, nout = t.nout, B = t.B;
  gz += m * t.cap * nout + j;
  g += m * t.P;
  for (int i = threadIdx.x; i <= nin; i += blockDim.x) {
    const int ic = min(i, nin - 1);
    const float* x = t.x + ic;
    const __nv_bfloat16* in = t.in + m * t.cap * nin + ic;
    float s = 0.f;
    for (int b = 0; b < B; ++b) {              // the bias's thread walks along with its warp
      const float v = FIRST ? x[(long)b * nin] : __bfloat162float(in[(long)b * nin]);
      s = fmaf(gz[(long)b * nout], i == nin ? 1.f : v, s);
    }
    g[i == nin ? boff + j : woff + (long)j * nin + i] = s;
  }
}

// gradient through the layer and the SiLU before it; a thread per input
__global__ void __launch_bounds__(1024) k_dense_bgrad(const LayerArgs t, const float* gz, const float* zprev, float* gprev) {
  const int tiles = (t.B + BT - 1) / BT, m = blockIdx.x / tiles, b0 = (blockIdx.x - m * tiles) * BT, i = threadIdx.x;
  const int nin = t.nin, nout = t.nout;
  if (i >= nin) return;
  const float* w = t.w + m * t.P + i;
  for (int b = b0; b < min(t.B, b0 + BT); ++b) {
    const float* gb = gz + (m * t.cap + b) * nout;
    float s = 0.f;
    for (int j = 0; j < nout; ++j) s = fmaf(w[(long)j * nin], gb[j], s);
    const long o = (m * t.cap + b) * nin + i;
    gprev[o] = s * dsilu(zprev[o]);
  }
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

// Which form a call takes: the two are bit for bit the same, and which is faster turns on every
// size, so both times are estimated (us per step or pass) from what each form does.
//   Clusters: networks (forward: 64-sample pieces of them) in waves of 14, and in each product of
//   a wave its passes over a block's columns, and the multiply-adds of a lane.
//   Layers: per product the longer of one thread's chain and the multiply-adds of all networks at
//   the rate that the kernel reaches with the GPU full.
// The constants are fitted (rms 9 to 20%) to trainings and predictions of 2025 combinations: 1 to
// 5 hidden layers of 16 to 512, 1 to 48 networks, batches of 32 to 8192.  A step in us, layers /
// clusters: 5 networks 4-128-128-128-3, batch 32 267 / 41 (resident), 2048 1310 / 1140; one
// 4-256-256-256-3, batch 512 950 / 960, 2048 1830 / 3700; 48 of 4-16-16-16-3, batch 64 124 / 95,
// 2048 670 / 1440.
struct ClusterCost { double call, product, pass, term; };
constexpr ClusterCost STEPS_COST{16.2, 1.15, 0.955, 4.45e-4}, RESIDENT_COST{13.8, 0.98, 0.648, 2.43e-4},
    FORWARD_COST{44.9, 0.81, 0.383, 4.68e-4};
constexpr int CLUSTERS_AT_ONCE = 14;   // clusters of 8 SMs that find room in the GPU's parts
double cluster_us(const Net& n, int mode, int B, const ClusterCost& c) {
  const auto up = [](long a, long b) { return (double)((a + b - 1) / b); };
  const auto product = [&](int rows, int cols, int terms) {
    return c.product + up(cols, TW) * (up(rows, RG) * up(terms, KC) * c.pass + up(rows, 32) * 32 * terms * c.term);
  };
  const int rows = mode == FORWARD ? std::min(B, 64) : B;
  double t = 0;
  for (int l = 0; l < n.nl; ++l) {
    const int nin = n.width[l], nout = n.width[l + 1], ci = (nin + CL - 1) / CL, co = (nout + CL - 1) / CL;
    t += product(rows, co, nin);
    if (mode != FORWARD) t += product(nin, co, B) + (l ? product(B, ci, nout) : 0.0);
  }
  return c.call + t * up(mode == FORWARD ? (long)n.M * ((B + 63) / 64) : n.M, CLUSTERS_AT_ONCE);
}
double layers_us(const Net& n, int mode, int B) {
  double t = mode == FORWARD ? 23.6 : 47.5;
  for (int l = 0; l < n.nl; ++l) {
    const double nin = n.width[l], nout = n.width[l + 1], fma = (double)n.M * B * nin * nout;
    if (mode == FORWARD) { t += 6.8 + std::max(0.149 * nin, 3.38e-7 * fma); continue; }
    t += std::max(0.073 * nin, 9.0e-7 * fma) + std::max(0.06 * B * std::ceil((nin + 1) / 128), 2.73e-7 * fma);
    if (l) t += std::max(0.99 * nout, 2.47e-7 * fma);
  }
  return t;
}

// One step (or forward pass) layer by layer.
cudaError_t run_layers(const StepArgs& t, const StepInfo& si, float* xs, float* ys) {
  LayerArgs q{};
  const float *x = t.x, *y = t.y;
  if (t.idx) {
    const int n0 = t.width[0], no = t.width[t.nl];
    k_gather<<<std::min(((long)si.B * (n0 + no) + 255) / 256, 1024L), 256>>>(x, y, t.idx + si.s0, si.B, n0, no, xs, ys);
    x = xs;
    y = ys;
  }
  q.B = si.B; q.cap = t.cap; q.P = t.P;
  const auto layer = [&](int l) {
    q.nin = t.width[l]; q.nout = t.width[l + 1];
    q.w = t.p + t.woff[l]; q.bias = t.p + t.boff[l];
    q.x = l ? nullptr : x;
    q.in = l ? t.a[l - 1] : nullptr;
  };
  const unsigned tiles = (unsigned)t.M * ((si.B + BT - 1) / BT);
  const auto threads = [](int n) { return (n + 31) / 32 * 32; };
  const int nl = t.nl;
  cudaError_t e = cudaFuncSetAttribute(k_dense_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, BT * 1024 * (int)sizeof(float));
  if (e) return e;
  for (int l = 0; l < nl; ++l) {
    layer(l);
    k_dense_fwd<<<tiles, threads(std::max(q.nin, q.nout)), sizeof(float) * BT * q.nin>>>(q, l == nl - 1 ? t.out : t.z[l], l == nl - 1 ? nullptr : t.a[l]);
  }
  if (t.mode != FORWARD) {
    k_mse<<<t.M, 256>>>(q, t.out, y, t.gz[nl - 1], si.slot >= 0 ? t.loss + (long)si.slot * t.M : nullptr);
    for (int l = nl - 1; l >= 0; --l) {
      layer(l);
      const dim3 grid(t.M, q.nout);
      if (l) k_dense_wgrad<false><<<grid, 128>>>(q, t.gz[l], t.g, t.woff[l], t.boff[l]);
      else k_dense_wgrad<true><<<grid, 128>>>(q, t.gz[l], t.g, t.woff[l], t.boff[l]);
      if (l) k_dense_bgrad<<<tiles, threads(q.nin)>>>(q, t.gz[l], t.z[l - 1], t.gz[l - 1]);
    }
    if (t.mode == TRAIN) k_adam<<<296, 256>>>(t.p, t.g, t.m1, t.m2, t.P * t.M, t.lr, t.b1, t.b2, t.eps, si.c1, si.c2);
  }
  return cudaGetLastError();
}

// Runs `steps` (one for FORWARD and GRADIENT) over the uploaded samples; order: sample
// index of every row of the steps, null for the order they lie in.
int run_steps(Net* n, int mode, const std::vector<StepInfo>& steps, const std::vector<int>* order, int slots, float lr) {
  int maxB = 0;
  for (const StepInfo& q : steps) maxB = std::max(maxB, q.B);
  ResArgs ra;
  const bool resident = mode != FORWARD && res_layout(*n, maxB, ra.L);
  // clusters only where their estimate is clearly the lower
  const bool layers = layers_us(*n, mode, maxB) < 1.1 * cluster_us(*n, mode, maxB, mode == FORWARD ? FORWARD_COST : resident ? RESIDENT_COST : STEPS_COST);
  long lc = (long)n->loss_cap * n->M;
  cudaError_t e = cudaSuccess;
  if (order) e = grow(&n->idx, &n->idx_cap, (long)order->size());
  if (!e && slots) e = grow(&n->loss, &lc, (long)slots * n->M);
  n->loss_cap = (int)(lc / n->M);
  if (!e && order) e = cudaMemcpy(n->idx, order->data(), sizeof(int) * order->size(), cudaMemcpyHostToDevice);
  if (!e && layers && order) e = grow(&n->xs, &n->xs_cap, (long)maxB * n->width[0]);
  if (!e && layers && order) e = grow(&n->ys, &n->ys_cap, (long)maxB * n->width[n->nl]);
  if (!e && !layers) e = grow(&n->steps, &n->step_cap, (long)steps.size());
  if (!e && !layers) e = cudaMemcpy(n->steps, steps.data(), sizeof(StepInfo) * steps.size(), cudaMemcpyHostToDevice);
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
  if (layers) {
    for (size_t k = 0; k < steps.size() && !e; ++k) e = run_layers(t, steps[k], n->xs, n->ys);
  } else if (resident) {
    void (*const k)(ResArgs) = ra.L.Bp == 32 ? k_steps_resident<32> : ra.L.Bp == 64 ? k_steps_resident<64> : k_steps_resident<0>;
    // the limit belongs to the kernel: the same one from every network, or a call of a narrower
    // network in another thread could lower it between this and the launch
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM);
    ra.s = t;
    if (!e) k<<<n->M * CL, RT, ra.L.total * sizeof(float)>>>(ra);
  } else {
    t.rows = 64;                                // forward rows are independent: clusters of 64 samples
    const int gy = mode == FORWARD ? (steps[0].B + t.rows - 1) / t.rows : 1;
    e = cudaFuncSetAttribute(k_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STEP_SMEM);
    if (!e) k_steps<<<dim3(n->M * CL, gy), TW * 32, STEP_SMEM>>>(t);
  }
  e = e ? e : cudaGetLastError();
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
  void* ps[] = {n->p, n->g, n->m1, n->m2, n->loss, n->xd, n->yd, n->idx, n->steps, n->xs, n->ys, n->out};
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
        const double v = o[((size_t)m * n->cap + b) * nout + k];
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
