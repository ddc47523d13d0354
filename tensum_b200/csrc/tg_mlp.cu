// tg_mlp.cu -- the surrogate network of the multi-fidelity Monte Carlo estimator.
//
// A fixed-shape multilayer perceptron din -> 64 -> 64 -> 64 -> dout with GELU
// (0.5 x (1 + erf(x / sqrt 2))) after each hidden layer, trained in FP32 by
// full forward / backward passes written here (mean squared error, Adam), and
// evaluated in BF16 on the tensor cores for the large surrogate sample sets.
// The network only ever serves as a control variate; it has no counterpart in
// the reference.
//
// Parameters are one FP32 vector: W1[64][din] b1[64] W2[64][64] b2[64]
// W3[64][64] b3[64] W4[dout][64] b4[dout] (W[out][in], row major).
// Every reduction over the batch runs in a fixed order (each weight's thread sums
// its samples in sequence), so training is bitwise reproducible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "../../include/tensum_gpu.h"

namespace {

constexpr int H = 64;
constexpr int kMaxIn = 32;
constexpr int kMaxOut = 8;
thread_local std::string g_mlp_error;

struct Offs {
  int w1, b1, w2, b2, w3, b3, w4, b4, n;
};

__host__ __device__ inline Offs offsets(int din, int dout) {
  Offs o;
  o.w1 = 0; o.b1 = o.w1 + H * din;
  o.w2 = o.b1 + H; o.b2 = o.w2 + H * H;
  o.w3 = o.b2 + H; o.b3 = o.w3 + H * H;
  o.w4 = o.b3 + H; o.b4 = o.w4 + dout * H;
  o.n = o.b4 + dout;
  return o;
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
  // d/dx [x Phi(x)] = Phi(x) + x phi(x)
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.3989422804014327f * expf(-0.5f * x * x);
}

__device__ __forceinline__ void adam(float gp, float& th, float& m, float& v, float lr, float b1, float b2, float eps,
                                     float c1, float c2) {   // Kingma & Ba (2015) with bias correction
  const float mp = b1 * m + (1.0f - b1) * gp;
  const float vp = b2 * v + (1.0f - b2) * gp * gp;
  m = mp;
  v = vp;
  th -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

// ------------------------------------------------------------------- training
// Minibatch after minibatch in one launch of one cluster of 8 CTAs: a step is 0.3 MFLOP per
// 64 samples, so launches (five kernels and two copies a step before) and their single
// threads' chains of 64 x 64 multiply-adds were all of its 347 us.  Each CTA holds the
// weights in shared memory.  Per minibatch, (A) every CTA runs forward and backward for 8
// samples of each 64 (one thread per neuron and 2 samples) and stores activations and deltas in L2; (B) it owns 8 rows of each weight
// matrix, sums their gradients over the batch and applies Adam, whose moments stay in
// registers for the whole launch; the new weights go through L2 to every CTA.  Two cluster
// barriers a minibatch.  Every sum keeps the order of one thread adding its terms in
// sequence (neurons over inputs, gradients over samples), so results do not depend on the
// cluster: 256 samples, batch 64, 800 minibatches in 282 ms before and 7.9 ms now,
// the same weights bit for bit.  What is left of a minibatch's 9.8 us is latency: L2 round
// trips of weights, activations and deltas, the barriers, and chains of 64 multiply-adds.
// Large batches stay on the 8 SMs too: thread-per-sample kernels over the whole chip were slower
// at every size.  One loss and gradient of n samples in us, those / the cluster: 3 inputs and 3
// outputs, n = 64, 1000, 4096, 65536: 377 / 56, 795 / 165, 1595 / 515, 21898 / 6889; 32 and 8:
// 405 / 69, 845 / 263, 1626 / 855, 23781 / 13093.
constexpr int kCl = 8, kTrainThreads = 256, kTile = 64;
constexpr int kSmall = (8 * kMaxIn + 24 + 9 * kMaxOut + 2 * H - 1) / (2 * H);   // small gradients per thread
// Weight rows padded so that lanes over rows read 16-byte words, and lanes over columns
// 4-byte ones, without bank conflicts.
constexpr int kWP = H + 4, kXP = kMaxIn + 1;

struct Train {
  const float *X, *T;              // all samples
  int n, din, dout, batch, per_epoch;
  long first;                      // first minibatch of this launch, counted from the first epoch
  int count;
  float *theta, *m, *v, *g;
  float *A, *D, *D4, *Y;           // activations and deltas [sample][3][H], outputs of one minibatch
  float* losses;                   // per epoch (the last minibatch's), null: none
  const float2* corr;              // Adam's bias corrections per minibatch of this launch
  float lr;
  int update;                      // 0: the gradient goes to g and the weights stay
};

struct TrainSmem {
  alignas(16) float w2[H * kWP], w3[H * kWP], w1[H * kMaxIn], w4[kMaxOut * H], bias[3 * H + kMaxOut];
  float x[8][kMaxIn], t[8][kMaxOut];
  float gd[3][8][H];                        // gelu'(z)
  alignas(16) float a[2][8][H];
  alignas(16) float d[2][8][H];
  alignas(16) float d4[8][kMaxOut];
  alignas(16) float tA[2][kTile][H];        // (B) activations of layers 1, 2
  alignas(16) float tD[3][kTile][8];        // deltas of the CTA's 8 rows
  alignas(16) float tA3[kTile][8];          // layer-3 activations of its 8 columns of W4
  alignas(16) float tD4[kTile][kMaxOut];
  float tX[kTile][kMaxIn];
  float red[kTrainThreads];
};

__device__ __forceinline__ void cp16(void* smem, const void* gmem) {   // through L2, past L1
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp4(void* smem, const void* gmem) {    // read-only data
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kTrainThreads, 1) k_train(Train t) {
  extern __shared__ __align__(16) unsigned char raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(raw);
  const Offs o = offsets(t.din, t.dout);
  const int tid = threadIdx.x, rank = blockIdx.x, din = t.din, dout = t.dout;
  // gradients this thread owns: threads 0 .. 127 the CTA's 8 rows of one column gi of W2
  // (gl = 0) or W3 (1), the others up to kSmall of its small ones
  const int gi = tid & (H - 1), gl = (tid >> 6) & 1;
  const bool main = tid < 2 * H;
  const int n_w1 = 8 * din, n_w4 = 8 * dout, n_small = n_w1 + 24 + n_w4 + (rank == 0 ? dout : 0);
  int pp[8];
  float th[8], m[8], v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    pp[r] = -1;
    if (main) {
      pp[r] = (gl ? o.w3 : o.w2) + (8 * rank + r) * H + gi;
    } else if (r < kSmall) {
      int p = tid - 2 * H + r * 2 * H;
      if (p < n_w1) pp[r] = o.w1 + (8 * rank + p / din) * din + p % din;
      else if ((p -= n_w1) < 24) pp[r] = (p < 8 ? o.b1 : p < 16 ? o.b2 : o.b3) + 8 * rank + (p & 7);
      else if ((p -= 24) < n_w4) pp[r] = o.w4 + (p / 8) * H + 8 * rank + (p & 7);
      else if ((p -= n_w4) < dout && rank == 0) pp[r] = o.b4 + p;
    }
    th[r] = pp[r] >= 0 ? t.theta[pp[r]] : 0.0f;
    m[r] = pp[r] >= 0 && t.update ? t.m[pp[r]] : 0.0f;
    v[r] = pp[r] >= 0 && t.update ? t.v[pp[r]] : 0.0f;
  }
  for (int it = 0; it < t.count; ++it) {
    // the weights as every CTA left them and the first samples, all loads in flight at once
    const long mb = t.first + it;
    const int s0 = (int)(mb % t.per_epoch) * t.batch, nb = min(t.batch, t.n - s0);
    const float scale = 2.0f / ((float)nb * (float)dout);
    auto samples = [&](int base) {
      const int b = base + (tid >> 5), c = tid & 31;
      if (b < nb) {     // rows past the batch compute on what is there; nothing of theirs is kept
        if (c < din) cp4(&S.x[tid >> 5][c], t.X + (size_t)(s0 + b) * din + c);
        if (c < dout) cp4(&S.t[tid >> 5][c], t.T + (size_t)(s0 + b) * dout + c);
      }
    };
    for (int i = tid; i < H * H / 4; i += kTrainThreads) {
      const int w = (i >> 4) * kWP + 4 * (i & 15);
      cp16(S.w2 + w, t.theta + o.w2 + 4 * i);
      cp16(S.w3 + w, t.theta + o.w3 + 4 * i);
    }
    for (int i = tid; i < dout * (H / 4); i += kTrainThreads) cp16(S.w4 + 4 * i, t.theta + o.w4 + 4 * i);
    if (tid < 3 * (H / 4)) {
      const int l = tid / (H / 4), c = 4 * (tid % (H / 4));
      cp16(S.bias + l * H + c, t.theta + (l == 0 ? o.b1 : l == 1 ? o.b2 : o.b3) + c);
    }
    const float2 corr = t.update ? t.corr[it] : make_float2(1.0f, 1.0f);
    for (int i = tid; i < din * (H / 4); i += kTrainThreads) cp16(S.w1 + 4 * i, t.theta + o.w1 + 4 * i);
    if (tid < kMaxOut / 4) cp16(S.bias + 3 * H + 4 * tid, t.theta + o.b4 + 4 * tid);   // theta is padded
    samples(8 * rank);
    cp_wait();

    // ---- (A) forward and backward of this CTA's samples
    const int j = tid & (H - 1), g2 = 2 * (tid >> 6);      // neuron, first of 2 samples
    for (int base = 8 * rank; base < nb; base += 8 * kCl) {
      if (base >= 8 * kCl) {     // the last readers of x and t are a barrier behind
        samples(base);
        cp_wait();
      }
      __syncthreads();
      float acc[2];
      auto put = [&](int l) {     // activations of layer l to a[l & 1] and L2, gelu' for the way back
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float a = gelu(acc[q]);
          S.gd[l][g2 + q][j] = gelu_d(acc[q]);
          S.a[l & 1][g2 + q][j] = a;
          if (base + g2 + q < nb) __stcg(t.A + ((size_t)(base + g2 + q) * 3 + l) * H + j, a);
        }
      };
      acc[0] = acc[1] = S.bias[j];
      for (int i = 0; i < din; ++i) {
        const float w = S.w1[j * din + i];
        acc[0] = fmaf(w, S.x[g2][i], acc[0]);
        acc[1] = fmaf(w, S.x[g2 + 1][i], acc[1]);
      }
      put(0);
      __syncthreads();
      for (int l = 1; l < 3; ++l) {
        const float* w = (l == 1 ? S.w2 : S.w3) + j * kWP;
        const float(*in)[H] = S.a[(l - 1) & 1];
        acc[0] = acc[1] = S.bias[l * H + j];
#pragma unroll 8
        for (int i = 0; i < H; i += 4) {
          const float4 y = *reinterpret_cast<const float4*>(w + i);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float4 x = *reinterpret_cast<const float4*>(&in[g2 + q][i]);
            acc[q] = fmaf(y.w, x.w, fmaf(y.z, x.z, fmaf(y.y, x.y, fmaf(y.x, x.x, acc[q]))));
          }
        }
        put(l);
        __syncthreads();
      }
      if (tid < 8 * kMaxOut) {    // one thread per sample and output
        const int ls = tid / kMaxOut, k = tid % kMaxOut, b = base + ls;
        float d = 0.0f;
        if (k < dout) {
          float s = S.bias[3 * H + k];
#pragma unroll 8
          for (int i = 0; i < H; i += 4) {
            const float4 y = *reinterpret_cast<const float4*>(S.w4 + k * H + i);
            const float4 x = *reinterpret_cast<const float4*>(&S.a[0][ls][i]);
            s = fmaf(y.w, x.w, fmaf(y.z, x.z, fmaf(y.y, x.y, fmaf(y.x, x.x, s))));
          }
          if (b < nb) {
            d = (s - S.t[ls][k]) * scale;
            __stcg(t.Y + (size_t)b * dout + k, s);
          }
        }
        S.d4[ls][k] = d;
        if (b < nb) __stcg(t.D4 + (size_t)b * kMaxOut + k, d);
      }
      __syncthreads();
      for (int l = 2; l >= 0; --l) {     // deltas of layer l to d[l & 1] and L2
        acc[0] = acc[1] = 0.0f;
        if (l == 2) {
          for (int k = 0; k < dout; ++k) {
            const float w = S.w4[k * H + j];
            acc[0] = fmaf(w, S.d4[g2][k], acc[0]);
            acc[1] = fmaf(w, S.d4[g2 + 1][k], acc[1]);
          }
        } else {
          const float* w = (l == 1 ? S.w3 : S.w2) + j;
          const float(*in)[H] = S.d[(l + 1) & 1];
#pragma unroll 8
          for (int i = 0; i < H; i += 4) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const float4 x = *reinterpret_cast<const float4*>(&in[g2 + q][i]);
              acc[q] = fmaf(w[(i + 3) * kWP], x.w,
                            fmaf(w[(i + 2) * kWP], x.z, fmaf(w[(i + 1) * kWP], x.y, fmaf(w[i * kWP], x.x, acc[q]))));
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float d = acc[q] * S.gd[l][g2 + q][j];
          S.d[l & 1][g2 + q][j] = d;
          if (base + g2 + q < nb) __stcg(t.D + ((size_t)(base + g2 + q) * 3 + l) * H + j, d);
        }
        __syncthreads();
      }
    }
    cluster_sync();

    // ---- (B) gradients of the CTA's rows, summed over the batch in sample order
    float g[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int b0 = 0; b0 < nb; b0 += kTile) {
      const int cnt = min(kTile, nb - b0);
      __syncthreads();
      for (int i = tid; i < cnt * (H / 4); i += kTrainThreads) {
        const int b = i / (H / 4), c = 4 * (i % (H / 4));
        const float* A = t.A + (size_t)(b0 + b) * 3 * H + c;
        cp16(&S.tA[0][b][c], A);
        cp16(&S.tA[1][b][c], A + H);
      }
      for (int i = tid; i < cnt * 8; i += kTrainThreads) {   // 16-byte halves: layers 0..2 of D, layer 3's A
        const int b = i >> 3, k = (i >> 1) & 3, c = 4 * (i & 1);
        const float* src = (k < 3 ? t.D + ((size_t)(b0 + b) * 3 + k) * H : t.A + ((size_t)(b0 + b) * 3 + 2) * H) + 8 * rank;
        cp16((k < 3 ? &S.tD[k][b][0] : &S.tA3[b][0]) + c, src + c);
      }
      for (int i = tid; i < cnt * (kMaxOut / 4); i += kTrainThreads)
        cp16(&S.tD4[0][0] + 4 * i, t.D4 + (size_t)b0 * kMaxOut + 4 * i);
      for (int b = tid >> 5; b < cnt; b += kTrainThreads / 32)
        if ((tid & 31) < din) cp4(&S.tX[b][tid & 31], t.X + (size_t)(s0 + b0 + b) * din + (tid & 31));
      cp_wait();
      __syncthreads();
      if (main) {
#pragma unroll 8
        for (int b = 0; b < cnt; ++b) {
          const float a = S.tA[gl][b][gi];
          const float4 d = *reinterpret_cast<const float4*>(&S.tD[gl + 1][b][0]);
          const float4 e = *reinterpret_cast<const float4*>(&S.tD[gl + 1][b][4]);
          g[0] = fmaf(d.x, a, g[0]); g[1] = fmaf(d.y, a, g[1]); g[2] = fmaf(d.z, a, g[2]); g[3] = fmaf(d.w, a, g[3]);
          g[4] = fmaf(e.x, a, g[4]); g[5] = fmaf(e.y, a, g[5]); g[6] = fmaf(e.z, a, g[6]); g[7] = fmaf(e.w, a, g[7]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < kSmall; ++q) {
          int p = tid - 2 * H + q * 2 * H;
          if (p >= n_small) continue;
          float s = g[q];
          if (p < n_w1) {
            const int r = p / din, i = p % din;
#pragma unroll 16
            for (int b = 0; b < cnt; ++b) s = fmaf(S.tD[0][b][r], S.tX[b][i], s);
          } else if ((p -= n_w1) < 24) {
#pragma unroll 16
            for (int b = 0; b < cnt; ++b) s += S.tD[p >> 3][b][p & 7];
          } else if ((p -= 24) < n_w4) {
#pragma unroll 16
            for (int b = 0; b < cnt; ++b) s = fmaf(S.tD4[b][p / 8], S.tA3[b][p & 7], s);
          } else {
            p -= n_w4;
#pragma unroll 16
            for (int b = 0; b < cnt; ++b) s += S.tD4[b][p];
          }
          g[q] = s;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (pp[r] < 0) continue;
      if (t.update) {
        adam(g[r], th[r], m[r], v[r], t.lr, 0.9f, 0.999f, 1e-8f, corr.x, corr.y);
        __stcg(t.theta + pp[r], th[r]);
      } else {
        t.g[pp[r]] = g[r];
      }
    }
    if (t.losses && rank == 0 && mb % t.per_epoch == t.per_epoch - 1) {   // the epoch's last minibatch
      float s = 0.0f;
      for (int i = tid; i < nb * dout; i += kTrainThreads) {
        const float d = __ldcg(t.Y + i) - t.T[(size_t)s0 * dout + i];
        s = fmaf(d, d, s);
      }
      S.red[tid] = s;
      __syncthreads();
      for (int h = kTrainThreads / 2; h > 0; h >>= 1) {
        if (tid < h) S.red[tid] += S.red[tid + h];
        __syncthreads();
      }
      if (tid == 0) t.losses[mb / t.per_epoch] = S.red[0] / ((float)nb * (float)dout);
    }
    cluster_sync();
  }
  if (t.update)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (pp[r] < 0) continue;
      t.m[pp[r]] = m[r];
      t.v[pp[r]] = v[r];
    }
}

// ------------------------------------------------------------------- inference
// A sample's inputs and outputs as the caller has them: FP32 in network units, or FP64 in
// physical ones, standardised and scaled back in FP64 as numpy would, rounding included.
struct Scaling {
  const double *xm, *xs, *ym, *ys;
};
__device__ __forceinline__ float input(const float* X, size_t i, int, const Scaling&) { return X[i]; }
__device__ __forceinline__ float input(const double* X, size_t i, int c, const Scaling& s) {
  return (float)__ddiv_rn(__dsub_rn(X[i], s.xm[c]), s.xs[c]);
}
__device__ __forceinline__ void output(float* Y, size_t i, int, const Scaling&, float y) { Y[i] = y; }
__device__ __forceinline__ void output(double* Y, size_t i, int c, const Scaling& s, float y) {
  Y[i] = __dadd_rn(__dmul_rn((double)y, s.ys[c]), s.ym[c]);
}

// FP32 inference: tiles of 32 samples, one thread per neuron and 8 samples, so that a weight is
// read from shared memory once for eight multiply-adds (one thread per sample with its
// activations in local memory, and every pre-activation written out, before: 2^20 inputs on
// the device in 5.7 ms, now 0.93).
constexpr int kInferTile = 32, kInferThreads = 256;
struct InferSmem {
  alignas(16) float w2[H * kWP], w3[H * kWP];
  float w1[H * kXP], w4[kMaxOut * H], bias[3 * H + kMaxOut];
  float x[kInferTile][kMaxIn];
  alignas(16) float a[2][kInferTile][H];
};

template <class IO>
__global__ void __launch_bounds__(kInferThreads)
    k_infer_fp32(const float* __restrict__ theta, int din, int dout, const IO* __restrict__ X, int n, IO* __restrict__ Y,
                 Scaling sc) {
  extern __shared__ __align__(16) unsigned char raw[];
  InferSmem& S = *reinterpret_cast<InferSmem*>(raw);
  const Offs o = offsets(din, dout);
  const int tid = threadIdx.x;
  for (int i = tid; i < H * H; i += kInferThreads) {
    S.w2[(i >> 6) * kWP + (i & 63)] = theta[o.w2 + i];
    S.w3[(i >> 6) * kWP + (i & 63)] = theta[o.w3 + i];
  }
  for (int i = tid; i < H * din; i += kInferThreads) S.w1[(i / din) * kXP + i % din] = theta[o.w1 + i];
  for (int i = tid; i < dout * H; i += kInferThreads) S.w4[i] = theta[o.w4 + i];
  if (tid < H) {
    S.bias[tid] = theta[o.b1 + tid]; S.bias[H + tid] = theta[o.b2 + tid]; S.bias[2 * H + tid] = theta[o.b3 + tid];
  }
  if (tid < dout) S.bias[3 * H + tid] = theta[o.b4 + tid];
  const int j = tid & (H - 1), g8 = 8 * (tid >> 6);
  for (long long base = (long long)blockIdx.x * kInferTile; base < n; base += (long long)gridDim.x * kInferTile) {
    __syncthreads();
    for (int i = tid; i < kInferTile * din; i += kInferThreads)
      S.x[i / din][i % din] = base + i / din < n ? input(X, (size_t)base * din + i, i % din, sc) : 0.0f;
    __syncthreads();
    float acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = S.bias[j];
    for (int i = 0; i < din; ++i) {
      const float w = S.w1[j * kXP + i];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = fmaf(w, S.x[g8 + q][i], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) S.a[0][g8 + q][j] = gelu(acc[q]);
    __syncthreads();
    for (int l = 1; l < 3; ++l) {
      const float* w = (l == 1 ? S.w2 : S.w3) + j * kWP;
      const float(*in)[H] = S.a[(l - 1) & 1];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = S.bias[l * H + j];
#pragma unroll 2
      for (int i = 0; i < H; i += 4) {
        const float4 y = *reinterpret_cast<const float4*>(w + i);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 x = *reinterpret_cast<const float4*>(&in[g8 + q][i]);
          acc[q] = fmaf(y.w, x.w, fmaf(y.z, x.z, fmaf(y.y, x.y, fmaf(y.x, x.x, acc[q]))));
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) S.a[l & 1][g8 + q][j] = gelu(acc[q]);
      __syncthreads();
    }
    for (int e = tid; e < kInferTile * dout; e += kInferThreads) {
      const int r = e / dout, k = e % dout;
      if (base + r >= n) continue;
      float s = S.bias[3 * H + k];
#pragma unroll 16
      for (int i = 0; i < H; ++i) s = fmaf(S.w4[k * H + i], S.a[0][r][i], s);
      output(Y, (size_t)(base + r) * dout + k, k, sc, s);
    }
  }
}

// ---------------------------------------------------------------- BF16 inference
// Each warp takes 16 samples; a hidden layer is the 16 x 64 activation tile
// times W^T (64 x 64) on the tensor cores: 8 column tiles of 8 x 4 k-steps of
// mma.sync.m16n8k16 (BF16 in, FP32 accumulate).  Fragment ownership follows the
// PTX ISA layout of m16n8k16: with g = lane / 4 and t = lane % 4, A rows g and
// g + 8, columns 2t, 2t+1 (+8); B (k x n) rows 2t, 2t+1 (+8), column g; C rows
// g, g + 8, columns 2t, 2t + 1.
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}

__device__ __forceinline__ void mma_bf16(float* c, const unsigned* a, const unsigned* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

constexpr int kInferWarps = 8, kBP = H + 8;   // padded rows: the 8 columns of a B fragment on distinct banks

// The activations stay in registers: a layer's C fragments, biased, activated and rounded,
// are the next layer's A fragments (columns 8 nt + 2 t, + 1 of C are rows of the k-step
// nt / 2).  Only the last layer's go through shared memory, for the output sums over all
// columns in order.  2^20 inputs on the device
// in 0.62 ms before, 0.36 now.
template <class IO>
__global__ void __launch_bounds__(32 * kInferWarps)
    k_infer_bf16(const float* __restrict__ theta, int din, int dout, const IO* __restrict__ X, int n,
                 IO* __restrict__ Y, Scaling sc) {
  __shared__ __nv_bfloat16 sw[2][H * kBP];         // W2, W3 in BF16, [out][in]
  __shared__ float w1[kMaxIn][H];                  // W1 transposed
  __shared__ float w4[H * kMaxOut];
  __shared__ float bias[3 * H + kMaxOut];          // b1, b2, b3, b4
  extern __shared__ __align__(16) unsigned char raw[];
  const Offs o = offsets(din, dout);
  for (int i = threadIdx.x; i < H * H; i += blockDim.x) {
    sw[0][(i >> 6) * kBP + (i & 63)] = __float2bfloat16_rn(theta[o.w2 + i]);
    sw[1][(i >> 6) * kBP + (i & 63)] = __float2bfloat16_rn(theta[o.w3 + i]);
  }
  for (int i = threadIdx.x; i < H * din; i += blockDim.x) w1[i % din][i / din] = theta[o.w1 + i];
  for (int i = threadIdx.x; i < dout * H; i += blockDim.x) w4[i] = theta[o.w4 + i];
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    bias[i] = theta[o.b1 + i]; bias[H + i] = theta[o.b2 + i]; bias[2 * H + i] = theta[o.b3 + i];
  }
  for (int i = threadIdx.x; i < dout; i += blockDim.x) bias[3 * H + i] = theta[o.b4 + i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  float(*A)[H + 1] = reinterpret_cast<float(*)[H + 1]>(raw) + 16 * warp;     // per-warp tile: inputs, then activations
  const long long tiles = ((long long)n + 15) / 16;
  for (long long tile = (long long)blockIdx.x * kInferWarps + warp; tile < tiles;
       tile += (long long)gridDim.x * kInferWarps) {
    const long long base = tile * 16;
    const int rows = n - base < 16 ? (int)(n - base) : 16;
    for (int e = lane; e < 16 * din; e += 32)
      A[e / din][e % din] = e / din < rows ? input(X, (size_t)base * din + e, e % din, sc) : 0.0f;
    __syncwarp();
    // layer 1 in FP32 (din is small)
    float c[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      c[nt][0] = c[nt][2] = bias[nt * 8 + 2 * t];
      c[nt][1] = c[nt][3] = bias[nt * 8 + 2 * t + 1];
    }
    for (int i = 0; i < din; ++i) {
      const float xg = A[g][i], xh = A[g + 8][i];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const float2 w = *reinterpret_cast<const float2*>(&w1[i][nt * 8 + 2 * t]);
        c[nt][0] = fmaf(w.x, xg, c[nt][0]); c[nt][1] = fmaf(w.y, xg, c[nt][1]);
        c[nt][2] = fmaf(w.x, xh, c[nt][2]); c[nt][3] = fmaf(w.y, xh, c[nt][3]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int q = 0; q < 4; ++q) c[nt][q] = gelu(c[nt][q]);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      unsigned a[4][4];
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        a[ks][0] = pack_bf16(c[2 * ks][0], c[2 * ks][1]);
        a[ks][1] = pack_bf16(c[2 * ks][2], c[2 * ks][3]);
        a[ks][2] = pack_bf16(c[2 * ks + 1][0], c[2 * ks + 1][1]);
        a[ks][3] = pack_bf16(c[2 * ks + 1][2], c[2 * ks + 1][3]);
      }
      const float* bl = bias + (l + 1) * H;
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.0f;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          // B[k][n] = W[n][k]: column n = nt * 8 + g, rows k0 + 2t, +1 and +8, +9
          const __nv_bfloat16* wr = sw[l] + (nt * 8 + g) * kBP + ks * 16 + 2 * t;
          unsigned b[2];
          b[0] = *reinterpret_cast<const unsigned*>(wr);
          b[1] = *reinterpret_cast<const unsigned*>(wr + 8);
          mma_bf16(c[nt], a[ks], b);
        }
        const int col = nt * 8 + 2 * t;
        c[nt][0] = gelu(c[nt][0] + bl[col]);
        c[nt][1] = gelu(c[nt][1] + bl[col + 1]);
        c[nt][2] = gelu(c[nt][2] + bl[col]);
        c[nt][3] = gelu(c[nt][3] + bl[col + 1]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int col = nt * 8 + 2 * t;
      A[g][col] = c[nt][0]; A[g][col + 1] = c[nt][1];
      A[g + 8][col] = c[nt][2]; A[g + 8][col + 1] = c[nt][3];
    }
    __syncwarp();
    // output layer in FP32
    for (int e = lane; e < rows * dout; e += 32) {
      const int r = e / dout, j = e % dout;
      float s = bias[3 * H + j];
#pragma unroll 16
      for (int i = 0; i < H; ++i) s = fmaf(w4[j * H + i], A[r][i], s);
      output(Y, (size_t)(base + r) * dout + j, j, sc, s);
    }
    __syncwarp();
  }
}
constexpr size_t kBf16Smem = sizeof(float) * 16 * kInferWarps * (H + 1);

}  // namespace

struct tg_mlp {
  int din = 0, dout = 0, np = 0, sms = 148;
  long long step = 0;
  cudaStream_t stream = nullptr;
  float *theta = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;
  // training scratch, grown on demand
  int cap = 0;
  float *X = nullptr, *T = nullptr, *A = nullptr, *Y = nullptr, *D = nullptr, *D4 = nullptr, *losses = nullptr;
  int cap_losses = 0;
  float2* corr = nullptr;           // kMaxBatches bias corrections
  // tg_mlp_predict_scaled: scaling vectors followed by the rows of a call without staging, and
  // the staging lanes: a stream each and equal parts of one pinned and one device block
  double* scale = nullptr;
  size_t scale_rows = 0;
  static constexpr int kLanes = 4, kRows = 32768, kFirstRows = 256;
  cudaStream_t lane[kLanes] = {};
  char *pin = nullptr, *dev = nullptr;
  size_t lane_bytes = 0;
  size_t plain_bytes = 0;           // moved without staging by calls of more than kRows rows
  std::string err;
};
constexpr int kMaxBatches = 4096;   // minibatches of one training launch (64 samples each: about 40 ms)
constexpr size_t kPlainBytes = size_t(16) << 20;   // see tg_mlp_predict_scaled

namespace {

tg_status mfail(tg_mlp* h, tg_status st, const std::string& msg) {
  if (h) h->err = msg;
  g_mlp_error = msg;
  return st;
}

#define TM_CUDA(h, call)                                                                          \
  do {                                                                                            \
    cudaError_t e_ = (call);                                                                      \
    if (e_ != cudaSuccess)                                                                        \
      return mfail((h), TG_CUDA_ERROR, std::string(#call " failed: ") + cudaGetErrorString(e_)); \
  } while (0)

tg_status reserve(tg_mlp* h, int n) {
  if (n <= h->cap) return TG_OK;
  cudaFree(h->X); cudaFree(h->T); cudaFree(h->A); cudaFree(h->Y); cudaFree(h->D); cudaFree(h->D4);
  h->X = h->T = h->A = h->Y = h->D = h->D4 = nullptr;
  h->cap = 0;
  TM_CUDA(h, cudaMalloc((void**)&h->X, (size_t)n * h->din * sizeof(float)));
  TM_CUDA(h, cudaMalloc((void**)&h->T, (size_t)n * h->dout * sizeof(float)));
  TM_CUDA(h, cudaMalloc((void**)&h->Y, (size_t)n * h->dout * sizeof(float)));
  TM_CUDA(h, cudaMalloc((void**)&h->D4, (size_t)n * kMaxOut * sizeof(float)));
  TM_CUDA(h, cudaMalloc((void**)&h->A, (size_t)n * 3 * H * sizeof(float)));
  TM_CUDA(h, cudaMalloc((void**)&h->D, (size_t)n * 3 * H * sizeof(float)));
  h->cap = n;
  return TG_OK;
}

tg_status reserve_losses(tg_mlp* h, int n) {
  if (!h->corr) TM_CUDA(h, cudaMalloc((void**)&h->corr, kMaxBatches * sizeof(float2)));
  if (n <= h->cap_losses) return TG_OK;
  cudaFree(h->losses);
  h->losses = nullptr;
  h->cap_losses = 0;
  TM_CUDA(h, cudaMalloc((void**)&h->losses, (size_t)n * sizeof(float)));
  h->cap_losses = n;
  return TG_OK;
}

Train train_args(tg_mlp* h, int n, int batch) {
  Train t{};
  t.X = h->X; t.T = h->T;
  t.n = n; t.din = h->din; t.dout = h->dout; t.batch = batch; t.per_epoch = (n + batch - 1) / batch;
  t.theta = h->theta; t.m = h->m; t.v = h->v; t.g = h->g;
  t.A = h->A; t.D = h->D; t.D4 = h->D4; t.Y = h->Y;
  t.losses = h->losses;
  return t;
}

// The inference kernel of a precision over n inputs on `st`.
template <class IO>
void enqueue_infer(const tg_mlp* h, const IO* X, int n, IO* Y, const Scaling& sc, int precision, cudaStream_t st) {
  if (precision == 1) {
    const long long tiles = ((long long)n + 15) / 16;
    const int grid = (int)std::min<long long>((tiles + kInferWarps - 1) / kInferWarps, 4LL * h->sms);
    k_infer_bf16<IO><<<grid, 32 * kInferWarps, kBf16Smem, st>>>(h->theta, h->din, h->dout, X, n, Y, sc);
  } else {
    const int grid = (int)std::min<long long>(((long long)n + kInferTile - 1) / kInferTile, 3LL * h->sms);
    k_infer_fp32<IO><<<grid, kInferThreads, sizeof(InferSmem), st>>>(h->theta, h->din, h->dout, X, n, Y, sc);
  }
}

}  // namespace

extern "C" {

tg_status tg_mlp_create(int din, int dout, unsigned long long seed, tg_mlp** out) {
  if (!out) return mfail(nullptr, TG_INVALID_ARG, "out is NULL");
  *out = nullptr;
  if (din < 1 || din > kMaxIn || dout < 1 || dout > kMaxOut)
    return mfail(nullptr, TG_INVALID_ARG, "din must be 1..32 and dout 1..8");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return mfail(nullptr, TG_NO_DEVICE, "no CUDA device visible; the GPU path has no CPU fallback");
  tg_mlp* h = new (std::nothrow) tg_mlp();
  if (!h) return mfail(nullptr, TG_INVALID_ARG, "out of host memory");
  h->din = din; h->dout = dout;
  h->np = offsets(din, dout).n;
  int device = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device);
  // He-style uniform initialisation from a 64-bit linear congruential stream (Knuth's MMIX constants)
  std::vector<float> th(h->np, 0.0f);
  const Offs o = offsets(din, dout);
  unsigned long long st = seed * 6364136223846793005ULL + 1442695040888963407ULL;
  auto uni = [&]() {
    st = st * 6364136223846793005ULL + 1442695040888963407ULL;
    return (double)(st >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](int off, int rows, int cols) {
    const double a = std::sqrt(6.0 / cols);
    for (int i = 0; i < rows * cols; ++i) th[off + i] = (float)((2.0 * uni() - 1.0) * a);
  };
  fill(o.w1, H, din); fill(o.w2, H, H); fill(o.w3, H, H); fill(o.w4, dout, H);
  cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->theta, (h->np + kMaxOut) * sizeof(float));   // copied in 16-byte words
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->m, h->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->v, h->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->g, h->np * sizeof(float));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(TrainSmem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_infer_fp32<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(InferSmem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_infer_fp32<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(InferSmem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_infer_bf16<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBf16Smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_infer_bf16<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBf16Smem);
  if (e == cudaSuccess) e = cudaMemset(h->theta, 0, (h->np + kMaxOut) * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(h->theta, th.data(), h->np * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(h->m, 0, h->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(h->v, 0, h->np * sizeof(float));
  if (e != cudaSuccess) {
    tg_mlp_destroy(h);
    return mfail(nullptr, TG_CUDA_ERROR, cudaGetErrorString(e));
  }
  *out = h;
  return TG_OK;
}

tg_status tg_mlp_destroy(tg_mlp* h) {
  if (!h) return TG_OK;
  if (h->stream) cudaStreamSynchronize(h->stream);
  cudaFree(h->theta); cudaFree(h->m); cudaFree(h->v); cudaFree(h->g); cudaFree(h->losses); cudaFree(h->corr);
  cudaFree(h->X); cudaFree(h->T); cudaFree(h->A); cudaFree(h->Y); cudaFree(h->D); cudaFree(h->D4); cudaFree(h->scale);
  for (cudaStream_t s : h->lane)
    if (s) cudaStreamDestroy(s);
  cudaFreeHost(h->pin);
  cudaFree(h->dev);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return TG_OK;
}

const char* tg_mlp_last_error(const tg_mlp* h) { return h ? h->err.c_str() : g_mlp_error.c_str(); }

int tg_mlp_n_params(const tg_mlp* h) { return h ? h->np : 0; }

tg_status tg_mlp_get_params(tg_mlp* h, float* theta) {
  if (!h || !theta) return mfail(h, TG_INVALID_ARG, "NULL argument");
  TM_CUDA(h, cudaMemcpyAsync(theta, h->theta, h->np * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
  TM_CUDA(h, cudaStreamSynchronize(h->stream));
  return TG_OK;
}

tg_status tg_mlp_set_params(tg_mlp* h, const float* theta) {
  if (!h || !theta) return mfail(h, TG_INVALID_ARG, "NULL argument");
  TM_CUDA(h, cudaMemcpyAsync(h->theta, theta, h->np * sizeof(float), cudaMemcpyHostToDevice, h->stream));
  TM_CUDA(h, cudaMemsetAsync(h->m, 0, h->np * sizeof(float), h->stream));
  TM_CUDA(h, cudaMemsetAsync(h->v, 0, h->np * sizeof(float), h->stream));
  TM_CUDA(h, cudaStreamSynchronize(h->stream));
  h->step = 0;
  return TG_OK;
}

// Loss and parameter gradient of one batch (host arrays), for gradient checks.
tg_status tg_mlp_loss_grad(tg_mlp* h, const float* X, const float* T, int n, float* loss, float* grad) {
  if (!h || !X || !T || n < 1) return mfail(h, TG_INVALID_ARG, "bad batch");
  tg_status st = reserve(h, n);
  if (st != TG_OK || (st = reserve_losses(h, 1)) != TG_OK) return st;
  TM_CUDA(h, cudaMemcpyAsync(h->X, X, (size_t)n * h->din * sizeof(float), cudaMemcpyHostToDevice, h->stream));
  TM_CUDA(h, cudaMemcpyAsync(h->T, T, (size_t)n * h->dout * sizeof(float), cudaMemcpyHostToDevice, h->stream));
  Train t = train_args(h, n, n);
  t.count = 1;
  k_train<<<kCl, kTrainThreads, sizeof(TrainSmem), h->stream>>>(t);
  TM_CUDA(h, cudaGetLastError());
  if (loss) TM_CUDA(h, cudaMemcpyAsync(loss, h->losses, sizeof(float), cudaMemcpyDeviceToHost, h->stream));
  if (grad) TM_CUDA(h, cudaMemcpyAsync(grad, h->g, h->np * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
  TM_CUDA(h, cudaStreamSynchronize(h->stream));
  return TG_OK;
}

// Adam training on (X, T) (host arrays, n samples) in mini-batches taken in
// order, `epochs` passes.  losses (may be NULL) receives the last batch loss of
// every epoch.
tg_status tg_mlp_train(tg_mlp* h, const float* X, const float* T, int n, int epochs, int batch, float lr,
                       float* losses) {
  if (!h || !X || !T || n < 1 || epochs < 1 || batch < 1) return mfail(h, TG_INVALID_ARG, "bad training set");
  if (batch > n) batch = n;
  tg_status st = reserve(h, n);
  if (st != TG_OK || (st = reserve_losses(h, epochs)) != TG_OK) return st;
  TM_CUDA(h, cudaMemcpyAsync(h->X, X, (size_t)n * h->din * sizeof(float), cudaMemcpyHostToDevice, h->stream));
  TM_CUDA(h, cudaMemcpyAsync(h->T, T, (size_t)n * h->dout * sizeof(float), cudaMemcpyHostToDevice, h->stream));
  const float b1 = 0.9f, b2 = 0.999f;
  Train t = train_args(h, n, batch);
  t.lr = lr;
  t.update = 1;
  if (!losses) t.losses = nullptr;
  const long total = (long)t.per_epoch * epochs;
  const long most = std::max(1, kMaxBatches / std::max(1, (batch + kTile - 1) / kTile));
  std::vector<float2> corr;
  cudaError_t e = cudaSuccess;
  for (long at = 0; at < total && e == cudaSuccess; at += most) {
    t.first = at;
    t.count = (int)std::min(most, total - at);
    corr.resize(t.count);
    for (int i = 0; i < t.count; ++i) {
      ++h->step;
      corr[i].x = 1.0f - std::pow(b1, (float)h->step);
      corr[i].y = 1.0f - std::pow(b2, (float)h->step);
    }
    t.corr = h->corr;
    // corr is reused by the next launch, in stream order; the host copy is staged at the call
    e = cudaMemcpyAsync(h->corr, corr.data(), t.count * sizeof(float2), cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) {
      k_train<<<kCl, kTrainThreads, sizeof(TrainSmem), h->stream>>>(t);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess && losses)
    e = cudaMemcpyAsync(losses, h->losses, (size_t)epochs * sizeof(float), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) return mfail(h, TG_CUDA_ERROR, cudaGetErrorString(e));
  return TG_OK;
}

// Evaluation of n inputs (host or device arrays; device when on_device != 0):
// precision 0 = FP32 SIMT (the training path), 1 = BF16 tensor cores.
tg_status tg_mlp_predict(tg_mlp* h, const float* X, int n, float* Y, int precision, int on_device) {
  if (!h || !X || !Y || n < 1) return mfail(h, TG_INVALID_ARG, "bad prediction set");
  const float* dX = X;
  float* dY = Y;
  float* own = nullptr;
  if (!on_device) {
    TM_CUDA(h, cudaMalloc((void**)&own, (size_t)n * (h->din + h->dout) * sizeof(float)));
    TM_CUDA(h, cudaMemcpyAsync(own, X, (size_t)n * h->din * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    dX = own;
    dY = own + (size_t)n * h->din;
  }
  enqueue_infer(h, dX, n, dY, Scaling{}, precision, h->stream);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && !on_device)
    e = cudaMemcpyAsync(Y, dY, (size_t)n * h->dout * sizeof(float), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(own);
  if (e != cudaSuccess) return mfail(h, TG_CUDA_ERROR, cudaGetErrorString(e));
  return TG_OK;
}

// The staging lanes of a call that moves `bytes`: kLanes parts that take it in 32 chunks, 1 MiB
// at least, a power of two.  False: no pinned memory to be had.
static bool stage_lanes(tg_mlp* h, size_t bytes) {
  const size_t most = (size_t)tg_mlp::kRows * (h->din + h->dout) * sizeof(double);
  size_t want = size_t(1) << 20;
  while (want < most && want < bytes / 32) want *= 2;
  if (want <= h->lane_bytes) return true;
  cudaFreeHost(h->pin);
  cudaFree(h->dev);
  h->pin = h->dev = nullptr;
  h->lane_bytes = 0;
  cudaError_t e = cudaMallocHost((void**)&h->pin, tg_mlp::kLanes * want);
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->dev, tg_mlp::kLanes * want);
  for (cudaStream_t& s : h->lane)
    if (e == cudaSuccess && !s) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  h->lane_bytes = want;
  return true;
}

// The same from and to physical units, host arrays in FP64: Y = ym + ys net((X - xm) / xs).
// A large set goes in chunks through a few host threads, each copying its chunks into pinned
// memory, so that copies both ways and the network overlap.  Page-locking takes 1 to 4 ms and
// more with its size, about what 16 MB lose by pageable copies, so a network gets that memory
// once its large calls have moved so much: a study often makes one call.  ms of a new network's
// first call / of later ones in FP32, with the scaling in numpy and pageable copies: 2^20 inputs
// of 3 43 / 43, 100 000 of 20 9.4 / 8.7, 100 000 of 3 4.2 / 4.2; with four pinned buffers of
// 32768 rows at the first large call 13 / 2.2, 20 / 1.1, 12.7 / 0.6; now 11 / 2.2, 6.3 / 0.9,
// 1.3 / 0.4.
tg_status tg_mlp_predict_scaled(tg_mlp* h, const double* X, int n, const double* xm, const double* xs, const double* ym,
                                const double* ys, double* Y, int precision) {
  if (!h || !X || !Y || !xm || !xs || !ym || !ys || n < 1) return mfail(h, TG_INVALID_ARG, "bad prediction set");
  const int din = h->din, dout = h->dout;
  const size_t row = (din + dout) * sizeof(double), bytes = n * row;
  bool plain = n <= tg_mlp::kRows;
  if (!plain && !h->pin && h->plain_bytes + bytes < kPlainBytes) {
    h->plain_bytes += bytes;
    plain = true;
  }
  if (!plain) plain = !stage_lanes(h, bytes);
  const int ns = 2 * (din + dout);
  const size_t want = plain ? n : 0;
  if (!h->scale || want > h->scale_rows) {
    TM_CUDA(h, cudaStreamSynchronize(h->stream));
    cudaFree(h->scale);
    h->scale = nullptr;
    h->scale_rows = 0;
    const size_t rows = std::max<size_t>(tg_mlp::kFirstRows, want);
    TM_CUDA(h, cudaMalloc((void**)&h->scale, ns * sizeof(double) + rows * row));
    h->scale_rows = rows;
  }
  const Scaling S{h->scale, h->scale + din, h->scale + 2 * din, h->scale + 2 * din + dout};
  // a small call is bound by its copies (5 us each): scaling and rows go in one, into memory
  // that is kept (200 rows of 3 inputs 53 -> 45 us)
  constexpr size_t kOne = 2048;
  double in[kOne];
  std::memcpy(in, xm, din * sizeof(double));
  std::memcpy(in + din, xs, din * sizeof(double));
  std::memcpy(in + 2 * din, ym, dout * sizeof(double));
  std::memcpy(in + 2 * din + dout, ys, dout * sizeof(double));
  const size_t nx = (size_t)n * din;
  const bool one = plain && ns + nx <= kOne;
  if (one) std::memcpy(in + ns, X, nx * sizeof(double));
  TM_CUDA(h, cudaMemcpyAsync(h->scale, in, (one ? ns + nx : ns) * sizeof(double), cudaMemcpyHostToDevice, h->stream));
  if (plain) {
    double *dx = h->scale + ns, *dy = dx + nx;
    cudaError_t e = one ? cudaSuccess : cudaMemcpyAsync(dx, X, nx * sizeof(double), cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) {
      enqueue_infer(h, (const double*)dx, n, dy, S, precision, h->stream);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(Y, dy, (size_t)n * dout * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    const cudaError_t e2 = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess || e2 != cudaSuccess) return mfail(h, TG_CUDA_ERROR, cudaGetErrorString(e != cudaSuccess ? e : e2));
    return TG_OK;
  }
  const int per = (int)(h->lane_bytes / row);       // rows of a lane's chunk
  const int chunks = (int)((n + (long long)per - 1) / per), lanes = std::min<int>(tg_mlp::kLanes, chunks);
  TM_CUDA(h, cudaStreamSynchronize(h->stream));      // weights and scaling are in place
  int device = 0;
  TM_CUDA(h, cudaGetDevice(&device));
  std::vector<cudaError_t> errs(lanes, cudaSuccess);
  auto work = [&](int l) {
    cudaError_t e = cudaSetDevice(device);
    double *pin = (double*)(h->pin + l * h->lane_bytes), *dev = (double*)(h->dev + l * h->lane_bytes);
    double *pout = pin + (size_t)per * din, *dout_ = dev + (size_t)per * din;
    for (int c = l; c < chunks && e == cudaSuccess; c += lanes) {
      const size_t r0 = (size_t)c * per;
      const int rows = (int)std::min<size_t>(per, n - r0);
      std::memcpy(pin, X + r0 * din, (size_t)rows * din * sizeof(double));
      e = cudaMemcpyAsync(dev, pin, (size_t)rows * din * sizeof(double), cudaMemcpyHostToDevice, h->lane[l]);
      if (e != cudaSuccess) break;
      enqueue_infer(h, (const double*)dev, rows, dout_, S, precision, h->lane[l]);
      if ((e = cudaGetLastError()) != cudaSuccess) break;
      e = cudaMemcpyAsync(pout, dout_, (size_t)rows * dout * sizeof(double), cudaMemcpyDeviceToHost, h->lane[l]);
      if (e == cudaSuccess) e = cudaStreamSynchronize(h->lane[l]);
      if (e == cudaSuccess) std::memcpy(Y + r0 * dout, pout, (size_t)rows * dout * sizeof(double));
    }
    errs[l] = e;
  };
  std::vector<std::thread> th;
  int started = 1;
  try {
    for (; started < lanes; ++started) th.emplace_back(work, started);
  } catch (const std::system_error&) {   // no thread to be had: this one does the rest
  }
  work(0);
  for (int l = started; l < lanes; ++l) work(l);
  for (auto& x : th) x.join();
  for (cudaError_t e : errs)
    if (e != cudaSuccess) return mfail(h, TG_CUDA_ERROR, cudaGetErrorString(e));
  return TG_OK;
}

}  // extern "C"
