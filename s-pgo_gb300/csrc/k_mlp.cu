// Learned LM damping controller: a 16 -> 64 -> 64 -> 2 MLP with exact GELU.
//
// No counterpart in the reference (S-PGO has no damping schedule at all).
// Parameters are one flat FP32 vector: W1 [64x16] (out x in), b1 [64],
// W2 [64x64], b2 [64], W3 [2x64], b3 [2]  (5378 floats).  Outputs: out0 =
// proposed change of log10(lambda), out1 = logit that the current damping gives
// an accepted step.  Training loss per sample: (out0 - t0)^2 + BCE(out1, t1),
// averaged over the batch.
//
// Kernels: FP32 forward; forward, loss and parameter gradient of 16 samples a CTA (no
// atomics on the parameters) and the sum of the CTAs' gradients; Adam; and the BF16
// inference the LM loop runs (warp per problem, FP32 accumulation).
#include <cuda_bf16.h>
#include <cstddef>

#include "kernels.cuh"
#include "dfloat.cuh"

#include <type_traits>

namespace spgo {

constexpr int kIn = 16, kH = 64, kOut = 2;
constexpr int kW1 = 0, kB1 = kW1 + kH * kIn, kW2 = kB1 + kH, kB2 = kW2 + kH * kH, kW3 = kB2 + kH,
              kB3 = kW3 + kOut * kH, kParams = kB3 + kOut;
static_assert(kParams == SPGO_MLP_PARAMS, "parameter count");

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * expf(-0.5f * x * x) * 0.39894228040143268f;
}

// One CTA takes kSamples samples, eight at a time: thread = (sample, hidden unit), the weights
// in shared memory with rows padded to an odd pitch (threads read consecutive units of a row or
// of a column without bank conflicts), activations and deltas beside them.  A thread per sample
// instead, walking both 64-wide layers alone, left 512 samples on 4 SMs: forward 105 us and
// deltas 141 us, where this takes 12 us for both and the gradient (35 us before).
constexpr int kSamples = 16;
constexpr int kMlpThreads = 512;
constexpr int kCachePerSample = 6 * kH + 2;
static_assert(kCachePerSample == SPGO_MLP_CACHE_PER_SAMPLE, "cache size");
// (the gradient's partial sums below: one set of parameters per CTA but the first fits the
// scratch of the samples of any batch)
static_assert(kParams <= kSamples * kCachePerSample, "partial gradients fit the cache");

struct MlpTrain {
  float w1[kH][kIn + 1], w2[kH][kH + 1], w3[kOut][kH], b1[kH], b2[kH], b3[kOut], pad[2];
  float x[kSamples][kIn], h1[kSamples][kH], h2[kSamples][kH], dz1[kSamples][kH], dz2[kSamples][kH];
  float o[kSamples][kOut], d[kSamples][kOut], loss[kSamples];
  float part[kMlpThreads / 32][kOut];
};
static_assert(offsetof(MlpTrain, x) % 16 == 0 && kSamples * kIn % 4 == 0, "vector reads of the activations");

__device__ __forceinline__ void mlp_load(MlpTrain &m, const float *theta, const float *X, int s0, int n) {
  for (int i = threadIdx.x; i < kH * kIn; i += blockDim.x) m.w1[i / kIn][i % kIn] = theta[kW1 + i];
  for (int i = threadIdx.x; i < kH * kH; i += blockDim.x) m.w2[i / kH][i % kH] = theta[kW2 + i];
  for (int i = threadIdx.x; i < kOut * kH; i += blockDim.x) m.w3[i / kH][i % kH] = theta[kW3 + i];
  for (int i = threadIdx.x; i < kH; i += blockDim.x) {
    m.b1[i] = theta[kB1 + i];
    m.b2[i] = theta[kB2 + i];
    if (i < kOut) m.b3[i] = theta[kB3 + i];
  }
  for (int i = threadIdx.x; i < kSamples * kIn; i += blockDim.x)
    m.x[i / kIn][i % kIn] = s0 + i / kIn < n ? X[(size_t)s0 * kIn + i] : 0.f;
}

// samples q .. q + 7 of the CTA through both layers; z1, z2 of the thread's (sample, unit) and
// the outputs in m.o
__device__ __forceinline__ void mlp_layers(MlpTrain &m, int q, float &z1, float &z2) {
  const int s = q + threadIdx.x / kH, j = threadIdx.x % kH, lane = threadIdx.x & 31;
  z1 = m.b1[j];
#pragma unroll
  for (int k = 0; k < kIn; ++k) z1 += m.w1[j][k] * m.x[s][k];
  m.h1[s][j] = gelu(z1);
  __syncthreads();
  z2 = m.b2[j];
#pragma unroll 16
  for (int k = 0; k < kH; ++k) z2 += m.w2[j][k] * m.h1[s][k];
  const float h2 = gelu(z2);
  m.h2[s][j] = h2;
  const float p0 = warp_sum(m.w3[0][j] * h2), p1 = warp_sum(m.w3[1][j] * h2);  // (two warps per sample)
  if (lane == 0) {
    m.part[threadIdx.x >> 5][0] = p0;
    m.part[threadIdx.x >> 5][1] = p1;
  }
  __syncthreads();
  if (j < kOut) m.o[s][j] = m.b3[j] + (m.part[(threadIdx.x / kH) * 2][j] + m.part[(threadIdx.x / kH) * 2 + 1][j]);
  __syncthreads();
}

// forward; cache (optional) holds z1 [n x 64] then z2 [n x 64]
__global__ void __launch_bounds__(kMlpThreads) k_mlp_fwd(const float *__restrict__ theta, const float *__restrict__ X,
                                                         int n, float *__restrict__ out, float *__restrict__ cache) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MlpTrain &m = *reinterpret_cast<MlpTrain *>(smem_raw);
  const int s0 = kSamples * blockIdx.x;
  mlp_load(m, theta, X, s0, n);
  __syncthreads();
  for (int q = 0; q < min(kSamples, n - s0); q += kMlpThreads / kH) {
    float z1, z2;
    mlp_layers(m, q, z1, z2);
    const int s = s0 + q + threadIdx.x / kH, j = threadIdx.x % kH;
    if (s >= n) continue;
    if (cache) {
      cache[(size_t)s * kH + j] = z1;
      cache[(size_t)n * kH + (size_t)s * kH + j] = z2;
    }
    if (j < kOut) out[2 * s + j] = m.o[s - s0][j];
  }
}

// Forward, loss and parameter gradient of the CTA's samples, no atomics on the parameters: the
// samples' deltas stay in shared memory, each thread sums 4 x 2 entries of W2's gradient (and
// its share of the others) over them, and the CTA writes its sums to part (CTA g > 0) or
// grad (CTA 0); k_mlp_sum adds them up.
__global__ void __launch_bounds__(kMlpThreads) k_mlp_grad(const float *__restrict__ theta, const float *__restrict__ X,
                                                          const float *__restrict__ T, int n, float *__restrict__ out,
                                                          float *__restrict__ part, float *__restrict__ grad,
                                                          float *__restrict__ loss) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MlpTrain &m = *reinterpret_cast<MlpTrain *>(smem_raw);
  const int s0 = kSamples * blockIdx.x, ns = min(kSamples, n - s0), tid = threadIdx.x;
  mlp_load(m, theta, X, s0, n);
  __syncthreads();
  const float inv_n = 1.f / (float)n;
  for (int q = 0; q < ns; q += kMlpThreads / kH) {
    float z1, z2;
    mlp_layers(m, q, z1, z2);
    const int s = q + tid / kH, j = tid % kH;
    if (j == 0) {
      m.d[s][0] = m.d[s][1] = m.loss[s] = 0.f;
      if (s < ns) {
        const float o0 = m.o[s][0], o1 = m.o[s][1], t0 = T[2 * (s0 + s)], t1 = T[2 * (s0 + s) + 1];
        const float sig = 1.f / (1.f + expf(-o1));
        m.loss[s] = (o0 - t0) * (o0 - t0) + (fmaxf(o1, 0.f) + log1pf(expf(-fabsf(o1)))) - t1 * o1;
        m.d[s][0] = 2.f * (o0 - t0) * inv_n;
        m.d[s][1] = (sig - t1) * inv_n;
        out[2 * (s0 + s)] = o0;
        out[2 * (s0 + s) + 1] = o1;
      }
    }
    __syncthreads();
    const float g2 = (m.d[s][0] * m.w3[0][j] + m.d[s][1] * m.w3[1][j]) * gelu_grad(z2);
    m.dz2[s][j] = g2;
    __syncthreads();
    float acc = 0.f;
#pragma unroll 16
    for (int k = 0; k < kH; ++k) acc += m.dz2[s][k] * m.w2[k][j];
    m.dz1[s][j] = acc * gelu_grad(z1);
  }
  __syncthreads();
  if (tid == 0) {
    float l = 0.f;
    for (int s = 0; s < ns; ++s) l += m.loss[s];
    atomicAdd(loss, l / (float)n);
  }
  float *dst = blockIdx.x ? part + (size_t)(blockIdx.x - 1) * kParams : grad;
  {  // W2: rows j0 .. j0 + 3, columns k0, k0 + 1
    const int j0 = 4 * (tid / 32), k0 = 2 * (tid % 32);
    float a[4][2] = {};
    for (int s = 0; s < ns; ++s) {
      const float2 h = *reinterpret_cast<const float2 *>(&m.h1[s][k0]);
      const float4 z = *reinterpret_cast<const float4 *>(&m.dz2[s][j0]);
      const float zv[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i][0] += zv[i] * h.x;
        a[i][1] += zv[i] * h.y;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 2; ++k) dst[kW2 + (j0 + i) * kH + k0 + k] = a[i][k];
  }
  for (int p = tid; p < kH * kIn; p += kMlpThreads) {
    const int j = p / kIn, k = p % kIn;
    float a = 0.f;
    for (int s = 0; s < ns; ++s) a += m.dz1[s][j] * m.x[s][k];
    dst[kW1 + p] = a;
  }
  if (tid < 2 * kH) {  // b1, b2
    const float(*z)[kH] = tid < kH ? m.dz1 : m.dz2;
    float a = 0.f;
    for (int s = 0; s < ns; ++s) a += z[s][tid % kH];
    dst[(tid < kH ? kB1 : kB2) + tid % kH] = a;
  } else if (tid < 4 * kH) {  // W3
    const int o = (tid - 2 * kH) / kH, j = tid % kH;
    float a = 0.f;
    for (int s = 0; s < ns; ++s) a += m.d[s][o] * m.h2[s][j];
    dst[kW3 + o * kH + j] = a;
  } else if (tid < 4 * kH + kOut) {  // b3
    float a = 0.f;
    for (int s = 0; s < ns; ++s) a += m.d[s][tid - 4 * kH];
    dst[kB3 + tid - 4 * kH] = a;
  }
}

// grad += the other CTAs' sums: 32 parameters a CTA, eight slices of the partial sums
__global__ void __launch_bounds__(256) k_mlp_sum(const float *__restrict__ part, int n_part, float *__restrict__ grad) {
  __shared__ float red[8][33];
  const int p = 32 * blockIdx.x + (threadIdx.x & 31), w = threadIdx.x >> 5;
  float a = 0.f;
  if (p < kParams) {
    if (w == 0) a = grad[p];
#pragma unroll 4
    for (int g = w; g < n_part; g += 8) a += part[(size_t)g * kParams + p];
  }
  red[w][threadIdx.x & 31] = a;
  __syncthreads();
  if (w == 0 && p < kParams) {
#pragma unroll
    for (int k = 1; k < 8; ++k) a += red[k][threadIdx.x & 31];
    grad[p] = a;
  }
}

__global__ void k_mlp_adam(float *theta, const float *grad, float *m, float *v, int step, float lr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  const float b1 = 0.9f, b2 = 0.999f, e = 1e-8f;
  const float g = grad[i];
  const float mi = b1 * m[i] + (1.f - b1) * g;
  const float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float mh = mi / (1.f - powf(b1, (float)step)), vh = vi / (1.f - powf(b2, (float)step));
  theta[i] -= lr * mh / (sqrtf(vh) + e);
}

// the controller's inference weights: each parameter rounded to BF16, stored as
// FP32 in the shared-memory layout below (weight matrices transposed)
__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16(v)); }

// BF16-weight inference, one feature vector per warp: lanes split the hidden
// units, FP32 accumulation.  The weights live in shared memory as FP32 copies of
// the BF16-rounded parameters, both matrices transposed so that lanes read
// consecutive hidden units; spgo_lm_set_controller writes that layout once into
// the workspace and every controller launch copies it in with 16-byte loads.
struct MlpSmem {
  float w1t[kIn][kH], b1[kH], w2t[kH][kH], b2[kH], w3[kOut][kH], b3[kOut];
  float pad[2];  // 16-byte multiple
};
static_assert(sizeof(MlpSmem) % 16 == 0, "float4 staging");

__global__ void k_mlp_deploy(const float *__restrict__ theta, MlpSmem *__restrict__ m) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kH * kIn) m->w1t[i % kIn][i / kIn] = bf16r(theta[kW1 + i]);
  if (i < kH * kH) m->w2t[i % kH][i / kH] = bf16r(theta[kW2 + i]);
  if (i < kH) {
    m->b1[i] = bf16r(theta[kB1 + i]);
    m->b2[i] = bf16r(theta[kB2 + i]);
    m->w3[0][i] = bf16r(theta[kW3 + i]);
    m->w3[1][i] = bf16r(theta[kW3 + kH + i]);
  }
  if (i < kOut) m->b3[i] = bf16r(theta[kB3 + i]);
  if (i < 2) m->pad[i] = 0.f;
}

__device__ void stage_mlp(const MlpSmem *__restrict__ src, MlpSmem &m) {
  const float4 *s4 = reinterpret_cast<const float4 *>(src);
  float4 *d4 = reinterpret_cast<float4 *>(&m);
  constexpr int n = (int)(sizeof(MlpSmem) / 16);
  for (int i0 = threadIdx.x; i0 < n; i0 += 8 * blockDim.x) {  // eight 16-byte loads in flight
    float4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i0 + q * blockDim.x;
      if (i < n) v[q] = s4[i];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i0 + q * blockDim.x;
      if (i < n) d4[i] = v[q];
    }
  }
}

__device__ void mlp_infer_warp(const MlpSmem &m, const float *x, float &o0, float &o1) {
  const int lane = threadIdx.x & 31;
  float h1[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int j = lane + 32 * q;
    float z = m.b1[j];
#pragma unroll
    for (int k = 0; k < kIn; ++k) z += m.w1t[k][j] * x[k];
    h1[q] = gelu(z);
  }
  float p0 = 0.f, p1 = 0.f;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int j = lane + 32 * q;
    float z = m.b2[j];
#pragma unroll 8
    for (int k = 0; k < kH; ++k) {
      const float hk = __shfl_sync(0xffffffffu, h1[k >> 5], k & 31);
      z += m.w2t[k][j] * hk;
    }
    const float h2 = gelu(z);
    p0 += m.w3[0][j] * h2;
    p1 += m.w3[1][j] * h2;
  }
  o0 = warp_sum(p0) + m.b3[0];
  o1 = warp_sum(p1) + m.b3[1];
}

__device__ __forceinline__ float feat_clip(double v) {
  return v == v ? (float)fmin(40.0, fmax(-40.0, v)) : 0.f;
}
__device__ __forceinline__ double lg(double v) { return log10(fmax(v, 1e-300)); }

// The controller's 16 inputs for problem b (see spgo_lm_features), each finite and
// clipped to [-40, 40], computed by one warp: the twelve logarithms they take
// (FP64, which this GPU runs at a small fraction of its FP32 rate) are spread over
// the lanes, one per lane, and broadcast; every lane then holds all 16 features.
// log2(nu) comes out as log10(nu) / log10(2) rounded: nu is a power of two.
__device__ void lm_features_warp(const PlanView &pv, const LMState &s, int b, float *f) {
  const int lane = threadIdx.x & 31;
  const double nres = fmax(1.0, (double)pv.p_nres[b]);
  double arg = 1.0;
  switch (lane) {
    case 0: arg = fmax(s.cost, 1e-300); break;
    case 1: arg = nres; break;
    case 2: arg = fmax(s.cost0, 1e-300); break;
    case 3: arg = fmax(s.lam, 1e-300); break;
    case 4: arg = fmax(s.gnorm, 1e-300); break;
    case 5: arg = fmax(s.dmean, 1e-300); break;
    case 6: arg = fmax(s.dmax, 1e-300); break;
    case 7: arg = fmax(s.dmin, 1e-300); break;
    case 8: arg = fmax(s.cmean, 1e-300); break;
    case 9: arg = fmax(s.last_rel, 1e-12); break;
    case 10: arg = fmax(s.last_predrel, 1e-16); break;
    case 11: arg = fmax(s.nu, 1.0); break;
    default: break;
  }
  const double mine = log10(arg);
  double Lg[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) Lg[k] = __shfl_sync(0xffffffffu, mine, k);
  f[0] = feat_clip(Lg[0] - Lg[1]);
  f[1] = feat_clip(Lg[0] - Lg[2]);
  f[2] = feat_clip(fmin(2.0, fmax(-2.0, s.rho1)));
  f[3] = feat_clip(fmin(2.0, fmax(-2.0, s.rho2)));
  f[4] = feat_clip(fmin(2.0, fmax(-2.0, s.rho3)));
  f[5] = feat_clip(Lg[3]);
  f[6] = feat_clip(Lg[4] - 0.5 * Lg[5]);
  f[7] = feat_clip(Lg[5] - Lg[1]);
  f[8] = feat_clip(Lg[6] - Lg[7]);
  f[9] = feat_clip(Lg[8]);
  f[10] = feat_clip((double)s.iters / 30.0);
  f[11] = feat_clip((double)s.last_acc);
  f[12] = feat_clip(Lg[9]);
  f[13] = feat_clip(Lg[10]);
  f[14] = feat_clip(rint(Lg[11] / 0.30102999566398120));  // log2 of a power of two
  f[15] = feat_clip((double)s.rej_streak / 5.0);
}

// Runs once per LM iteration after the linearisation pass, before the step is
// solved: at the first iteration and after every accepted step (the state was
// just relinearised and the cost is current), the controller's
// proposal lambda * 10^out0 replaces the schedule's lambda when its logit out1 > 0
// (it predicts that deviating from the schedule gives the lower cost).  After a
// rejected step no relinearisation happens and the Nielsen increase stands: the
// fallback whenever a step fails the gain-ratio test.  A proposal lowers lambda by at
// most a factor 10^-min_dl (prm.ctl_min_log10, default -6: the network's own range).
// Tightening the bound does not make the network's choices safer: its proposals were
// learned with the full range, and cutting them short leaves lambda neither where the
// schedule nor where the network would put it.
__global__ void k_controller(PlanView pv, WorkView wv, const MlpSmem *Wd, float min_dl) {
  __shared__ MlpSmem m;
  stage_mlp(Wd, m);
  __syncthreads();
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= pv.B) return;
  LMState &s = wv.lm[b];
  if (s.status != 0 || !(s.iters == 0 || s.last_acc)) return;
  float x[kIn];
  lm_features_warp(pv, s, b, x);
  float o0, o1;
  mlp_infer_warp(m, x, o0, o1);
  if ((threadIdx.x & 31) == 0 && o1 > 0.f) {
    const double dl = fmin(3.0, fmax((double)min_dl, (double)o0));
    s.lam = fmin(1e12, fmax(1e-14, s.lam * exp10(dl)));
  }
}

__global__ void k_features(PlanView pv, WorkView wv, float *feat) {
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // warp per problem
  if (b >= pv.B) return;
  float x[kIn];
  lm_features_warp(pv, wv.lm[b], b, x);
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < kIn; ++k) feat[(size_t)b * kIn + k] = x[k];
}

// FP32 path of k_lm_stats: the maxima and minimum are exact in float and the sums
// run in double-float, on the FP32 pipes (FP64 runs at a small fraction of their
// rate on this GPU).  One CTA, blockDim a multiple of 32.
__device__ void lm_stats_f32(const PlanView &pv, const WorkView &wv, LMState &s, int b, int P, const float *A,
                             const float *g) {
  float gmx = 0.f, dmx = 0.f, dmn = INFINITY;
  df ds = df_make(0.f), cs = df_make(0.f);
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    gmx = fmaxf(gmx, fabsf(g[i]));
    const float d = A[(size_t)i * P + i];
    ds = ds + df_make(d);
    dmx = fmaxf(dmx, d);
    dmn = fminf(dmn, d);
  }
  const int l0 = pv.p_lm_off[b], lc = pv.p_lm_cnt[b];
  const float *C = reinterpret_cast<const float *>(wv.C) + l0;
  for (int i0 = threadIdx.x; i0 < lc; i0 += 8 * blockDim.x) {  // eight loads in flight
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i0 + q * blockDim.x;
      v[q] = i < lc ? C[i] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) cs = cs + df_make(v[q]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gmx = fmaxf(gmx, __shfl_xor_sync(0xffffffffu, gmx, o));
    dmx = fmaxf(dmx, __shfl_xor_sync(0xffffffffu, dmx, o));
    dmn = fminf(dmn, __shfl_xor_sync(0xffffffffu, dmn, o));
    ds = ds + df{__shfl_xor_sync(0xffffffffu, ds.h, o), __shfl_xor_sync(0xffffffffu, ds.l, o)};
    cs = cs + df{__shfl_xor_sync(0xffffffffu, cs.h, o), __shfl_xor_sync(0xffffffffu, cs.l, o)};
  }
  __shared__ float r7[32][7];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    r7[w][0] = gmx; r7[w][1] = ds.h; r7[w][2] = ds.l; r7[w][3] = dmx; r7[w][4] = dmn;
    r7[w][5] = cs.h; r7[w][6] = cs.l;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
      gmx = fmaxf(gmx, r7[k][0]);
      ds = ds + df{r7[k][1], r7[k][2]};
      dmx = fmaxf(dmx, r7[k][3]);
      dmn = fminf(dmn, r7[k][4]);
      cs = cs + df{r7[k][5], r7[k][6]};
    }
    s.gnorm = (double)gmx;
    s.dmean = P ? ((double)ds.h + (double)ds.l) / P : 0.0;
    s.dmax = (double)dmx;
    s.dmin = P ? (double)dmn : 0.0;
    s.cmean = lc ? ((double)cs.h + (double)cs.l) / lc : 0.0;
  }
}

// per-problem statistics of the fresh linearisation: max |g|, diag(A) mean/max/min, mean C
template <typename T>
__global__ void k_lm_stats(PlanView pv, WorkView wv) {
  __shared__ double red[4][32];
  const int b = blockIdx.x;
  LMState &s = wv.lm[b];
  if (s.status != 0 || !s.relin) return;
  const int P = 6 * pv.p_npose[b];
  const T *A = reinterpret_cast<const T *>(wv.A) + pv.p_S_off[b];
  const T *g = reinterpret_cast<const T *>(wv.g) + pv.p_param_off[b];
  if constexpr (std::is_same<T, float>::value) {
    lm_stats_f32(pv, wv, s, b, P, A, g);
    return;
  }
  double gmax = 0.0, dsum = 0.0, dmax = 0.0, dmin = 1e300, csum = 0.0;
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    gmax = fmax(gmax, fabs((double)g[i]));
    const double d = (double)A[(size_t)i * P + i];
    dsum += d;
    dmax = fmax(dmax, d);
    dmin = fmin(dmin, d);
  }
  const int l0 = pv.p_lm_off[b], lc = pv.p_lm_cnt[b];
  for (int i = threadIdx.x; i < lc; i += blockDim.x) csum += (double)reinterpret_cast<const T *>(wv.C)[l0 + i];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gmax = fmax(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
    dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
    csum += __shfl_xor_sync(0xffffffffu, csum, o);
  }
  __shared__ double r5[32][5];
  if (lane == 0) {
    r5[w][0] = gmax; r5[w][1] = dsum; r5[w][2] = dmax; r5[w][3] = dmin; r5[w][4] = csum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
      r5[0][0] = fmax(r5[0][0], r5[k][0]);
      r5[0][1] += r5[k][1];
      r5[0][2] = fmax(r5[0][2], r5[k][2]);
      r5[0][3] = fmin(r5[0][3], r5[k][3]);
      r5[0][4] += r5[k][4];
    }
    s.gnorm = r5[0][0];
    s.dmean = P ? r5[0][1] / P : 0.0;
    s.dmax = r5[0][2];
    s.dmin = P ? r5[0][3] : 0.0;
    s.cmean = lc ? r5[0][4] / lc : 0.0;
  }
  (void)red;
}

int launch_lm_stats(const PlanView &pv, const WorkView &wv, int f64, void *stream) {
  if (f64)
    k_lm_stats<double><<<pv.B, 128, 0, (cudaStream_t)stream>>>(pv, wv);
  else
    k_lm_stats<float><<<pv.B, 128, 0, (cudaStream_t)stream>>>(pv, wv);
  ++g_launches;
  return (int)cudaGetLastError();
}

int launch_controller(const PlanView &pv, const WorkView &wv, const Params &prm, const void *Wd, void *stream) {
  k_controller<<<grid_for(pv.B, 8), 256, 0, (cudaStream_t)stream>>>(pv, wv, reinterpret_cast<const MlpSmem *>(Wd),
                                                                    prm.ctl_min_log10);
  ++g_launches;
  return (int)cudaGetLastError();
}

int launch_features(const PlanView &pv, const WorkView &wv, float *feat, void *stream) {
  k_features<<<grid_for(pv.B, 4), 128, 0, (cudaStream_t)stream>>>(pv, wv, feat);
  ++g_launches;
  return (int)cudaGetLastError();
}

int launch_mlp_deploy(const float *theta, void *dst, void *stream) {
  k_mlp_deploy<<<grid_for(kH * kH, 256), 256, 0, (cudaStream_t)stream>>>(theta, reinterpret_cast<MlpSmem *>(dst));
  ++g_launches;
  return (int)cudaGetLastError();
}
size_t mlp_deployed_bytes() { return sizeof(MlpSmem); }

}  // namespace spgo

using namespace spgo;

extern "C" int spgo_mlp_forward(const float *d_params, const float *d_X, int32_t n, float *d_out, float *d_cache,
                                void *stream) {
  if (!d_params || !d_X || !d_out || n < 0) return SPGO_ERR_INVALID_ARG;
  if (n == 0) return SPGO_OK;
  cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpTrain));
  k_mlp_fwd<<<grid_for(n, kSamples), kMlpThreads, sizeof(MlpTrain), (cudaStream_t)stream>>>(d_params, d_X, n, d_out,
                                                                                          d_cache);
  ++g_launches;
  return cudaGetLastError() == cudaSuccess ? SPGO_OK : SPGO_ERR_CUDA;
}

extern "C" int spgo_mlp_grad(const float *d_params, const float *d_X, const float *d_T, int32_t n, float *d_grad,
                             float *d_loss, float *d_out, float *d_cache, void *stream) {
  if (!d_params || !d_X || !d_T || !d_grad || !d_loss || !d_out || !d_cache || n <= 0) return SPGO_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  cudaMemsetAsync(d_loss, 0, sizeof(float), st);
  const int ctas = grid_for(n, kSamples);
  cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpTrain));
  k_mlp_grad<<<ctas, kMlpThreads, sizeof(MlpTrain), st>>>(d_params, d_X, d_T, n, d_out, d_cache, d_grad, d_loss);
  ++g_launches;
  if (ctas > 1) {
    k_mlp_sum<<<grid_for(kParams, 32), 256, 0, st>>>(d_cache, ctas - 1, d_grad);
    ++g_launches;
  }
  return cudaGetLastError() == cudaSuccess ? SPGO_OK : SPGO_ERR_CUDA;
}

extern "C" int spgo_mlp_adam(float *d_params, const float *d_grad, float *d_m, float *d_v, int32_t step, float lr,
                             void *stream) {
  if (!d_params || !d_grad || !d_m || !d_v || step < 1) return SPGO_ERR_INVALID_ARG;
  k_mlp_adam<<<grid_for(kParams, 256), 256, 0, (cudaStream_t)stream>>>(d_params, d_grad, d_m, d_v, step, lr);
  ++g_launches;
  return cudaGetLastError() == cudaSuccess ? SPGO_OK : SPGO_ERR_CUDA;
}
