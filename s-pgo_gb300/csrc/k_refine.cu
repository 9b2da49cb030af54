// Iterative refinement of the mixed path's LM step.
//
// The FP32 reduced system (pose Hessian from FP32 pair sums, tensor-core Schur
// complement, FP32 Cholesky) gives a step whose error, on the ill-conditioned
// systems of the circle scenes, reaches 1e-3 relative.  Such steps do not change
// where LM converges, but they change where it is after a fixed iteration budget,
// and the accepted cost then differs from the FP64 solver's by far more than the
// 1e-6 the solvers are compared at.  The cause is the accumulation of the normal
// equations (the sums over observations and landmarks, which cancel in S = A -
// W D^-1 W^T and in the gradient), not the FP32 Jacobian itself.
//
// So the FP32 system only preconditions.  Each refinement step forms the
// residual of the whole damped system
//   r_p = J_p^T W (r - J x) - lam diag(A) x_p,   r_a = J_a^T W (r - J x) - (lam C + eps) x_a
// from the FP32 Jacobian rows, recomputed per observation as the linearisation formed
// them (jac_rows.cuh), with every product J e exact (two-product) and every sum in double-float / FP64, then applies the FP32
// system's inverse: x_p += S^-1 (r_p - W D^-1 r_a), x_a += D^-1 (r_a - W^T dx_p).
// The first residual pass also sums the accurate gradient J^T W r, which the
// predicted decrease of the gain ratio uses.
//
//   k_pair_twists     per problem: the world twist of every pose pair's poses,
//                     W(lo, hi) = sum_{i in [lo, hi)} Ad_i x_i about c_lo (FP64 sums,
//                     stored FP32), so J_o x_p = s_o K_o W(lo, hi) per observation
//   k_resid_pass      per landmark chunk: the inverse-depth step of the chunk's
//                     landmarks, then one thread per observation: e = r - J x and its
//                     dual s K^T W e (pair records, FP64 atomics per run of equal
//                     target frame) and j_a^T W e (per landmark, FP64); then
//                     t = D^-1 r_a and W t into the pose right-hand side
//   k_resid_solve     per problem: the pair records reduced to per-pose vectors
//                     (FP64), the right-hand side, and the solve with the stored FP32
//                     factor; systems too wide for one CTA take the same reduction
//                     from k_rs_sums_large, k_rs_scan_large and k_rs_rhs_large (spread
//                     over the GPU) and the multi-CTA substitutions of k_chol_large.cu
//   k_backsub_refined per chunk: the last inverse-depth correction, the candidate
//                     inverse depths and their share of the predicted decrease
//
// Replaces nothing in the reference, whose GPU step is an FP32 Gauss-Newton step
// solved once (src/Optimization/Solver_cuda.cu:594-782, linear_solvers.cu:195-218).
#include <algorithm>

#include "kernels.cuh"
#include "frames.cuh"
#include "jac_rows.cuh"
#include "chol_subst.cuh"

namespace spgo {

// a problem takes (the next step of) the refinement: running, its step not failed, and
// its refinement not yet converged (outer_tol)
__device__ __forceinline__ bool refine_active(const WorkView &wv, int b) {
  return problem_active(wv.lm, b, GATE_RUNNING) && !wv.lm[b].fail && !wv.lm[b].ref_done;
}

// ---- pose-pair twists -------------------------------------------------------
// Ad_i x_i = [R_i psi_i ; (c_i - o) x R_i psi_i + R_i rho_i] about origin o (the
// convention of the pose blocks, k_system.cu).  With the prefix sums
// Om(k) = sum_{i<k} R_i psi_i and V(k) = sum_{i<k} c_i x R_i psi_i + R_i rho_i,
// W(lo, hi) = [Om(hi) - Om(lo) ; V(hi) - V(lo) - c_lo x (Om(hi) - Om(lo))].
// Only differences of the prefix sums enter, so a CTA takes a slice of consecutive lo's and
// sums over their own poses and the D after them; the slices are as long as still gives every SM a
// CTA (kTwSlice at most), so that a batch's windows are one CTA each and few windows or a long
// trajectory spread over the GPU (500 poses: 141 us on one SM's FP64 pipe, 12 us spread out).
// Bound by FP64 instructions, 64 cycles each for a quarter of an SM, so every phase spreads over
// all four (64 windows of up to 32 poses, two slices each: 11.5 us with a thread per pose and a
// slice per window, 7.5 us so).
constexpr int kTwThreads = 192;  // (six warps: one per component in the scan)
constexpr int kTwSlice = 32;

__global__ void __launch_bounds__(kTwThreads) k_pair_twists(PlanView pv, WorkView wv, int slice) {
  grid_enter();
  __shared__ double tw_s[(kTwSlice + SPGO_MAX_WINDOW + 1) * 6];
  const int b = blockIdx.x, l0 = slice * blockIdx.y;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b], fo = pv.p_frame_off[b], po = pv.p_param_off[b];
  if (l0 >= N || !refine_active(wv, b)) return;
  const int n = min(N - l0, slice + D);  // the slice's poses and the D after them
  for (int t = threadIdx.x; t < 3 * n; t += blockDim.x) {  // thread per (pose, row)
    const int i = t / 3, r = t % 3;
    const float *Rh = wv.fr_Rf + (size_t)(fo + l0 + i) * 18 + 3 * r, *Rl = wv.fr_Rl + (size_t)(fo + l0 + i) * 18 + 3 * r;
    const double *x = wv.delta + po + 6 * (l0 + i);
    double R[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) R[k] = (double)Rh[k] + (double)Rl[k];
    tw_s[(size_t)(i + 1) * 6 + r] = R[0] * x[0] + R[1] * x[1] + R[2] * x[2];
    tw_s[(size_t)(i + 1) * 6 + 3 + r] = R[0] * x[3] + R[1] * x[4] + R[2] * x[5];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * n; t += blockDim.x) {
    const int i = t / 3, k = t % 3, k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
    const double *c = wv.fr_c + (size_t)(fo + l0 + i) * 6;
    double *o = tw_s + (size_t)(i + 1) * 6;
    o[3 + k] += c[k1] * o[k2] - c[k2] * o[k1];
  }
  if (threadIdx.x < 6) tw_s[threadIdx.x] = 0.0;
  __syncthreads();
  for (int k = threadIdx.x >> 5; k < 6; k += kTwThreads / 32) {  // warp scan per component
    const int lane = threadIdx.x & 31;
    double carry = 0.0;
    for (int s = 0; s < n; s += 32) {
      double v = s + lane < n ? tw_s[(s + lane + 1) * 6 + k] : 0.0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
      }
      v += carry;
      if (s + lane < n) tw_s[(s + lane + 1) * 6 + k] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  float *out = wv.twist + ((size_t)pv.p_pair_off[b] + (size_t)l0 * D) * 6;
  for (int t = threadIdx.x; t < min(slice, N - l0) * D; t += blockDim.x) {
    const int lo = t / D, hi = lo + t % D + 1;  // relative to l0
    if (l0 + hi > N) continue;
    const double *c = wv.fr_c + (size_t)(fo + l0 + lo) * 6;
    double dw[3], dv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dw[k] = tw_s[hi * 6 + k] - tw_s[lo * 6 + k];
      dv[k] = tw_s[hi * 6 + 3 + k] - tw_s[lo * 6 + 3 + k];
    }
    float *o = out + (size_t)t * 6;
    o[0] = (float)dw[0];
    o[1] = (float)dw[1];
    o[2] = (float)dw[2];
    o[3] = (float)(dv[0] - (c[1] * dw[2] - c[2] * dw[1]));
    o[4] = (float)(dv[1] - (c[2] * dw[0] - c[0] * dw[2]));
    o[5] = (float)(dv[2] - (c[0] * dw[1] - c[1] * dw[0]));
  }
}

int launch_pair_twists(const PlanView &pv, const WorkView &wv, void *stream) {
  const int nmax = pv.max_P / 6;
  int slice = kTwSlice;
  while (slice > 8 && (long long)pv.B * ((nmax + slice - 1) / slice) < kSmCount) slice /= 2;
  launch(k_pair_twists, dim3(pv.B, (nmax + slice - 1) / slice), kTwThreads, 0, (cudaStream_t)stream, pv, wv, slice);
  ++g_launches;
  return (int)cudaGetLastError();
}

// ---- residual pass ------------------------------------------------------------
constexpr int kRpThreads = 128;
constexpr int kRpWarps = kRpThreads / 32;
constexpr int kRpPitch = 33;

struct RefSmem {
  float X[SPGO_CHUNK][3];   // anchor point, world axes, relative to the anchor centre
  float dX[SPGO_CHUNK][3];  // dX / d alpha
  float da[SPGO_CHUNK];     // inverse-depth step (FP32 copy for the residuals)
  __align__(16) float t[SPGO_CHUNK];  // D^-1 r_a
  int a[SPGO_CHUNK];
  float dlh[kRpWarps][SPGO_CHUNK];  // j_a^T W e, per warp, double-float (h, l)
  float dll[kRpWarps][SPGO_CHUNK];
  int key[kRpWarps][32];
  float bt[2][SPGO_CHUNK];  // warps 0 and 1: partial W^T x_p over their slab row blocks
};

// dynamic shared memory (W = window frames): the pair origins' offsets [W][3] and the per-warp
// staging [warps][6][33] of the pair duals (double-float) | the window's rotations [W][18]
// (both cameras) | the pair twists [W][6]
struct RpLayout {
  size_t xpo, stage, rw, tws, total;
  __host__ __device__ explicit RpLayout(int max_nb) {
    const size_t W = (size_t)max_nb + 1;
    xpo = 0;
    stage = xpo + W * 3 * sizeof(df);
    rw = stage + (size_t)kRpWarps * 6 * kRpPitch * sizeof(df);
    tws = rw + W * 18 * sizeof(float);
    total = tws + W * 6 * sizeof(float);
  }
};

// The accurate gradient itself (J^T W r, pose and inverse-depth parts) comes from the
// linearisation, which sums it exactly (k_jacobian.cu, k_system.cu); each pass here
// forms only the duals of e.
template <bool FIRST>
__global__ void __launch_bounds__(kRpThreads, 8) k_resid_pass(PlanView pv, WorkView wv, Params prm,
                                                           const double *__restrict__ alpha_state) {
  grid_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ RefSmem sm;
  const int2 cb = pv.ch_sched[blockIdx.x];
  const int c = cb.x, b = cb.y;
  if (!refine_active(wv, b)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f0 = pv.ch_f0[c], nb = pv.ch_nb[c], lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
  const int fo = pv.p_frame_off[b], po = pv.p_param_off[b];
  const float *intr = pv.p_intr + 8 * b;
  const float fxs[2] = {intr[0], intr[4]}, fys[2] = {intr[1], intr[5]};
  const double lam = wv.lm[b].lam;
  const float eps = prm.eps;
  {
    // the chunk's observation records (slot, frame, residuals) towards L2 while the
    // prologue runs: one prefetch per 128-byte line
    const int64_t ob0 = pv.lm_obs[lm0], oe0 = pv.lm_obs[lm0 + cnt];
    const float *res0 = wv.res + (size_t)wv.lm[b].res_sel * (size_t)pv.O * 4;
    const int nres = (int)(((oe0 - ob0) * 16 + 127) / 128), nfr = (int)(((oe0 - ob0) * 4 + 127) / 128);
    for (int k = tid; k < nres + nfr; k += blockDim.x) {
      const void *a = k < nres ? (const void *)(reinterpret_cast<const char *>(res0 + 4 * ob0) + 128 * k)
                               : (const void *)(reinterpret_cast<const char *>(pv.obs_frame + ob0) + 128 * (k - nres));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
    }
  }
  const RpLayout lay(pv.max_nb);
  float *Rw = reinterpret_cast<float *>(smem_raw + lay.rw);
  df *xpo = reinterpret_cast<df *>(smem_raw + lay.xpo);
  float *tws = reinterpret_cast<float *>(smem_raw + lay.tws);
  df *stage = reinterpret_cast<df *>(smem_raw + lay.stage);
  const int D = pv.p_pair_D[b];
  const float *slab = reinterpret_cast<const float *>(wv.slab) + pv.ch_slab[c];
  const float *Cv = reinterpret_cast<const float *>(wv.C);
  const int rows = 6 * nb;

  if (warp < 2) {
    // inverse-depth step: first pass x_a = D^-1 (g_a - W^T x_p) from the FP32 system,
    // later x_a += t - D^-1 W^T dx_p (the previous pass's t and pose correction); warps
    // 0 and 1 take alternate 32-row blocks of the slab for W^T x_p
    const double *v = (FIRST ? wv.delta : wv.ddelta) + po + 6 * f0;
    float s0 = 0.f, s1 = 0.f;
    for (int rb = 32 * warp; rb < rows; rb += 64) {
      const float dv = rb + lane < rows ? (float)v[rb + lane] : 0.f;
      const float *sr = slab + (size_t)rb * SPGO_CHUNK + lane;
      const int nr = min(32, rows - rb);
      float q[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) q[k] = k < nr ? sr[(size_t)k * SPGO_CHUNK] : 0.f;
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        s0 += q[k] * __shfl_sync(0xffffffffu, dv, k);
        s1 += q[k + 1] * __shfl_sync(0xffffffffu, dv, k + 1);
      }
    }
    sm.bt[warp][lane] = s0 + s1;
  }
  if (warp == 0) {
    // the chunk's anchor points, as the cost pass at this state formed them (the same
    // points the linearisation used)
    if (lane < cnt) {
      const int li = lm0 + lane;
      const float4 *xa = reinterpret_cast<const float4 *>(wv.xanc + ((size_t)wv.lm[b].res_sel * pv.L + li) * 8);
      const float4 x0 = xa[0], x1 = xa[1];
      sm.X[lane][0] = x0.x;
      sm.X[lane][1] = x0.y;
      sm.X[lane][2] = x0.z;
      sm.dX[lane][0] = x0.w;
      sm.dX[lane][1] = x1.x;
      sm.dX[lane][2] = x1.y;
      sm.a[lane] = pv.lm_host[li];
    }
#pragma unroll
    for (int w = 0; w < kRpWarps; ++w) sm.dlh[w][lane] = sm.dll[w][lane] = 0.f;
  }
  if (warp < 2) named_sync(1, 64);  // both partial sums written
  if (warp == 1) {
    if (lane < cnt) {
      const int li = lm0 + lane;
      const float C = Cv[li];
      const float Dd = C * (float)(1.0 + lam) + eps;
      const float s = sm.bt[0][lane] + sm.bt[1][lane];
      double da;
      if (FIRST)
        da = (double)((reinterpret_cast<const float *>(wv.ga)[li] - s) / Dd);
      else
        da = wv.dal[li] + (double)(wv.tl[li] - s / Dd);
      wv.dal[li] = da;
      sm.da[lane] = (float)da;
    }
  } else if (warp >= 2) {
    // the window's rotations, and per window frame n the offset c_a - c_n of the pair
    // origin (n < a) and the twist of the pair (a, n)
    const int ah = pv.lm_host[lm0], fh = fo + ah;
    for (int idx = tid - 64; idx < (nb + 1) * 18; idx += blockDim.x - 64)
      Rw[idx] = wv.fr_Rf[(size_t)(fo + f0) * 18 + idx];
    for (int f = tid - 64; f < nb + 1; f += blockDim.x - 64) {
      const int n = f0 + f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        df d = df_make(0.f);
        if (n < ah) {
          const size_t x = (size_t)fh * 6 + k, y = (size_t)(fo + n) * 6 + k;
          d = df_sub(wv.fr_ch[x], wv.fr_ch[y]) + df_make(wv.fr_cl[x] - wv.fr_cl[y]);
        }
        xpo[3 * f + k] = d;
      }
      const int lo = min(ah, n), hi = max(ah, n);
      float t6v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (hi > lo && hi - lo <= D) {  // a pair that observations of this chunk can form
        const float *tw = wv.twist + ((size_t)pv.p_pair_off[b] + (size_t)lo * D + (hi - lo - 1)) * 6;
#pragma unroll
        for (int k = 0; k < 6; ++k) t6v[k] = tw[k];
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) tws[6 * f + k] = t6v[k];
    }
  }
  __syncthreads();

  const int64_t ob = pv.lm_obs[lm0], oe = pv.lm_obs[lm0 + cnt];
  const float lscale = prm.loss_scale;
  // residuals at the linearisation point: the state's half of the residual store
  const float *res_buf = wv.res + (size_t)wv.lm[b].res_sel * (size_t)pv.O * 4;
  const float *tcam_buf = wv.tcam + (size_t)wv.lm[b].res_sel * (size_t)pv.O * 6;
  for (int64_t base = ob + (tid & ~31); base < oe; base += blockDim.x) {
    const int64_t o = base + lane;
    // this observation's weighted rows W and its weighted linearised residuals
    // w r - W (p + dX x_a), p the displacement of its point by the pose step so far; with g = sum W e (exact
    // four-product sums) its duals are dX . g (landmark) and s [Xp x g; g] (pose pair): the
    // structure and the rounded rows of the Jacobian pass
    using M = Num<float>;
    df g[3], gx[3], vle = df_make(0.f);
#pragma unroll
    for (int k = 0; k < 3; ++k) g[k] = gx[k] = df_make(0.f);
    int key = -1, slot = -1;
    if (o < oe) {
      slot = pv.obs_slot[o];
      const int n = pv.obs_frame[o];
      const float4 rl = reinterpret_cast<const float4 *>(res_buf)[o];
      const int a = sm.a[slot];
      const int fw = n - f0;
      const float boost = (prm.near_boost && abs(n - a) < 2) ? 16.f : 1.f;
      const float da = sm.da[slot];
      // point relative to the pair origin (the left centre of frame min(a, n)), the
      // pair's twist (zero without a pose term)
      df Xp[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) Xp[k] = M::shift(sm.X[slot][k], xpo[3 * fw + k]);
      const float sgn = n > a ? 1.f : -1.f;
      const float *tw = tws + 6 * fw;
      const Vec3<float> om = v3<float>(tw[0], tw[1], tw[2]);
      const Vec3<float> ox = cross(om, v3<float>(Xp[0].h, Xp[1].h, Xp[2].h));
      const float p[3] = {sgn * (tw[3] + ox.x), sgn * (tw[4] + ox.y), sgn * (tw[5] + ox.z)};  // by the poses
      const float2 *tp = reinterpret_cast<const float2 *>(tcam_buf + (size_t)o * 6);
      const float2 t01 = tp[0], t23 = tp[1], t45 = tp[2];
      float W[4][3], e[4];
      const float *Rn = Rw + fw * 18;
      weighted_rows(prm.loss, lscale, boost, fxs[0], fys[0], Rn, t01.x, t01.y, t23.x, rl.x, rl.y, W, e);
      weighted_rows(prm.loss, lscale, boost, fxs[1], fys[1], Rn + 9, t23.y, t45.x, t45.y, rl.z, rl.w, W + 2, e + 2);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        // the inverse-depth entry W . dX cancels (dX runs along the anchor ray, the rows are
        // nearly across it): compensated, so that the residual belongs to the same J.  (The rest
        // in FP32: with p and all four products in double-float the refined step was no nearer
        // to the FP64 one, median 6.9e-7 against 7.2e-7 of the step over 256 windows.)
        const float ja = M::round(M::dot(M::of(W[q][0]), M::of(W[q][1]), M::of(W[q][2]), sm.dX[slot][0],
                                         sm.dX[slot][1], sm.dX[slot][2]));
        e[q] -= ja * da + (W[q][0] * p[0] + W[q][1] * p[1] + W[q][2] * p[2]);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) g[k] = M::sum4(W[0][k], e[0], W[1][k], e[1], W[2][k], e[2], W[3][k], e[3]);
      vle = M::dot(g[0], g[1], g[2], sm.dX[slot][0], sm.dX[slot][1], sm.dX[slot][2]);
      if (n != a) {
        key = n;
#pragma unroll
        for (int k = 0; k < 3; ++k) g[k] = M::scale(sgn, g[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k)
          gx[k] = M::cross(Xp[(k + 1) % 3], g[(k + 2) % 3], Xp[(k + 2) % 3], g[(k + 1) % 3]);
      }
    }
    {
      // the warp's own landmark accumulators: lanes sharing a landmark (different
      // frames) add in rounds of their rank among those peers, no atomics
      const unsigned peers = __match_any_sync(0xffffffffu, slot);
      const int rank = __popc(peers & ((1u << lane) - 1u));
      for (int r = 0; __any_sync(0xffffffffu, slot >= 0 && rank >= r); ++r) {
        if (slot >= 0 && rank == r) {
          df_acc a;
          a.h = sm.dlh[warp][slot];
          a.l = sm.dll[warp][slot];
          a.add(vle.h, vle.l);
          sm.dlh[warp][slot] = a.h;
          sm.dll[warp][slot] = a.l;
        }
        __syncwarp();
      }
    }
    // stage the six pair duals; then 24 lanes, one per (dual, 8-observation segment),
    // each sum their segment's runs of equal target frame and add every run to its
    // pair record (FP64; a run crossing a segment boundary arrives in two parts)
    df *st = stage + (size_t)warp * 6 * kRpPitch;
    int *keys = sm.key[warp];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      st[k * kRpPitch + lane] = gx[k];
      st[(3 + k) * kRpPitch + lane] = g[k];
    }
    keys[lane] = key;
    __syncwarp();
    if (__any_sync(0xffffffffu, key >= 0) && lane < 24) {
      const int host_a = sm.a[0];
      const int v = lane % 6, i0 = (lane / 6) * 8;
      const df *col = st + v * kRpPitch;
      double *rec0 = wv.pdual + (size_t)pv.p_pair_off[b] * 6 + v;
      auto emit = [&](int n, const df_acc &a) {
        const int lo = min(host_a, n), hi = max(host_a, n);
        atomicAdd(rec0 + ((size_t)lo * D + (hi - lo - 1)) * 6, df_acc_value(a));
      };
      df_acc acc;
      int cur = keys[i0];
#pragma unroll
      for (int i = i0; i < i0 + 8; ++i) {
        const int k = keys[i];
        if (k != cur) {
          if (cur >= 0) emit(cur, acc);
          acc = df_acc();
          cur = k;
        }
        M::acc(acc, col[i]);
      }
      if (cur >= 0) emit(cur, acc);
    }
    __syncwarp();
  }
  __syncthreads();
  // landmark residuals r_a = j_a^T W e - (lam C + eps) x_a, t = D^-1 r_a
  if (tid < cnt) {
    const int li = lm0 + tid;
    const float C = Cv[li];
    const float Dd = C * (float)(1.0 + lam) + eps;
    df_acc acc;
#pragma unroll
    for (int w = 0; w < kRpWarps; ++w) acc.add(sm.dlh[w][tid], sm.dll[w][tid]);
    const double dsum = df_acc_value(acc);
    const double ra = dsum - (lam * (double)C + (double)eps) * wv.dal[li];  // summed in FP64
    const float t = (float)ra / Dd;  // (t is an FP32 preconditioner term: no FP64 division)
    sm.t[tid] = t;
    wv.tl[li] = t;
  } else if (tid < SPGO_CHUNK) {
    sm.t[tid] = 0.f;
  }
  __syncthreads();
  // W t into the pose right-hand side: thread per slab row, its 32 landmark entries read
  // as eight 16-byte loads (the chunk's slab starts 16-byte aligned, rows are 128 bytes)
  const float4 *t4 = reinterpret_cast<const float4 *>(sm.t);
  for (int r = tid; r < rows; r += blockDim.x) {
    const float4 *sr = reinterpret_cast<const float4 *>(slab + (size_t)r * SPGO_CHUNK);
    float4 x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = sr[q];
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 t = t4[q];
      v0 += x[q].x * t.x + x[q].y * t.y;
      v1 += x[q].z * t.z + x[q].w * t.w;
    }
    const float v = v0 + v1;
    if (v != 0.f) atomicAdd(wv.rhsB + po + 6 * f0 + r, v);
  }
}

int launch_resid_pass(const PlanView &pv, const WorkView &wv, const Params &prm, const double *alpha, int first,
                      void *stream) {
  if (pv.n_chunks == 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t sm = RpLayout(pv.max_nb).total;
  if (first)
    launch(k_resid_pass<true>, pv.n_chunks, kRpThreads, sm, st, pv, wv, prm, alpha);
  else
    launch(k_resid_pass<false>, pv.n_chunks, kRpThreads, sm, st, pv, wv, prm, alpha);
  ++g_launches;
  return (int)cudaGetLastError();
}

// ---- pair records -> per-pose right-hand side, and the solve ---------------------
// A record (lo, hi) holds m = [m_w ; m_v] about c_lo; about the world origin it is
// n = [m_w + c_lo x m_v ; m_v].  Pose i collects every record with lo <= i < hi,
// moved to c_i: sum n_w - c_i x sum m_v.  With diff(k) = sum_{lo = k} n - sum_{hi = k} n
// that sum is the prefix sum of diff up to i.  Then r(i) = [R_i^T (.)_w ; R_i^T (.)_v].
// The row sums (fixed lo) re-centre linearly: sum_hi n = sum_hi m_w + c_lo x sum_hi m_v;
// the column sums (fixed hi) take c_lo x m_v per record.  One thread per (row or column,
// component), no atomics.  Bound by FP64 instructions (64 cycles of a quarter SM each) and the
// substitutions' chain: 64 windows of up to 32 poses 29.2 us with a serial prefix, a thread per
// pose in the right-hand side and warps that ran through rows and columns alike, 19.7 us so.
constexpr int kRsThreads = 256;

// shared memory: centres, row and column sums | cb | y | the packed factor
// (as stored by the factorisation)
__host__ __device__ inline size_t rs_layout(int max_Ps, int max_N, size_t *off_cb, size_t *off_y, size_t *off_L) {
  auto up = [](size_t x) { return (x + 15) & ~(size_t)15; };
  size_t o = up((size_t)(max_N + 1) * 15 * sizeof(double));  // centres [N+1][3], rows, columns [N+1][6]
  *off_cb = o;
  o = up(o + (size_t)max_Ps * sizeof(int));
  *off_y = o;
  o = up(o + (size_t)max_Ps * sizeof(float));
  *off_L = o;
  return up(o + ((size_t)max_Ps * (max_Ps + 1) / 2 + kPanel) * sizeof(float));  // (+ kPanel: chol_substitute)
}

size_t resid_solve_smem(int max_P_small, int max_N) {
  size_t a, b, c;
  return rs_layout(max_P_small, max_N, &a, &b, &c);
}

// 16-byte asynchronous global -> shared copies (no registers held while in flight)
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

__global__ void __launch_bounds__(kRsThreads) k_resid_solve(PlanView pv, WorkView wv, float outer_tol) {
  grid_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int b = pv.fs_prob[blockIdx.x];
  if (!refine_active(wv, b)) return;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b], P = 6 * N;
  const int fo = pv.p_frame_off[b], po = pv.p_param_off[b];
  const int tid = threadIdx.x, nt = blockDim.x;
  size_t o_cb, o_y, o_L;
  rs_layout(pv.max_P_small, pv.max_P / 6, &o_cb, &o_y, &o_L);
  const bool small = P <= pv.max_P_small;
  if (!small && wv.lg_red) return;  // wide problems: the grid-wide kernels below
  const size_t npk = (size_t)P * (P + 1) / 2;
  float *Lm = reinterpret_cast<float *>(smem_raw + o_L);
  if (small) {
    // the stored factor (contiguous, 16-byte aligned: S offsets are multiples
    // of 36 floats) start copying now and land while the pair duals are reduced
    const float *fac = wv.facs + pv.p_S_off[b];
    const size_t n = npk, n4 = n / 4;
    for (size_t k = tid; k < n4; k += nt) cp_async16(Lm + 4 * k, fac + 4 * k);
    for (size_t k = 4 * n4 + tid; k < n; k += nt) Lm[k] = fac[k];
  }
  double *cs = reinterpret_cast<double *>(smem_raw);  // [N + 1][3] left camera centres
  double *rowm = cs + (size_t)(N + 1) * 3;            // [N + 1][6]: sum over hi of m(lo, hi)
  double *colm = rowm + (size_t)(N + 1) * 6;          // [N + 1][6]: sum over lo of n(lo, hi)
  for (int k = tid; k < N * 3; k += nt)
    cs[k] = wv.fr_c[(size_t)(fo + k / 3) * 6 + k % 3];
  __syncthreads();
  double *recs = wv.pdual + (size_t)pv.p_pair_off[b] * 6;
  // Three kinds of sums, each from a warp's first lane on, so that no warp runs through two kinds:
  // rows (all components), columns' m_v, and columns' m_w with the records moved from c_lo.
  const int w_row = (6 * N + 31) / 32, w_col = (3 * N + 31) / 32, lane = tid & 31;
  for (int w = tid >> 5; w < w_row + 2 * w_col; w += nt >> 5) {
    if (w < w_row) {
      const int t = 32 * w + lane, lo = t / 6, k = t % 6;
      if (lo >= N) continue;
      const double *r = recs + (size_t)lo * D * 6 + k;
      const int nd = min(D, N - lo);
      double acc = 0.0;
#pragma unroll 8
      for (int d = 0; d < nd; ++d) acc += r[(size_t)d * 6];
      rowm[lo * 6 + k] = acc;
      continue;
    }
    const bool moved = w >= w_row + w_col;
    const int t = 32 * (w - w_row - (moved ? w_col : 0)) + lane, hi = t / 3 + 1, k = t % 3;
    if (hi > N) continue;
    double acc = 0.0;
    if (moved) {
      const int k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
#pragma unroll 4
      for (int lo = max(0, hi - D); lo < hi; ++lo) {
        const double *r = recs + ((size_t)lo * D + (hi - lo - 1)) * 6;
        acc = fma(-cs[lo * 3 + k2], r[3 + k1], fma(cs[lo * 3 + k1], r[3 + k2], acc + r[k]));
      }
      colm[hi * 6 + k] = acc;
    } else {
#pragma unroll 8
      for (int lo = max(0, hi - D); lo < hi; ++lo) acc += recs[((size_t)lo * D + (hi - lo - 1)) * 6 + 3 + k];
      colm[hi * 6 + 3 + k] = acc;
    }
  }
  if (tid < 6) colm[tid] = 0.0;  // no record ends at pose 0
  __syncthreads();
  for (size_t k = tid; k < (size_t)N * D * 6; k += nt) recs[k] = 0.0;  // cleared for the next pass
  // pose i's term: its row sums moved from c_i, less the column sums of the records ending there
  for (int t = tid; t < 6 * N; t += nt) {
    const int i = t / 6, k = t % 6, k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
    const double *m = rowm + i * 6, *c = cs + i * 3;
    double v = m[k] - colm[t];
    if (k < 3) v = fma(-c[k2], m[3 + k1], fma(c[k1], m[3 + k2], v));
    colm[t] = v;  // (read and written by this thread alone)
  }
  __syncthreads();
  // its prefix over the poses, a warp per component: the sum of the records covering pose i
  for (int k = tid >> 5; k < 6; k += nt >> 5) {
    double carry = 0.0;
    for (int s = 0; s < N; s += 32) {
      double v = s + lane < N ? colm[(s + lane) * 6 + k] : 0.0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
      }
      v += carry;
      if (s + lane < N) rowm[(s + lane) * 6 + k] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  for (int t = tid; t < 3 * N; t += nt) {  // m_w about c_i
    const int i = t / 3, k = t % 3, k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
    const double *c = cs + i * 3;
    double *S = rowm + i * 6;
    S[k] -= c[k1] * S[3 + k2] - c[k2] * S[3 + k1];
  }
  __syncthreads();
  float *y = reinterpret_cast<float *>(smem_raw + o_y);
  const double lam = wv.lm[b].lam;
  const float *A = reinterpret_cast<const float *>(wv.A) + pv.p_S_off[b];
  for (int p = tid; p < P; p += nt) {  // R_i^T of both halves, a thread per unknown
    const int i = p / 6, k = p % 6, r = k < 3 ? k : k - 3;
    const float *Rh = wv.fr_Rf + (size_t)(fo + i) * 18 + r, *Rl = wv.fr_Rl + (size_t)(fo + i) * 18 + r;
    const double *S = rowm + i * 6 + (k < 3 ? 0 : 3);
    double out = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) out += ((double)Rh[3 * q] + (double)Rl[3 * q]) * S[q];
    const double x = wv.delta[po + p];
    const double rhs = out - lam * (double)A[(size_t)p * P + p] * x - (double)wv.rhsB[po + p];
    wv.rhsB[po + p] = 0.f;
    if (small)
      y[p] = (float)rhs;
    else
      reinterpret_cast<float *>(wv.lg_y)[po + p] = (float)rhs;
  }
  if (!small) return;  // the multi-CTA substitutions (k_chol_large.cu) follow
  int *cb = reinterpret_cast<int *>(smem_raw + o_cb);
  for (int k = tid; k < P; k += nt) cb[k] = k * P - (k * (k + 1)) / 2;
  cp_async_wait_all();
  __syncthreads();
  chol_substitute<float>(Lm, cb, y, nullptr, P);
  __shared__ unsigned mx_dx, mx_x;  // largest |correction|, |step| (float bits: non-negative floats order as ints)
  if (tid == 0) mx_dx = mx_x = 0u;
  __syncthreads();
  for (int k = tid; k < P; k += nt) {
    const double dx = (double)y[k];
    const double x = wv.delta[po + k] + dx;
    wv.delta[po + k] = x;
    wv.ddelta[po + k] = dx;
    if (outer_tol > 0.f) {
      atomicMax(&mx_dx, __float_as_uint(fabsf((float)dx)));
      atomicMax(&mx_x, __float_as_uint(fabsf((float)x)));
    }
  }
  __syncthreads();
  // converged: the correction is a small fraction of the step, further steps are skipped
  if (tid == 0 && outer_tol > 0.f && __uint_as_float(mx_dx) <= outer_tol * __uint_as_float(mx_x))
    wv.lm[b].ref_done = 1;
}

// ---- the same reduction for wide problems, spread over the GPU ----------------------
// One CTA per problem puts a wide problem's FP64 pair sums on one SM (GB300 issues FP64
// at 1/64 of its FP32 rate): for P = 3000 that was 267 us per refinement step.  Here
//   k_rs_sums_large   four lanes per (pose, component): the row sums (over hi) and the
//                     column sums (over lo, moved to c_lo) of the pair duals, into lg_red
//   k_rs_scan_large   one CTA: the rows' prefix over the poses, as segment sums, an
//                     exclusive scan of the segments and a second walk of each segment
//   k_rs_rhs_large    thread per unknown: the world-to-pose transform, the right-hand side
//                     into lg_y for the multi-CTA substitutions; clears the pair duals
// (100 poses with windows of 41: 20.1 and 8.3 us with a thread per sum and per pose, 7.8 and 5.1 us so)
// The per-pose values are those of k_resid_solve; only the prefix is summed in another
// order (FP64, segments of ~N / 42 poses).
// (FP64-bound: small CTAs spread the sums over the SMs, and the centres come as FP64)
__global__ void __launch_bounds__(64) k_rs_sums_large(PlanView pv, WorkView wv, int b) {
  grid_enter();
  if (!refine_active(wv, b)) return;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b], fo = pv.p_frame_off[b];
  // row sums of all components, then columns' m_v, then columns' m_w, each kind from a warp's
  // first lane on
  const int wr = (6 * N + 7) / 8, wc = (3 * N + 7) / 8, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int kind = w < wr ? 0 : w < wr + wc ? 1 : 2, part = threadIdx.x & 3;
  const int g = 8 * (w - (kind == 0 ? 0 : kind == 1 ? wr : wr + wc)) + ((threadIdx.x & 31) >> 2);
  double *rowm = wv.lg_red + ((size_t)pv.p_pose_off[b] + b) * 12, *colm = rowm + (size_t)(N + 1) * 6;
  const double *recs = wv.pdual + (size_t)pv.p_pair_off[b] * 6;
  auto cen = [&](int f, int k) { return wv.fr_c[(size_t)(fo + f) * 6 + k]; };
  double acc = 0.0;
  double *out = nullptr;
  if (kind == 0) {
    const int lo = g / 6, k = g % 6;
    if (lo < N) {
      const double *r = recs + (size_t)lo * D * 6 + k;
      const int nd = min(D, N - lo);
#pragma unroll 4
      for (int d = part; d < nd; d += 4) acc += r[(size_t)d * 6];
      out = rowm + lo * 6 + k;
      if (lo == 0 && part == 0) colm[k] = 0.0;  // no record ends at pose 0
    }
  } else {
    const int hi = g / 3 + 1, k = g % 3;
    if (hi <= N) {
      if (kind == 1) {
#pragma unroll 4
        for (int lo = max(0, hi - D) + part; lo < hi; lo += 4) acc += recs[((size_t)lo * D + (hi - lo - 1)) * 6 + 3 + k];
        out = colm + hi * 6 + 3 + k;
      } else {
        const int k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
#pragma unroll 4
        for (int lo = max(0, hi - D) + part; lo < hi; lo += 4) {
          const double *r = recs + ((size_t)lo * D + (hi - lo - 1)) * 6;
          acc = fma(-cen(lo, k2), r[3 + k1], fma(cen(lo, k1), r[3 + k2], acc + r[k]));
        }
        out = colm + hi * 6 + k;
      }
    }
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  if (out && part == 0) *out = acc;
}

constexpr int kScanSegs = 42;  // segments per component: 6 x 42 = 252 of the 256 threads

// dynamic shared memory: the per-pose terms [N][6] (FP64)
__global__ void __launch_bounds__(256) k_rs_scan_large(PlanView pv, WorkView wv, int b) {
  grid_enter();
  if (!refine_active(wv, b)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *val = reinterpret_cast<double *>(smem_raw);
  __shared__ double seg[6][kScanSegs];
  const int N = pv.p_npose[b], fo = pv.p_frame_off[b], tid = threadIdx.x;
  double *rowm = wv.lg_red + ((size_t)pv.p_pose_off[b] + b) * 12;
  const double *colm = rowm + (size_t)(N + 1) * 6;
  // pose i's term: its row sums moved from c_i (the origin of the records starting there)
  // less the column sums of the records ending there
  for (int t = tid; t < 6 * N; t += blockDim.x) {
    const int i = t / 6, k = t % 6, k1 = (k + 1) % 3, k2 = (k + 2) % 3;
    const double *m = rowm + i * 6;
    double nrow = m[k];
    if (k < 3) {
      const double c1 = wv.fr_c[(size_t)(fo + i) * 6 + k1], c2 = wv.fr_c[(size_t)(fo + i) * 6 + k2];
      nrow += c1 * m[3 + k2] - c2 * m[3 + k1];
    }
    val[t] = nrow - colm[t];
  }
  __syncthreads();
  const int len = (N + kScanSegs - 1) / kScanSegs;
  const int k = tid / kScanSegs, s = tid % kScanSegs, i0 = s * len, i1 = min(N, i0 + len);
  if (tid < 6 * kScanSegs) {
    double acc = 0.0;
    for (int i = i0; i < i1; ++i) acc += val[i * 6 + k];
    seg[k][s] = acc;
  }
  __syncthreads();
  if (tid < 6) {  // exclusive scan of the segment sums
    double acc = 0.0;
    for (int q = 0; q < kScanSegs; ++q) {
      const double v = seg[tid][q];
      seg[tid][q] = acc;
      acc += v;
    }
  }
  __syncthreads();
  if (tid < 6 * kScanSegs) {
    double acc = seg[k][s];
    for (int i = i0; i < i1; ++i) {
      acc += val[i * 6 + k];
      rowm[i * 6 + k] = acc;  // the sum of the records covering pose i
    }
  }
}

__global__ void __launch_bounds__(64) k_rs_rhs_large(PlanView pv, WorkView wv, int b) {
  grid_enter();
  if (!refine_active(wv, b)) return;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b], P = 6 * N;
  const int fo = pv.p_frame_off[b], po = pv.p_param_off[b];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const double *rowm = wv.lg_red + ((size_t)pv.p_pose_off[b] + b) * 12;
  // the pair duals are summed: cleared for the next pass
  double *recs = wv.pdual + (size_t)pv.p_pair_off[b] * 6;
  for (size_t q = t; q < (size_t)N * D * 6; q += (size_t)gridDim.x * blockDim.x) recs[q] = 0.0;
  if (t >= P) return;
  const int i = t / 6, k = t % 6, r = k < 3 ? k : k - 3;
  const float *A = reinterpret_cast<const float *>(wv.A) + pv.p_S_off[b];
  const float *Rh = wv.fr_Rf + (size_t)(fo + i) * 18 + r, *Rl = wv.fr_Rl + (size_t)(fo + i) * 18 + r;
  const double *c = wv.fr_c + (size_t)(fo + i) * 6, *S = rowm + i * 6;
  double m[3];  // m_w about c_i, or m_v
  if (k < 3) {
    m[0] = S[0] - (c[1] * S[5] - c[2] * S[4]);
    m[1] = S[1] - (c[2] * S[3] - c[0] * S[5]);
    m[2] = S[2] - (c[0] * S[4] - c[1] * S[3]);
  } else {
#pragma unroll
    for (int q = 0; q < 3; ++q) m[q] = S[3 + q];
  }
  double out = 0.0;
#pragma unroll
  for (int q = 0; q < 3; ++q) out += ((double)Rh[3 * q] + (double)Rl[3 * q]) * m[q];
  const double x = wv.delta[po + t];
  const double rhs = out - wv.lm[b].lam * (double)A[(size_t)t * P + t] * x - (double)wv.rhsB[po + t];
  wv.rhsB[po + t] = 0.f;
  reinterpret_cast<float *>(wv.lg_y)[po + t] = (float)rhs;
}

int launch_resid_reduce_large(const PlanView &pv, const WorkView &wv, int b, int N, void *stream) {
  if (!wv.lg_red) return 0;  // (the FP64 path has no refinement)
  cudaStream_t st = (cudaStream_t)stream;
  launch(k_rs_sums_large, ((6 * N + 7) / 8 + 2 * ((3 * N + 7) / 8) + 1) / 2, 64, 0, st, pv, wv, b);  // (a warp per 8 sums)
  const size_t sm = (size_t)N * 6 * sizeof(double);
  cudaFuncSetAttribute(k_rs_scan_large, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  launch(k_rs_scan_large, 1, 256, sm, st, pv, wv, b);
  launch(k_rs_rhs_large, std::max((6 * N + 63) / 64, 96), 64, 0, st, pv, wv, b);  // (the clearing wants the CTAs)
  g_launches += 3;
  return (int)cudaGetLastError();
}

int launch_resid_solve(const PlanView &pv, const WorkView &wv, const Params &prm, int first, void *stream) {
  (void)first;  // every pass reduces the same duals of e
  const size_t sm = resid_solve_smem(pv.max_P_small, pv.max_P / 6);
  cudaStream_t st = (cudaStream_t)stream;
  cudaFuncSetAttribute(k_resid_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  launch(k_resid_solve, pv.B, kRsThreads, sm, st, pv, wv, prm.outer_steps > 1 ? prm.outer_tol : 0.f);
  ++g_launches;
  return (int)cudaGetLastError();
}

// ---- the last inverse-depth correction, candidate and predicted decrease -------------
// one warp per chunk, lane = landmark slot: x_a += t - D^-1 W^T dx_p, alpha' =
// clamp(alpha + x_a), pred += x_a (g_a + (lam C + eps) x_a) with the accurate g_a
__global__ void k_backsub_refined(PlanView pv, WorkView wv, Params prm, const double *alpha, double *alpha_out) {
  grid_enter();
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int slot = threadIdx.x & 31;
  if (c >= pv.n_chunks) return;
  const int b = pv.ch_prob[c];
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  const bool failed = wv.lm[b].fail != 0;
  const int f0 = pv.ch_f0[c], nb = pv.ch_nb[c], lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
  const int po = pv.p_param_off[b];
  const float *slab = reinterpret_cast<const float *>(wv.slab) + pv.ch_slab[c];
  const double *dl = wv.ddelta + po + 6 * f0;
  const int rows = 6 * nb;
  float s0 = 0.f, s1 = 0.f;
  if (!failed) {
    for (int rb = 0; rb < rows; rb += 32) {
      const float dv = rb + slot < rows ? (float)dl[rb + slot] : 0.f;
      const float *sr = slab + (size_t)rb * SPGO_CHUNK + slot;
      const int nr = min(32, rows - rb);
      float v[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) v[k] = k < nr ? sr[(size_t)k * SPGO_CHUNK] : 0.f;
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        s0 += v[k] * __shfl_sync(0xffffffffu, dv, k);
        s1 += v[k + 1] * __shfl_sync(0xffffffffu, dv, k + 1);
      }
    }
  }
  double pred = 0.0;
  if (slot < cnt && !failed) {
    const int li = lm0 + slot;
    const double lam = wv.lm[b].lam;
    const float C = reinterpret_cast<const float *>(wv.C)[li];
    const float Dd = C * (float)(1.0 + lam) + prm.eps;
    const double da = wv.dal[li] + (double)(wv.tl[li] - (s0 + s1) / Dd);
    pred = da * (wv.gaacc[li] + (lam * (double)C + (double)prm.eps) * da);
    const int u = pv.lm_user[li];
    alpha_out[u] = fmin(fmax(alpha[u] + da, (double)prm.alpha_min), (double)prm.alpha_max);
  }
  pred = warp_sum(pred);
  if (slot == 0 && pred != 0.0) atomicAdd(wv.pred_acc + b, pred);
}

int launch_backsub_refined(const PlanView &pv, const WorkView &wv, const Params &prm, const double *alpha,
                           double *alpha_out, void *stream) {
  if (pv.n_chunks == 0) return 0;
  launch(k_backsub_refined, grid_for(pv.n_chunks, 4), 128, 0, (cudaStream_t)stream, pv, wv, prm, alpha, alpha_out);
  ++g_launches;
  return (int)cudaGetLastError();
}

}  // namespace spgo
