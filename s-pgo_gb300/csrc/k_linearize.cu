// Pose chain and the cost pass; the Jacobian pass is k_jacobian.cu.
//
// Replaces S-PGO's computeGlobalPoses (src/Optimization/Solver_cuda.cu:440-493),
// LevenbergMarquardt (Solver_cuda.cu:49-310, helpers src/Optimization/LMutils.cu:538-628)
// and compute_B_C_inv (Solver_cuda.cu:322-345).
//
// Factorisation used instead of the reference's dense J_T (4O x 6N) rows: the
// Jacobian of observation o (landmark anchored in frame a, seen in frame n)
// with respect to incremental pose i in [lo, hi) = [min(a,n), max(a,n)) is
//     J_{o,i} = s_o * K_o * Ad_i,   s_o = +1 (n > a) or -1 (n < a),
// where K_o = [ (X - x) x u_k , u_k ] (2x6, u = dpi/dt R_n^T) is the derivative
// with respect to a world-frame twist about an origin x, and Ad_i maps frame i's
// perturbation (psi, rho) to that world twist.  So one observation costs O(1)
// instead of O(window), and
//   * the pose-pose blocks come from per-(lo, hi) accumulators
//     M_{lo,hi} = sum K^T K, m_{lo,hi} = sum s K^T r  (pairs, 27 values),
//     combined later by 2-D prefix sums (k_system.cu);
//   * the pose-depth column of landmark l is B_l(i) = Ad_i^T b_l(i),
//     b_l(i) = sum over its observations covering i of s K^T j_alpha, written into
//     the chunk's landmark-contiguous slab for the Schur GEMM.
// Pair accumulators use the left centre of frame lo as origin and the slab
// uses the landmark's anchor centre, so no large world coordinates enter FP32.
#include "kernels.cuh"
#include "frames.cuh"
#include "dfloat.cuh"

#include <algorithm>
#include <type_traits>

namespace spgo {

// ---- global poses: G[0] = I, G[k+1] = G[k] inv(T_k); right camera G T_r_to_l ----
// FP64 path.  One CTA per problem: an inclusive scan of the 3x4 products in shared memory, three
// threads (rows) per frame, blockDim / 3 frames per pass with the running prefix carried between
// passes (the reference walks the chain with one thread, Solver_cuda.cu:472-491).  Bound by the
// scan's FP64 instructions, 64 cycles each for a quarter of an SM: a row's product takes 12, where
// a lane per frame took 36 and 32 frames shared one quarter of the SM (100 poses: 57 us, 17.3
// us so; 10 poses: 18.6 and 8.5 us).
constexpr int kChainFrames = 128;

// row r of frame f, G its 3x4 pose
__device__ __forceinline__ void write_frame_row(const WorkView &wv, size_t f, int r, const double *G, const double *Trl) {
  double Gr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) Gr[j] = G[0] * Trl[j] + G[1] * Trl[4 + j] + G[2] * Trl[8 + j];
  Gr[3] += G[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const size_t q = f * 18 + 3 * r + j;
    wv.fr_Rd[q] = G[j];
    wv.fr_Rd[q + 9] = Gr[j];
    const float gl = (float)G[j], gr = (float)Gr[j];
    wv.fr_Rf[q] = gl;
    wv.fr_Rf[q + 9] = gr;
    wv.fr_Rl[q] = (float)(G[j] - (double)gl);
    wv.fr_Rl[q + 9] = (float)(Gr[j] - (double)gr);
  }
  const size_t q = f * 6 + r;
  wv.fr_c[q] = G[3];
  wv.fr_c[q + 3] = Gr[3];
  const float hl = (float)G[3], hr = (float)Gr[3];
  wv.fr_ch[q] = hl;
  wv.fr_ch[q + 3] = hr;
  wv.fr_cl[q] = (float)(G[3] - (double)hl);
  wv.fr_cl[q + 3] = (float)(Gr[3] - (double)hr);
}

// row p of a product P M of 3x4 poses
__device__ __forceinline__ void compose_row(const double *p, const double *M, double *o) {
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j] = p[0] * M[j] + p[1] * M[4 + j] + p[2] * M[8 + j];
  o[3] += p[3];
}

__global__ void __launch_bounds__(3 * kChainFrames) k_chain(PlanView pv, WorkView wv, const double *__restrict__ poses,
                                                            int gate) {
  grid_enter();
  const int b = blockIdx.x;
  if (!problem_active(wv.lm, b, gate)) return;
  __shared__ double buf[2][kChainFrames][12];
  __shared__ double last[12];
  const int N = pv.p_npose[b], fo = pv.p_frame_off[b], po = pv.p_pose_off[b];
  const int nf = blockDim.x / 3, f = threadIdx.x / 3, r = threadIdx.x % 3;
  const double *Trl = pv.p_Trl + 12 * b;
  if (f == 0) {
    const double I[4] = {r == 0 ? 1.0 : 0.0, r == 1 ? 1.0 : 0.0, r == 2 ? 1.0 : 0.0, 0.0};
    write_frame_row(wv, (size_t)fo, r, I, Trl);
  }
  for (int s = 0; s < N; s += nf) {
    const int k = s + f, n = min(nf, N - s);
    double m[4] = {0.0, 0.0, 0.0, 0.0};
    if (k < N) {  // row r of inv(T_k)
      const double *T = poses + 12 * (size_t)(po + k);
#pragma unroll
      for (int j = 0; j < 3; ++j) m[j] = T[4 * j + r];
      m[3] = -(m[0] * T[3] + m[1] * T[7] + m[2] * T[11]);
    }
    int cur = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) buf[0][f][4 * r + j] = m[j];
    __syncthreads();
    // inclusive scan: M_k <- M_0 M_1 ... M_k (earlier factors on the left)
    for (int d = 1; d < n; d <<= 1) {
      if (f >= d) {
        double p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = buf[cur][f - d][4 * r + j];
        compose_row(p, buf[cur][f], m);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) buf[cur ^ 1][f][4 * r + j] = m[j];
      cur ^= 1;
      __syncthreads();
    }
    if (s > 0) {
      double p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) p[j] = last[4 * r + j];
      compose_row(p, buf[cur][f], m);
    }
    if (k < N) write_frame_row(wv, (size_t)(fo + k + 1), r, m, Trl);
    __syncthreads();  // (every product with the carried prefix is formed)
    if (f == nf - 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) last[4 * r + j] = m[j];
    }
    __syncthreads();
  }
}

template <typename T>
struct CostSmem {
  T X[SPGO_CHUNK][3];      // anchor point, world axes, relative to the anchor centre
  float Xl[SPGO_CHUNK][3]; // FP32 path: low words of X as a double-float
  double cost[8];
};

// Dynamic shared memory: CostSmem, then (FP32 path) dc [W][6] float x 2 = the host's left
// centre minus every window frame's camera centres, hi and lo (W = max_nb + 1 frames).
template <typename T>
__host__ __device__ inline size_t cost_smem(int max_nb, size_t *dc) {
  *dc = (sizeof(CostSmem<T>) + 15) & ~(size_t)15;
  return *dc + ((size_t)max_nb + 1) * 12 * sizeof(float);
}

// ---- cost pass -----------------------------------------------------------------
// One CTA per chunk of <= 32 landmarks.  Phase A: per-landmark anchor point.  Phase B: one
// thread per observation: both cameras' residuals and the robust cost; on the FP32 path in
// double-float (FP64-accurate cost for the gain ratio), stored as FP32 per observation with
// the camera-frame points, and per landmark the anchor points, for the Jacobian and residual
// passes at this state.  The Jacobian pass (k_jacobian.cu) always follows a cost pass at the
// same state (the first one after a reset, or the accepted candidate's): forming residuals
// from pixel-sized FP32 quantities instead (~3e-5 px rounding) would move the optimum by
// ~1e-5 m.
// Register cap (FP32): 64, a latency-bound stream over the observations that runs in small
// CTAs and gains from the extra resident warps (16 instead of 12 64-thread CTAs per SM).
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 1) k_cost(PlanView pv, WorkView wv, Params prm,
                                                   const double *__restrict__ alpha_state, int gate) {
  grid_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int2 cb = pv.ch_sched[blockIdx.x];
  const int c = cb.x, b = cb.y;
  if (!problem_active(wv.lm, b, gate)) return;
  const int tid = threadIdx.x;
  const int f0 = pv.ch_f0[c], nb = pv.ch_nb[c], lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
  const int fo = pv.p_frame_off[b];
  const float *intr = pv.p_intr + 8 * b;
  const T fxs[2] = {(T)intr[0], (T)intr[4]}, fys[2] = {(T)intr[1], (T)intr[5]};
  const T cxs[2] = {(T)intr[2], (T)intr[6]}, cys[2] = {(T)intr[3], (T)intr[7]};
  CostSmem<T> &sm = *reinterpret_cast<CostSmem<T> *>(smem_raw);
  size_t off_dc;
  cost_smem<T>(pv.max_nb, &off_dc);
  float *dch = reinterpret_cast<float *>(smem_raw + off_dc);  // [W][6] hi, then [W][6] lo
  float *dcl = dch + (size_t)(pv.max_nb + 1) * 6;
  const int64_t ob = pv.lm_obs[lm0], oe = pv.lm_obs[lm0 + cnt];
  const int host = pv.lm_host[lm0];  // every landmark of the chunk has this host
  // the cost pass of the state after a reset writes the state's half of the stores, a
  // candidate's the other half
  const int sel = wv.lm[b].res_sel;
  const size_t half = (size_t)(gate != GATE_FIRST ? 1 - sel : sel);
  float *res_buf = wv.res + half * (size_t)pv.O * 4;
  float *tcam_buf = wv.tcam ? wv.tcam + half * (size_t)pv.O * 6 : nullptr;  // mixed path: camera-frame points
  float *xanc_buf = wv.xanc ? wv.xanc + half * (size_t)pv.L * 8 : nullptr;   // and anchor points
  // each thread's observation record is loaded one loop pass ahead (the first one here, so
  // its DRAM latency overlaps phase A), so a pass does not open with a round trip to DRAM
  int nx_slot = 0, nx_n = 0;
  float4 nx_z = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load_obs = [&](int64_t o) {
    if (o < oe) {
      nx_slot = pv.obs_slot[o];
      nx_n = pv.obs_frame[o];
      nx_z = reinterpret_cast<const float4 *>(pv.obs_uv)[o];
    }
  };
  load_obs(ob + tid);

  // phase A
  if (tid < cnt) {
    const int li = lm0 + tid;
    const T alpha = (T)alpha_state[pv.lm_user[li]];
    const T ua = (T)pv.lm_uv[2 * li], va = (T)pv.lm_uv[2 * li + 1];
    const T *Ra = FramesT<T>::R(wv, fo + host, 0);
    const Vec3<T> ta = v3<T>((ua - cxs[0]) / fxs[0] / alpha, (va - cys[0]) / fys[0] / alpha, T(1) / alpha);
    Vec3<T> X = mul(Ra, ta);
    if constexpr (std::is_same<T, float>::value) {
      // the same point as a double-float, for the residuals
      const df al = df_from_double(alpha_state[pv.lm_user[li]]);
      const df t3[3] = {df_sub(pv.lm_uv[2 * li], intr[2]) / df_make(intr[0]) / al,
                        df_sub(pv.lm_uv[2 * li + 1], intr[3]) / df_make(intr[1]) / al, df_make(1.f) / al};
      const float *Rh = wv.fr_Rf + (size_t)(fo + host) * 18, *Rl = wv.fr_Rl + (size_t)(fo + host) * 18;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const df v = df{Rh[3 * k], Rl[3 * k]} * t3[0] + df{Rh[3 * k + 1], Rl[3 * k + 1]} * t3[1] +
                     df{Rh[3 * k + 2], Rl[3 * k + 2]} * t3[2];
        sm.Xl[tid][k] = v.l;
        if (k == 0) X.x = v.h;
        if (k == 1) X.y = v.h;
        if (k == 2) X.z = v.h;
      }
    }
    sm.X[tid][0] = X.x; sm.X[tid][1] = X.y; sm.X[tid][2] = X.z;
    if (xanc_buf) {  // kept for the Jacobian and residual passes at this state, with d / d alpha
      float4 *xa = reinterpret_cast<float4 *>(xanc_buf + (size_t)li * 8);
      xa[0] = make_float4((float)X.x, (float)X.y, (float)X.z, (float)(-X.x / alpha));
      xa[1] = make_float4((float)(-X.y / alpha), (float)(-X.z / alpha), 0.f, 0.f);
    }
  }
  if constexpr (std::is_same<T, float>::value) {
    // the host's left centre minus every window frame's camera centres, as double-floats
    const int fh = fo + host;
    for (int idx = tid; idx < (nb + 1) * 6; idx += blockDim.x) {
      const int f = idx / 6, cam = (idx / 3) & 1, k = idx % 3;
      const size_t fn = (size_t)(fo + f0 + f);
      df d = df_sub(wv.fr_ch[(size_t)fh * 6 + k], wv.fr_ch[fn * 6 + cam * 3 + k]);
      d = d + df_make(wv.fr_cl[(size_t)fh * 6 + k] - wv.fr_cl[fn * 6 + cam * 3 + k]);
      dch[idx] = d.h;
      dcl[idx] = d.l;
    }
  }
  __syncthreads();

  // phase B
  const T lscale = (T)prm.loss_scale;
  T cost_t = T(0);  // a thread sums a handful of terms; the FP64 reduction starts at the warp
  for (int64_t o = ob + tid; o < oe; o += blockDim.x) {
    const int slot = nx_slot, n = nx_n;
    const float4 z = nx_z;
    load_obs(o + blockDim.x);  // the next pass's record, in flight during this one
    float4 rstore = make_float4(0.f, 0.f, 0.f, 0.f);  // residuals to keep
    float tstore[6];                                    // and the camera-frame points
    const Vec3<T> X = v3<T>(sm.X[slot][0], sm.X[slot][1], sm.X[slot][2]);
    const int fn = fo + n;
    const T boost = (prm.near_boost && abs(n - host) < 2) ? T(16) : T(1);
#pragma unroll
    for (int cam = 0; cam < 2; ++cam) {
      const T *Rn = FramesT<T>::R(wv, fn, cam);
      const T fx = fxs[cam], fy = fys[cam];
      T r0, r1;
      if constexpr (std::is_same<T, float>::value) {
        // residual in double-float: X + (c_a - c_n), rotated, then projected as
        // r = ((z - c) t_z - f t_x) / t_z (the small numerator carries the
        // precision, the division is plain FP32)
        const float *Rl = wv.fr_Rl + (size_t)fn * 18 + cam * 9;
        const int fw = n - f0;
        df Xc[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
          Xc[k] = df{sm.X[slot][k], sm.Xl[slot][k]} + df{dch[fw * 6 + cam * 3 + k], dcl[fw * 6 + cam * 3 + k]};
        df tt[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
          tt[k] = df_dot3(Rn[k], Rl[k], Rn[3 + k], Rl[3 + k], Rn[6 + k], Rl[6 + k], Xc[0], Xc[1], Xc[2]);
        const df nu = df_sub(cam ? z.z : z.x, cxs[cam]) * tt[2] - tt[0] * fx;
        const df nv = df_sub(cam ? z.w : z.y, cys[cam]) * tt[2] - tt[1] * fy;
        const float itz = 1.f / tt[2].h;
        r0 = (nu.h + nu.l) * itz;
        r1 = (nv.h + nv.l) * itz;
        tstore[3 * cam] = tt[0].h;
        tstore[3 * cam + 1] = tt[1].h;
        tstore[3 * cam + 2] = tt[2].h;
        if (cam) {
          rstore.z = r0;
          rstore.w = r1;
        } else {
          rstore.x = r0;
          rstore.y = r1;
        }
      } else {
        const Vec3<T> d = FramesT<T>::rel(wv, fo + host, 0, fn, cam);
        const Vec3<T> t = mulT(Rn, v3<T>(X.x + d.x, X.y + d.y, X.z + d.z));
        const T izr = T(1) / t.z;
        r0 = (T)(cam ? z.z : z.x) - (fx * t.x * izr + cxs[cam]);
        r1 = (T)(cam ? z.w : z.y) - (fy * t.y * izr + cys[cam]);
      }
      T rho;
      (void)robust<T>(prm.loss, lscale, r0 * r0 + r1 * r1, rho);
      cost_t += T(0.5) * boost * rho;
    }
    if constexpr (std::is_same<T, float>::value) {
      reinterpret_cast<float4 *>(res_buf)[o] = rstore;
      if (tcam_buf) {  // 24 bytes at 8-byte alignment
        float2 *tp = reinterpret_cast<float2 *>(tcam_buf + (size_t)o * 6);
        tp[0] = make_float2(tstore[0], tstore[1]);
        tp[1] = make_float2(tstore[2], tstore[3]);
        tp[2] = make_float2(tstore[4], tstore[5]);
      }
    }
  }
  // cost: warp sums, then one FP64 atomic per CTA
  const double cost = warp_sum((double)cost_t);
  if ((tid & 31) == 0) sm.cost[tid >> 5] = cost;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sm.cost[w];
    if (t != 0.0) atomicAdd(wv.cost_acc + b, t);
  }
}

// ---- the FP32 path's pose chain in double-float ----
// The same scan with 3x4 products in double-float (~48 significant bits, the
// precision of the FP32 path's frame tables: fr_Rf + fr_Rl, fr_ch + fr_cl), on the
// FP32 pipes instead of FP64 (which runs at a small fraction of their rate on
// this GPU).  Writes only the tables the FP32 kernels read.
// row p of a product P M
__device__ __forceinline__ void compose_row_df(const df *p, const df *M, df *o) {
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j] = df_dot3(p[0].h, p[0].l, p[1].h, p[1].l, p[2].h, p[2].l, M[j], M[4 + j], M[8 + j]);
  o[3] = o[3] + p[3];
}

// row r of frame f, G its 3x4 pose (also the left centre as FP64, h + l, which the refinement's
// FP64 sums read)
__device__ __forceinline__ void write_frame_row_df(const WorkView &wv, size_t f, int r, const df *G, const df *Trl) {
  df Gr[4];
  compose_row_df(G, Trl, Gr);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const size_t q = f * 18 + 3 * r + j;
    wv.fr_Rf[q] = G[j].h;
    wv.fr_Rf[q + 9] = Gr[j].h;
    wv.fr_Rl[q] = G[j].l;
    wv.fr_Rl[q + 9] = Gr[j].l;
  }
  const size_t q = f * 6 + r;
  wv.fr_ch[q] = G[3].h;
  wv.fr_ch[q + 3] = Gr[3].h;
  wv.fr_cl[q] = G[3].l;
  wv.fr_cl[q + 3] = Gr[3].l;
  wv.fr_c[q] = (double)G[3].h + (double)G[3].l;
}

// As k_chain, one CTA per problem, three threads (rows) per frame, up to kChainDfFrames frames a
// pass (in place: two barriers per step of the scan).  Bound by the scan's latency: 10 poses 8.3 us
// and 500 poses 36 us with a lane per frame, 5.3 and 24 us so (a row is a third of a frame).
constexpr int kChainDfFrames = 256;

__global__ void __launch_bounds__(3 * kChainDfFrames) k_chain_df(PlanView pv, WorkView wv,
                                                                 const double *__restrict__ poses, int gate) {
  grid_enter();
  const int b = blockIdx.x;
  if (!problem_active(wv.lm, b, gate)) return;
  __shared__ df buf[kChainDfFrames][12];
  __shared__ df Trl[12], last[12];
  const int N = pv.p_npose[b], fo = pv.p_frame_off[b], po = pv.p_pose_off[b];
  const int nf = blockDim.x / 3, f = threadIdx.x / 3, r = threadIdx.x % 3;
  if (threadIdx.x < 12) Trl[threadIdx.x] = df_from_double(pv.p_Trl[12 * b + threadIdx.x]);
  for (int s = 0; s < N; s += nf) {
    const int k = s + f, n = min(nf, N - s);
    if (k < N) {  // row r of the pose, for its inverse [R^T, -R^T t]
      const double *T = poses + 12 * (size_t)(po + k) + 4 * r;
#pragma unroll
      for (int j = 0; j < 4; ++j) buf[f][4 * r + j] = df_from_double(T[j]);
    }
    __syncthreads();
    if (s == 0 && f == 0) {
      const df I[4] = {df_make(r == 0 ? 1.f : 0.f), df_make(r == 1 ? 1.f : 0.f), df_make(r == 2 ? 1.f : 0.f), df_make(0.f)};
      write_frame_row_df(wv, (size_t)fo, r, I, Trl);
    }
    df m[4];
    {
      const df *T = buf[f];
#pragma unroll
      for (int j = 0; j < 3; ++j) m[j] = T[4 * j + r];
      m[3] = -df_dot3(m[0].h, m[0].l, m[1].h, m[1].l, m[2].h, m[2].l, T[3], T[7], T[11]);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) buf[f][4 * r + j] = m[j];
    __syncthreads();
    // inclusive scan: M_k <- M_0 M_1 ... M_k (earlier factors on the left)
    for (int d = 1; d < n; d <<= 1) {
      const bool on = f >= d && f < n;
      if (on) {
        df p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = buf[f - d][4 * r + j];
        compose_row_df(p, buf[f], m);
      }
      __syncthreads();
      if (on) {
#pragma unroll
        for (int j = 0; j < 4; ++j) buf[f][4 * r + j] = m[j];
      }
      __syncthreads();
    }
    if (s > 0 && k < N) {
      df p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) p[j] = last[4 * r + j];
      compose_row_df(p, buf[f], m);
    }
    if (k < N) write_frame_row_df(wv, (size_t)(fo + k + 1), r, m, Trl);
    if (s + nf >= N) break;
    __syncthreads();  // (every product with the carried prefix is formed)
    if (f == nf - 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) last[4 * r + j] = m[j];
    }
    __syncthreads();
  }
}

int launch_chain(const PlanView &pv, const WorkView &wv, const double *poses, int gate, int f64, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const int warps = std::max(1, (pv.max_P / 6 + 31) / 32);  // of frames, three threads each
  if (f64)
    launch(k_chain, pv.B, 96 * std::min(kChainFrames / 32, warps), 0, st, pv, wv, poses, gate);
  else
    launch(k_chain_df, pv.B, 96 * std::min(kChainDfFrames / 32, warps), 0, st, pv, wv, poses, gate);
  ++g_launches;
  return (int)cudaGetLastError();
}

// Latency-bound: short CTAs, many per SM, where there are enough chunks to fill it (64 windows of
// 3731 chunks: 10.76 ms with 64 threads, 10.93 with 128, 11.33 with 256); twice the threads while
// all CTAs are resident at once, eight to an SM, and the longest chunk is what takes the time
// (GN step of 22 chunks: 104 us with 64, 92 with 128 or 256; LM step of 672: 1276, 1235, 1236).
constexpr int kCostThreads = 64, kCostThreadsFew = 128, kCostFew = 8 * kSmCount;

template <typename T>
int launch_linearize(const PlanView &pv, const WorkView &wv, const Params &prm, const double *alpha,
                     int cost_only, int gate, void *stream) {
  if (pv.n_chunks == 0) return 0;
  if (!cost_only) return launch_jacobian<T>(pv, wv, prm, alpha, gate, stream);
  const int nt = prm.cost_block > 0 ? prm.cost_block : pv.n_chunks <= kCostFew ? kCostThreadsFew : kCostThreads;
  size_t dc;
  launch(k_cost<T>, pv.n_chunks, nt, cost_smem<T>(pv.max_nb, &dc), (cudaStream_t)stream, pv, wv, prm, alpha, gate);
  ++g_launches;
  return (int)cudaGetLastError();
}

template int launch_linearize<float>(const PlanView &, const WorkView &, const Params &, const double *, int, int, void *);
template int launch_linearize<double>(const PlanView &, const WorkView &, const Params &, const double *, int, int, void *);

}  // namespace spgo
