// Reduced camera system: pose-pose Hessian from the (lo, hi) pair accumulators,
// the landmark Schur complement W D^-1 W^T, and S = A + damping - W D^-1 W^T.
//
// Replaces the reference's dense cuBLAS products A = J_T^T J_T, g_T = J_T^T r,
// B C^-1 B^T, B C^-1 g_a and the element-wise subtraction
// (src/Optimization/Solver_cuda.cu:626-730, kernel :35-45).
//
// Pose-pose blocks (incremental chain, S-PGO's parameterisation): for i <= j,
//   A(i, j) = Ad_i^T F(i, j) Ad_j,  F(i, j) = sum_{lo <= i, hi > j} M_{lo,hi},
// computed by a prefix sum over lo (fixed hi, re-centring the running sum on
// each row's camera centre) and a suffix sum over hi (fixed i).  Every sum is
// kept about a nearby camera centre, so the working precision (FP32 in the
// mixed path) never sees world-sized lever arms.
// g(i) = Ad_i^T sum_{lo <= i < hi} m_{lo,hi} is the e = 0 diagonal of the same sums.
#include <algorithm>
#include <type_traits>
#include "kernels.cuh"
#include "frames.cuh"
#include "dfloat.cuh"

namespace spgo {

__device__ __forceinline__ constexpr int t6(int i, int j) {  // symmetric 6x6 upper index, any order
  return i <= j ? i * 6 - (i * (i - 1)) / 2 + (j - i) : j * 6 - (j * (j - 1)) / 2 + (i - j);
}

// Moving a record from origin x to origin y = x - z: E_z^T M E_z and E_z^T m for
// E_z = [[I, 0], [-[z]x, I]] (K^y = K^x E_{x - y}).  With the 6x6 block M = [[P, Q], [Q^T, R]]
// (upper triangle, 21 values), m = [m_w; m_v] and Z = [z]x:  P' = P - Q Z + Z Q^T - Z R Z,
// Q' = Q + Z R,  R' = R,  m' = [m_w + Z m_v ; m_v].  The thread holds all 27 values, so the
// shared products are formed once (about a sixth of the arithmetic of one lane per component):
//   (Z R)[:, j] = z x R[:, j],  (Q Z)[i, :] = -(z x Q[i, :]),  ((Z R) Z)[i, :] = -(z x (Z R)[i, :]),
//   P' = P - Q Z - (Q Z)^T - (Z R) Z,  Q' = Q + Z R,  m_w' = m_w + z x m_v.
template <typename V>
__device__ __forceinline__ void cross3(const V *a, const V *b, V *o) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

// V = double, or df (the mixed path's reduction, on the FP32 pipes)
template <typename V>
__device__ __forceinline__ void shift_record(V *v, const V *z) {
  V P[3][3], Q[3][3], R[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      P[a][c] = v[t6(a, c)];
      Q[a][c] = v[t6(a, 3 + c)];
      R[a][c] = v[t6(3 + a, 3 + c)];
    }
  V ZR[3][3], QZ[3][3], ZRZ[3][3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {  // columns of Z R
    const V rc[3] = {R[0][j], R[1][j], R[2][j]};
    V o[3];
    cross3(z, rc, o);
    ZR[0][j] = o[0];
    ZR[1][j] = o[1];
    ZR[2][j] = o[2];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {  // rows of Q Z and (Z R) Z
    V o[3];
    cross3(z, Q[i], o);
    QZ[i][0] = -o[0];
    QZ[i][1] = -o[1];
    QZ[i][2] = -o[2];
    cross3(z, ZR[i], o);
    ZRZ[i][0] = -o[0];
    ZRZ[i][1] = -o[1];
    ZRZ[i][2] = -o[2];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int c = a; c < 3; ++c) v[t6(a, c)] = P[a][c] - QZ[a][c] - QZ[c][a] - ZRZ[a][c];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[t6(a, 3 + c)] = Q[a][c] + ZR[a][c];
  }
  const V mv[3] = {v[24], v[25], v[26]};
  V o[3];
  cross3(z, mv, o);
  v[21] += o[0];
  v[22] += o[1];
  v[23] += o[2];
}

// pass A (FP64), one CTA per (problem, hi): P(i, hi) = sum_{lo <= i} M(lo, hi) about c_i, each
// M(lo, hi) given about c_lo.  Reads and clears the records.  Every record is moved to the centre
// of the chain's first frame, the running sums are formed there and each is moved back to its own
// row's centre: lever arms stay within the frames that saw the pair's landmarks, and the two
// moves, some 110 FP64 instructions of 64 cycles each, run on all records at once instead of one
// after the other along the chain (101 poses with windows of 41: 202 us with a thread per chain,
// 12.7 us so).
__global__ void __launch_bounds__(SPGO_MAX_WINDOW) k_pair_prefix_rec(PlanView pv, WorkView wv) {
  grid_enter();
  const int b = blockIdx.y;
  if (!problem_active(wv.lm, b, GATE_RELIN)) return;
  __shared__ double v[SPGO_MAX_WINDOW][27];
  const int N = pv.p_npose[b], D = pv.p_pair_D[b], hi = 1 + blockIdx.x, tid = threadIdx.x;
  if (hi > N) return;
  const int fo = pv.p_frame_off[b], lo0 = max(0, hi - D), n = hi - lo0;
  // record (lo, hi)
  auto at = [&](int lo) { return ((size_t)pv.p_pair_off[b] + (size_t)lo * D + (hi - lo - 1)) * 27; };
  auto moved = [&](double *r, int from, int to) {
    const Vec3<double> zz = FramesT<double>::rel(wv, fo + from, 0, fo + to, 0);
    const double z[3] = {zz.x, zz.y, zz.z};
    shift_record(r, z);
  };
  for (int q = tid; q < n; q += blockDim.x) {
    double *rec = reinterpret_cast<double *>(wv.pair_acc) + at(lo0 + q);
    double r[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) r[k] = rec[k];
#pragma unroll
    for (int k = 0; k < 27; ++k) rec[k] = 0.0;  // cleared for the next linearisation
    if (q > 0) moved(r, lo0 + q, lo0);
#pragma unroll
    for (int k = 0; k < 27; ++k) v[q][k] = r[k];
  }
  __syncthreads();
  if (tid < 27) {
    double sum = 0.0;
    for (int q = 0; q < n; ++q) {
      sum += v[q][tid];
      v[q][tid] = sum;
    }
  }
  __syncthreads();
  for (int q = tid; q < n; q += blockDim.x) {
    double r[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) r[k] = v[q][k];
    if (q > 0) moved(r, lo0, lo0 + q);
    double *out = reinterpret_cast<double *>(wv.pairF) + at(lo0 + q);
#pragma unroll
    for (int k = 0; k < 27; ++k) out[k] = r[k];
  }
}

// pass B, one thread per (problem, i, component): F(i, i + e) = sum_{d' > e} P(i, i + d')
// (all about origin c_i), in place
template <typename T>
__global__ void k_pair_suffix(PlanView pv, WorkView wv) {
  grid_enter();
  const int b = blockIdx.y;
  if (!problem_active(wv.lm, b, GATE_RELIN)) return;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N * 27) return;
  const int i = t / 27, comp = t % 27;
  T *base = reinterpret_cast<T *>(wv.pairF) + ((size_t)pv.p_pair_off[b] + (size_t)i * D) * 27 + comp;
  T acc = T(0);
  int dp = min(D, N - i);
  for (; dp >= 8; dp -= 8) {  // eight records loaded before any is summed
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = base[(size_t)(dp - 1 - q) * 27];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      acc += v[q];
      base[(size_t)(dp - 1 - q) * 27] = acc;
    }
  }
  for (; dp >= 1; --dp) {
    T *p = base + (size_t)(dp - 1) * 27;
    acc += *p;
    *p = acc;
  }
}

// ---- the mixed path's pair reduction, in double-float ----------------------------
// The records arrive as FP64 sums (the linearisation's atomics).  FP64 arithmetic runs at
// a small fraction of the FP32 rate on this GPU, so the reduction runs in double-float
// (~48 bits on the FP32 pipes, far more than the FP32 blocks it produces keep).  Instead
// of re-centring a running sum along each chain (a serial chain of shifts), every record
// is moved once to the problem's own origin o = c_0 (its lever arms are at most the
// window's extent, tens of metres, which costs a few of the 48 bits), the prefix and
// suffix sums run about o, and A and g are formed from the sums about o.
__device__ __forceinline__ void df_rel_c(const WorkView &wv, int fx, int fy, df *z) {  // c_x - c_y, left cameras
#pragma unroll
  for (int k = 0; k < 3; ++k)
    z[k] = df_sub(wv.fr_ch[(size_t)fx * 6 + k], wv.fr_ch[(size_t)fy * 6 + k]) +
           df_make(wv.fr_cl[(size_t)fx * 6 + k] - wv.fr_cl[(size_t)fy * 6 + k]);
}

constexpr int kPrThreads = 896;  // thread per (pose, component) of a 33-pose window

// 0. every record (lo, hi): read (FP64) and cleared, split into double-float, moved from
// c_lo to o.  A CTA stages kShRecs records in shared memory (whole lines in and out); lane i of
// three moves row i of a record's P and Q (shift_record's formulas; row i of Z R, Q Z and (Z R) Z
// and column i of Q Z).  Bound by the latency of one record's double-float chain: a thread per
// record 11.4 us for a 10-pose window and 19.3 us for 64 of up to 32 poses, 7.2 and 11.2 us so.
constexpr int kShRecs = 32;

__global__ void __launch_bounds__(128) k_pair_shift_df(PlanView pv, WorkView wv) {
  grid_enter();
  const int b = blockIdx.y;
  if (!problem_active(wv.lm, b, GATE_RELIN)) return;
  __shared__ df v[kShRecs * 27];
  const int N = pv.p_npose[b], D = pv.p_pair_D[b], fo = pv.p_frame_off[b];
  const int r0 = blockIdx.x * kShRecs, n = min(kShRecs, N * D - r0);
  if (n <= 0) return;
  const size_t off = ((size_t)pv.p_pair_off[b] + r0) * 27;
  double *rec = reinterpret_cast<double *>(wv.pair_acc) + off;
  df *out = reinterpret_cast<df *>(wv.pairF) + off;
  auto valid = [&](int r) { return (r0 + r) / D + (r0 + r) % D + 1 <= N; };
  for (int q = threadIdx.x; q < 27 * n; q += blockDim.x) {
    if (!valid(q / 27)) continue;
    v[q] = df_split_double(rec[q]);
    rec[q] = 0.0;  // cleared for the next linearisation
  }
  __syncthreads();
  const int r = threadIdx.x >> 2, i = threadIdx.x & 3, lo = (r0 + r) / D;
  const bool mine = r < n && i < 3 && lo > 0 && valid(r);
  df p[3], q[3], mw;
  if (mine) {
    const df *m = v + 27 * r;
    const int i1 = i == 2 ? 0 : i + 1, i2 = i == 0 ? 2 : i - 1;
    df z[3], qi[3];
    df_rel_c(wv, fo + lo, fo, z);  // from c_lo to o = c_0
    const df z1 = i == 0 ? z[1] : i == 1 ? z[2] : z[0], z2 = i == 0 ? z[2] : i == 1 ? z[0] : z[1];
    df zr[3], qz[3], zrz[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      qi[j] = m[t6(i, 3 + j)];
      zr[j] = z1 * m[t6(3 + i2, 3 + j)] - z2 * m[t6(3 + i1, 3 + j)];
    }
    cross3(z, qi, qz);   // -(Q Z)[i, :]
    cross3(z, zr, zrz);  // -((Z R) Z)[i, :]
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const df qzc = z1 * m[t6(c, 3 + i2)] - z2 * m[t6(c, 3 + i1)];  // -(Q Z)[c, i]
      p[c] = m[t6(i, c)] + qz[c] + qzc + zrz[c];
      q[c] = qi[c] + zr[c];
    }
    mw = m[21 + i] + (z1 * m[24 + i2] - z2 * m[24 + i1]);
  }
  __syncthreads();
  if (mine) {
    df *m = v + 27 * r;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (c >= i) m[t6(i, c)] = p[c];
      m[t6(i, 3 + c)] = q[c];
    }
    m[21 + i] = mw;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 27 * n; k += blockDim.x)
    if (valid(k / 27)) out[k] = v[k];
}

// 1. thread per (hi, component): prefix over lo, P(i, hi) = sum_{lo <= i} M(lo, hi);
// 2. thread per (i, component): suffix over hi, F(i, i + e) = sum_{d > e} P(i, i + d).
// PHASE 0: both, one CTA per problem (the windows of a batch); 1, 2: one of them over a grid,
// for trajectories of more than kPrWide poses (500 poses on one SM took 150 us, spread out
// 12 us).  Whole Gauss-Newton steps with one launch and with two, us: a 10-pose window 86 and 88,
// 64 of 10 105 and 108, 64 of 32 392 and 396; 48 poses 277 and 272, 100 poses 321 and 297.
constexpr int kPrWide = 48;

template <int PHASE>
__global__ void __launch_bounds__(kPrThreads) k_pair_scan_df(PlanView pv, WorkView wv) {
  grid_enter();
  const int b = blockIdx.x;
  if (!problem_active(wv.lm, b, GATE_RELIN)) return;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b];
  const int tid = blockIdx.y * blockDim.x + threadIdx.x, nt = gridDim.y * blockDim.x;
  df *F = reinterpret_cast<df *>(wv.pairF) + (size_t)pv.p_pair_off[b] * 27;
  // the running sums: eight records loaded before any is summed and stored back (the
  // stores could alias later loads, so without that each step is a round trip)
  for (int t = PHASE == 2 ? N * 27 : tid; t < N * 27; t += nt) {
    const int hi = t / 27 + 1, comp = t % 27;
    df s = df_make(0.f);
    for (int lo0 = max(0, hi - D); lo0 < hi; lo0 += 8) {
      df v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (lo0 + q < hi) v[q] = F[((size_t)(lo0 + q) * D + (hi - lo0 - q - 1)) * 27 + comp];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (lo0 + q < hi) {
          s = s + v[q];
          F[((size_t)(lo0 + q) * D + (hi - lo0 - q - 1)) * 27 + comp] = s;
        }
    }
  }
  if (PHASE == 1) return;
  if (PHASE == 0) __syncthreads();
  for (int t = tid; t < N * 27; t += nt) {
    const int i = t / 27, comp = t % 27;
    df *base = F + (size_t)i * D * 27 + comp;
    df s = df_make(0.f);
    for (int dp0 = min(D, N - i); dp0 >= 1; dp0 -= 8) {
      df v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (dp0 - q >= 1) v[q] = base[(size_t)(dp0 - q - 1) * 27];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (dp0 - q >= 1) {
          s = s + v[q];
          base[(size_t)(dp0 - q - 1) * 27] = s;
        }
    }
  }
}

// A(i, j) = Ad_i^T F(i, j) Ad_j and g(i) = the same of F's gradient, F about an origin o (FP64:
// c_i; mixed: the problem's c_0) and Ad_k = [[R_k, 0], [[c_k - o]x R_k, R_k]]; the mixed path in
// double-float, rounded once to FP32, the unrounded g also to gacc (the refined step's predicted
// decrease).  One thread per column of a block: some 70 multiply-adds in a chain-bound kernel,
// where a thread per block had 350 (FP64, 64 cycles each: 10 us a window), and 460 with the move
// of F from o to c_i that the mixed path made first (16.6 us a window; 5.2 us so).
template <typename T>
__global__ void __launch_bounds__(128) k_pairs_to_A(PlanView pv, WorkView wv) {
  grid_enter();
  constexpr bool f64 = std::is_same<T, double>::value;
  using V = typename std::conditional<f64, double, df>::type;
  const int b = blockIdx.y;
  if (!problem_active(wv.lm, b, GATE_RELIN)) return;
  const int N = pv.p_npose[b], D = pv.p_pair_D[b];
  const int t = blockIdx.x * blockDim.x + threadIdx.x, col = t % 6, i = t / (6 * D), e = t / 6 - i * D;
  if (i >= N || e >= min(D, N - i)) return;
  const int j = i + e, P = 6 * N, fo = pv.p_frame_off[b], cc = col < 3 ? col : col - 3;
  const V *Fg = reinterpret_cast<const V *>(wv.pairF) + ((size_t)pv.p_pair_off[b] + (size_t)i * D + e) * 27;
  V F[21], Ri[9], a[3], lj[3], li[3];  // a: column cc of R_j
#pragma unroll
  for (int k = 0; k < 21; ++k) F[k] = Fg[k];
  if constexpr (f64) {
    const double *ri = FramesT<double>::R(wv, fo + i, 0), *rj = FramesT<double>::R(wv, fo + j, 0);
#pragma unroll
    for (int k = 0; k < 9; ++k) Ri[k] = ri[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = rj[3 * k + cc];
    const Vec3<double> c = FramesT<double>::rel(wv, fo + j, 0, fo + i, 0);
    lj[0] = c.x, lj[1] = c.y, lj[2] = c.z;
  } else {
    const float *h = wv.fr_Rf + (size_t)(fo + i) * 18, *l = wv.fr_Rl + (size_t)(fo + i) * 18;
    const float *hj = wv.fr_Rf + (size_t)(fo + j) * 18, *ljp = wv.fr_Rl + (size_t)(fo + j) * 18;
#pragma unroll
    for (int k = 0; k < 9; ++k) Ri[k] = df{h[k], l[k]};
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = df{hj[3 * k + cc], ljp[3 * k + cc]};
    df_rel_c(wv, fo + j, fo, lj);
    df_rel_c(wv, fo + i, fo, li);
  }
  // column col of Ad_j: [a; l_j x a] (col < 3), [0; a]
  V ad[6];
  cross3(lj, a, ad + 3);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ad[k] = col < 3 ? a[k] : V{};
    ad[3 + k] = col < 3 ? ad[3 + k] : a[k];
  }
  V w[6];
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    V u = F[t6(r, 0)] * ad[0];
#pragma unroll
    for (int k = 1; k < 6; ++k) u = u + F[t6(r, k)] * ad[k];
    w[r] = u;
  }
  auto to_frame_i = [&](V *x) {  // x[0..2] -= l_i x x[3..5]
    if constexpr (!f64) {
      V o[3];
      cross3(li, x + 3, o);
#pragma unroll
      for (int k = 0; k < 3; ++k) x[k] = x[k] - o[k];
    }
  };
  auto round_t = [](const V &x) {
    if constexpr (f64)
      return x;
    else
      return df_to_float(x);
  };
  to_frame_i(w);
  T out[6];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    out[r] = round_t(Ri[r] * w[0] + Ri[3 + r] * w[1] + Ri[6 + r] * w[2]);
    out[3 + r] = round_t(Ri[r] * w[3] + Ri[3 + r] * w[4] + Ri[6 + r] * w[5]);
  }
  T *A = reinterpret_cast<T *>(wv.A) + pv.p_S_off[b];
#pragma unroll
  for (int r = 0; r < 6; ++r) A[(size_t)(6 * i + r) * P + 6 * j + col] = out[r];
  if (i != j) {  // its transpose: 6 elements at 6i of row 6j + col (even offsets in a 256-byte aligned segment)
    using T2 = typename std::conditional<f64, double2, float2>::type;
    T2 *dst = reinterpret_cast<T2 *>(A + (size_t)(6 * j + col) * P + 6 * i);
#pragma unroll
    for (int r = 0; r < 3; ++r) dst[r] = T2{out[2 * r], out[2 * r + 1]};
  } else {
    V f[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) f[k] = Fg[21 + k];
    to_frame_i(f);
    V gr{};
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // (Ri in registers: its column by selection)
      const V rk = cc == 0 ? Ri[3 * k] : cc == 1 ? Ri[3 * k + 1] : Ri[3 * k + 2];
      gr = gr + rk * (col < 3 ? f[k] : f[3 + k]);
    }
    const int row = pv.p_param_off[b] + 6 * i + col;
    reinterpret_cast<T *>(wv.g)[row] = round_t(gr);
    if constexpr (!f64)
      if (wv.gacc) wv.gacc[row] = df_to_double(gr);
  }
}

// The pose-pair records are FP64 sums on both paths.  The FP64 path reduces them in
// FP64 along each chain; the mixed path (T = float) in double-float about one origin
// per problem, storing A and g as FP32.
template <typename T>
int launch_system(const PlanView &pv, const WorkView &wv, int gate, void *stream) {
  (void)gate;
  cudaStream_t st = (cudaStream_t)stream;
  const int nmax = pv.max_P / 6;
  const int nd = pv.max_D > 0 ? pv.max_D : 1;
  if constexpr (std::is_same<T, float>::value) {
    launch(k_pair_shift_df, dim3(grid_for((long long)nmax * nd, kShRecs), pv.B), 4 * kShRecs, 0, st, pv, wv);
    if (nmax <= kPrWide) {
      launch(k_pair_scan_df<0>, pv.B, std::min(kPrThreads, 32 * grid_for(27 * nmax, 32)), 0, st, pv, wv);
    } else {
      const dim3 grid(pv.B, grid_for((long long)nmax * 27, 128));
      launch(k_pair_scan_df<1>, grid, 128, 0, st, pv, wv);
      launch(k_pair_scan_df<2>, grid, 128, 0, st, pv, wv);
      ++g_launches;
    }
    launch(k_pairs_to_A<float>, dim3(grid_for((long long)nmax * nd * 6, 128), pv.B), 128, 0, st, pv, wv);
    g_launches += 3;
  } else {
    launch(k_pair_prefix_rec, dim3(nmax, pv.B), 32 * grid_for(std::min(nd, nmax), 32), 0, st, pv, wv);
    launch(k_pair_suffix<double>, dim3(grid_for((long long)nmax * 27, 128), pv.B), 128, 0, st, pv, wv);
    launch(k_pairs_to_A<double>, dim3(grid_for((long long)nmax * nd * 6, 128), pv.B), 128, 0, st, pv, wv);
    g_launches += 3;
  }
  return (int)cudaGetLastError();
}

// ---- landmark Schur complement ------------------------------------------------
// S_L(I, J) = sum over chunks of W_I diag(d) W_J^T with d_l = 1 / (C_l (1 + lam) + eps),
// g_L = sum W d g_a.  One CTA per work item = (problem, 48x48 output tile, <= 16 chunks);
// partial tiles are added atomically (S_L is cleared by the assembly that reads it).
template <typename T>
__global__ void __launch_bounds__(256) k_schur(PlanView pv, WorkView wv, Params prm, int gate) {
  grid_enter();
  const int w = blockIdx.x;
  const int b = pv.wk_prob[w];
  if (!problem_active(wv.lm, b, gate)) return;
  const int ti = pv.wk_ti[w], tj = pv.wk_tj[w];
  const int N = pv.p_npose[b], P = 6 * N;
  const double lam = wv.lm[b].lam;
  const T eps = (T)prm.eps;
  constexpr int TR = 6 * SPGO_TILE_BLOCKS;  // 48
  __shared__ T WI[TR][SPGO_CHUNK + 1];
  __shared__ T WJ[TR][SPGO_CHUNK + 1];
  __shared__ T dg[SPGO_CHUNK];
  const int tid = threadIdx.x;
  const int tr = tid / 16, tc = tid % 16;
  T acc[3][3];
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int y = 0; y < 3; ++y) acc[x][y] = T(0);
  T accg = T(0);
  const bool diag = (ti == tj);
  const T *Cv = reinterpret_cast<const T *>(wv.C);
  const T *gav = reinterpret_cast<const T *>(wv.ga);
  const T *slab_all = reinterpret_cast<const T *>(wv.slab);
  for (int k = pv.wk_cbeg[w]; k < pv.wk_cend[w]; ++k) {
    const int c = pv.wk_chunks[k];
    const int f0 = pv.ch_f0[c], nb = pv.ch_nb[c], lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
    const T *slab = slab_all + pv.ch_slab[c];
    for (int idx = tid; idx < TR * SPGO_CHUNK; idx += blockDim.x) {
      const int r = idx / SPGO_CHUNK, col = idx % SPGO_CHUNK;
      const int bi = SPGO_TILE_BLOCKS * ti + r / 6;
      const int bj = SPGO_TILE_BLOCKS * tj + r / 6;
      T dv = T(0);
      if (col < cnt) dv = T(1) / (Cv[lm0 + col] * (T)(1.0 + lam) + eps);
      T vi = T(0), vj = T(0);
      if (bi >= f0 && bi < f0 + nb && bi < N) vi = slab[(size_t)(6 * (bi - f0) + r % 6) * SPGO_CHUNK + col];
      if (bj >= f0 && bj < f0 + nb && bj < N) vj = slab[(size_t)(6 * (bj - f0) + r % 6) * SPGO_CHUNK + col];
      WI[r][col] = vi;
      WJ[r][col] = vj * dv;
      if (r == 0) dg[col] = (col < cnt) ? dv * gav[lm0 + col] : T(0);
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < SPGO_CHUNK; ++kk) {
      const T a0 = WI[3 * tr][kk], a1 = WI[3 * tr + 1][kk], a2 = WI[3 * tr + 2][kk];
      const T b0 = WJ[3 * tc][kk], b1 = WJ[3 * tc + 1][kk], b2 = WJ[3 * tc + 2][kk];
      acc[0][0] += a0 * b0; acc[0][1] += a0 * b1; acc[0][2] += a0 * b2;
      acc[1][0] += a1 * b0; acc[1][1] += a1 * b1; acc[1][2] += a1 * b2;
      acc[2][0] += a2 * b0; acc[2][1] += a2 * b1; acc[2][2] += a2 * b2;
    }
    if (diag && tid < TR) {
#pragma unroll 8
      for (int kk = 0; kk < SPGO_CHUNK; ++kk) accg += WI[tid][kk] * dg[kk];
    }
    __syncthreads();
  }
  T *SL = reinterpret_cast<T *>(wv.SL) + pv.p_S_off[b];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const int row = TR * ti + 3 * tr + x;
    if (row >= P) continue;
#pragma unroll
    for (int y = 0; y < 3; ++y) {
      const int col = TR * tj + 3 * tc + y;
      if (col <= row && acc[x][y] != T(0)) red_add(SL + (size_t)row * P + col, acc[x][y]);  // (the lower triangle)
    }
  }
  if (diag && tid < TR) {
    const int row = TR * ti + tid;
    if (row < P && accg != T(0)) red_add(reinterpret_cast<T *>(wv.gL) + pv.p_param_off[b] + row, accg);
  }
}

// ---- the FP64 path's Schur complement -------------------------------------------
// Bound by the FP64 pipe (2 FMA per SM and cycle on this part: everything else in the
// kernel is hidden behind it), so what counts is how many FP64 warp instructions it
// issues.  A landmark's column of W is non-zero only in its own window [lo, hi) of pose
// blocks, about 70 % of a circle problem's poses and 20 of a corridor's hundreds.  A warp
// owns 2 x 4 pose blocks of the 48x48 tile (3x3 outputs a lane) and multiplies only the
// landmarks whose window meets both its rows and its columns (one ballot per chunk); the
// warps above the diagonal of a diagonal tile do nothing, and 1 / D is formed once per
// landmark instead of once per tile row.  Counted on config-3 problems, this leaves 1.37x
// the FMAs of the exact per-landmark lower triangles, against 4.6x for whole tiles (a
// 1 x 8 block warp shape: 1.62x).  256-problem batch: 11.7 -> 4.1 ms a launch; one 10-pose
// window, whose 6 items left the GPU empty, 235 -> about 90 us.
// blockIdx.y splits an item's chunks where the plan has too few items to fill the GPU.
__global__ void __launch_bounds__(256) k_schur_f64(PlanView pv, WorkView wv, Params prm, int gate) {
  grid_enter();
  const int w = blockIdx.x;
  const int b = pv.wk_prob[w];
  if (!problem_active(wv.lm, b, gate)) return;
  const int c0 = pv.wk_cbeg[w], len = pv.wk_cend[w] - c0;
  const int kb = c0 + len * (int)blockIdx.y / (int)gridDim.y, ke = c0 + len * ((int)blockIdx.y + 1) / (int)gridDim.y;
  if (kb >= ke) return;
  const int ti = pv.wk_ti[w], tj = pv.wk_tj[w];
  const int P = 6 * pv.p_npose[b];
  const double lam1 = 1.0 + wv.lm[b].lam, eps = (double)prm.eps;
  constexpr int TR = 6 * SPGO_TILE_BLOCKS;  // 48
  __shared__ double WI[TR][SPGO_CHUNK + 1];
  __shared__ double WJ[TR][SPGO_CHUNK + 1];  // scaled by 1 / D
  __shared__ double dv[2][SPGO_CHUNK];
  __shared__ double gs[2][SPGO_CHUNK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool diag = ti == tj;
  const int wr = warp >> 1, wc = warp & 1;
  const int br = SPGO_TILE_BLOCKS * ti + 2 * wr, bc = SPGO_TILE_BLOCKS * tj + 4 * wc;  // the warp's first blocks
  const bool idle = diag && 2 * wr + 1 < 4 * wc;                                        // above the diagonal
  const int tr = 12 * wr + 3 * (lane >> 3), tc = 24 * wc + 3 * (lane & 7);              // the lane's first outputs
  double acc[3][3];
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int y = 0; y < 3; ++y) acc[x][y] = 0.0;
  double accg = 0.0;
  const double *Cv = reinterpret_cast<const double *>(wv.C);
  const double *gav = reinterpret_cast<const double *>(wv.ga);
  const double *slab_all = reinterpret_cast<const double *>(wv.slab);
  auto scales = [&](int k) {  // lane = landmark of chunk k: 1 / D and g_a
    const int c = pv.wk_chunks[k];
    const int lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
    dv[k & 1][lane] = lane < cnt ? 1.0 / (Cv[lm0 + lane] * lam1 + eps) : 0.0;
    gs[k & 1][lane] = lane < cnt ? gav[lm0 + lane] : 0.0;
  };
  if (warp == 0) scales(kb);
  for (int k = kb; k < ke; ++k) {
    const int c = pv.wk_chunks[k];
    const int f0 = pv.ch_f0[c], nb = pv.ch_nb[c], lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
    const double *slab = slab_all + pv.ch_slab[c];
    // this chunk's rows of the tile, before the barrier that ends the previous chunk
    constexpr int RPW = TR / 8;
    const int ri = 6 * (SPGO_TILE_BLOCKS * ti - f0) + warp, rj = 6 * (SPGO_TILE_BLOCKS * tj - f0) + warp;
    double vi[RPW], vj[RPW];
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      const int r = ri + 8 * q, s = rj + 8 * q;
      vi[q] = r >= 0 && r < 6 * nb ? slab[(size_t)r * SPGO_CHUNK + lane] : 0.0;
      vj[q] = diag ? vi[q] : (s >= 0 && s < 6 * nb ? slab[(size_t)s * SPGO_CHUNK + lane] : 0.0);
    }
    const int lo = lane < cnt ? pv.lm_lo[lm0 + lane] : 0, hi = lane < cnt ? pv.lm_hi[lm0 + lane] : 0;
    __syncthreads();
    const double d = dv[k & 1][lane];
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      WI[warp + 8 * q][lane] = vi[q];
      WJ[warp + 8 * q][lane] = vj[q] * d;
    }
    __syncthreads();
    if (warp == 7 && k + 1 < ke) scales(k + 1);
    // (a 1 / D that is not finite is never skipped: it has to reach S and fail the factor)
    const bool bad = (((unsigned)__double2hiint(d) >> 20) & 0x7ffu) == 0x7ffu;
    unsigned m = __ballot_sync(0xffffffffu, !idle && (bad || (lo < br + 2 && hi > br && lo < bc + 4 && hi > bc)));
    while (m) {
      const int kk = __ffs(m) - 1;
      m &= m - 1;
      const double a0 = WI[tr][kk], a1 = WI[tr + 1][kk], a2 = WI[tr + 2][kk];
      const double b0 = WJ[tc][kk], b1 = WJ[tc + 1][kk], b2 = WJ[tc + 2][kk];
      acc[0][0] += a0 * b0; acc[0][1] += a0 * b1; acc[0][2] += a0 * b2;
      acc[1][0] += a1 * b0; acc[1][1] += a1 * b1; acc[1][2] += a1 * b2;
      acc[2][0] += a2 * b0; acc[2][1] += a2 * b1; acc[2][2] += a2 * b2;
    }
    if (diag && tid < TR) {  // g_L row: the scaled rows times g_a
      for (int kk = 0; kk < cnt; ++kk) accg += WJ[tid][kk] * gs[k & 1][kk];
    }
  }
  double *SL = reinterpret_cast<double *>(wv.SL) + pv.p_S_off[b];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const int row = TR * ti + tr + x;
#pragma unroll
    for (int y = 0; y < 3; ++y) {
      const int col = TR * tj + tc + y;
      if (row < P && col <= row && acc[x][y] != 0.0) red_add(SL + (size_t)row * P + col, acc[x][y]);
    }
  }
  if (diag && tid < TR) {
    const int row = TR * ti + tid;
    if (row < P && accg != 0.0) red_add(reinterpret_cast<double *>(wv.gL) + pv.p_param_off[b] + row, accg);
  }
}

template <typename T>
int launch_schur(const PlanView &pv, const WorkView &wv, const Params &prm, void *stream) {
  if (pv.n_items == 0) return 0;
  if constexpr (std::is_same<T, double>::value) {
    // a chunk of one tile keeps an SM's FP64 pipe busy for several microseconds, so items
    // are split down to single chunks until there are four CTAs per SM
    const int sub = std::max(1, std::min(pv.wk_max_len, (4 * kSmCount + pv.n_items - 1) / pv.n_items));
    launch(k_schur_f64, dim3(pv.n_items, sub), 256, 0, (cudaStream_t)stream, pv, wv, prm, GATE_RUNNING);
  } else {
    launch(k_schur<T>, pv.n_items, 256, 0, (cudaStream_t)stream, pv, wv, prm, GATE_RUNNING);
  }
  ++g_launches;
  return (int)cudaGetLastError();
}

template int launch_system<float>(const PlanView &, const WorkView &, int, void *);
template int launch_system<double>(const PlanView &, const WorkView &, int, void *);
template int launch_schur<float>(const PlanView &, const WorkView &, const Params &, void *);
template int launch_schur<double>(const PlanView &, const WorkView &, const Params &, void *);

}  // namespace spgo
