// The Jacobian pass: normal equations of every observation, both precisions.
//
// The rows of an observation's pose Jacobian are linear functions of the 3-D point: with
// u = dpi/dt R_n^T (two rows per camera) and X the point relative to an origin x, a row about
// x is [X x u, u] and the inverse-depth entry is u . dX (dX = dX / d alpha).  So everything
// the observation adds to the normal equations follows from two small sums over its four
// rows, weighted by the robust weight w^2,
//     H = sum w^2 u u^T  (3x3, 6 values),    h = sum w^2 u r  (3 values):
//   pair record about c_lo (21 + 6 values):  [[X]x H [X]x^T, [X]x H; ., H],  s [X x h; h];
//   pose / inverse-depth column:  s [X x q; q] with q = H dX, about any origin, so the suffix
//     and prefix sums along the landmark's window run over q alone (3 values) and the
//     products with X and the rotation to each pose come after them;
//   C = dX . sum q and g_a = dX . sum h: no sums of their own over the observations.
// Forming the 27 record values and the column as products of 6-wide rows took 34 exact
// four-product sums an observation on the mixed path; here it is 9, and cross products.
//
// The sums that build the normal equations are not left to FP32 on the mixed path: the
// reduced camera system S = A + damping - W D^-1 W^T cancels most of A, and FP32 sums over
// thousands of observations put errors into A and W that, measured against S, reach its
// smallest eigenvalues (an FP32-assembled S of a badly initialised circle problem came out
// indefinite where the FP64 one has scaled smallest eigenvalue 4e-4).  So there H and h are
// exact sums (two-product, double-float) over FP32 rows, every further value is
// a double-float, a warp's run over the observations of one target frame is summed in
// double-float and goes to the FP64 pair record by an FP64 atomic (the pair reduction then
// runs in double-float about one origin, k_system.cu), and the slab is rounded to FP32 once,
// at the end.  The refinement's residual pass (k_refine.cu) uses the same rounded rows in the
// same structure: where S's small eigenvalues are at the FP32 rounding of A, a preconditioner
// from another rounding of the same Jacobian is no preconditioner (three problems of the
// 256-window batch stalled up to 2.8x above the FP64 cost).  (A slab accumulated in FP32, and
// one whose double-float moments were rounded before an FP32 rotation to the pose axes, left
// single ill-conditioned problems of the 256-window batch with an unusable preconditioner.)
// The residuals, camera-frame points and
// anchor points are the cost pass's at the same state, rounded once from double-float.  The
// FP64 path is the same kernel in double, forming those itself.
//
// One CTA per chunk of <= 32 landmarks of one host frame, observations sorted by target frame.
// Bound by instruction issue (mixed) and by the FP64 pipe (FP64).  256 windows (3.66 M
// observations): 752 -> 551 us (mixed) and 4.66 -> 2.34 ms (FP64) a pass against the products
// of 6-wide rows; a 500-pose corridor (3.1 M), 455 -> 335 us.
#include <type_traits>

#include "kernels.cuh"
#include "frames.cuh"
#include "jac_rows.cuh"

namespace spgo {

// upper-triangle index of a symmetric 6x6 / 3x3 (row i <= col j)
__device__ __forceinline__ constexpr int tri6(int i, int j) { return i * 6 - (i * (i - 1)) / 2 + (j - i); }
__device__ __forceinline__ constexpr int sym3(int i, int j) {
  return i <= j ? i * 3 - (i * (i - 1)) / 2 + (j - i) : j * 3 - (j * (j - 1)) / 2 + (i - j);
}

template <typename T>
struct JacSmem {
  T X[SPGO_CHUNK][3];   // anchor point, world axes, relative to the anchor centre
  T dX[SPGO_CHUNK][3];  // dX / d alpha
  typename Num<T>::V tot[3][SPGO_CHUNK];  // sum of q over the landmark's observations
  int lo[SPGO_CHUNK], hi[SPGO_CHUNK];
  unsigned rmask[SPGO_MAX_WINDOW];  // per window row: the landmarks whose window holds its frame
  int rsp[SPGO_MAX_WINDOW + 1];     // exclusive prefix of the rows' landmark counts
  int key[8][32];                   // per warp: target frame of each lane's observation (-1: none)
};
constexpr int kJacVals = 27;    // 21 Hessian + 6 gradient values per pair record
constexpr int kJacRound = 9;    // pair values staged per round (three rounds of 9)
constexpr int kJacSegs = 3;     // observation segments per staged value in the run sums
constexpr int kJacSegLen = 11;  // ceil(32 / 3)
constexpr int kJacPitch = 33;

// dynamic shared memory, 8-byte elements V: d [W][6] the host's left centre minus every window
// frame's camera centres | stage [warps][9][33] pair values, one round | rows [W][kJacRow][32]
// per window frame q (3) and dX . h, by landmark.  In place of the q's of a row later come the
// pose / inverse-depth entries: FP32 pairs (2 x 3 floats, in the 3 q's), or 6 doubles, which
// sets the FP64 path's row to 6 elements.  33-frame windows: 56 KB (mixed), 73 KB (FP64).
template <typename T>
constexpr int kJacRow = std::is_same<T, float>::value ? 4 : 6;
template <typename T>
struct JacLayout {
  size_t d, stage, rows, total;
  __host__ __device__ JacLayout(int max_nb, int warps) {
    const size_t W = (size_t)max_nb + 1;
    d = (sizeof(JacSmem<T>) + 15) & ~(size_t)15;
    stage = d + W * 6 * 8;
    rows = (stage + (size_t)warps * kJacRound * kJacPitch * 8 + 15) & ~(size_t)15;
    total = rows + W * kJacRow<T> * SPGO_CHUNK * 8;
  }
};

// Sums the staged values [V0, V0 + 9) over the runs of equal target frame: lane = (value,
// 11-observation segment); every run goes to its FP64 pair record (a run crossing a segment
// boundary arrives in parts)
template <typename T, int V0>
__device__ __forceinline__ void jac_runs(const typename Num<T>::V *st, const int *keys, int lane, int host_a, int D,
                                         double *pair_base) {
  if (lane >= kJacSegs * kJacRound) return;
  const int v = lane % kJacRound, i0 = (lane / kJacRound) * kJacSegLen, i1 = min(32, i0 + kJacSegLen);
  const typename Num<T>::V *col = st + v * kJacPitch;
  auto emit = [&](int n, const typename Num<T>::Acc &a) {
    const int lo = min(host_a, n), hi = max(host_a, n);
    atomicAdd(pair_base + ((size_t)lo * D + (hi - lo - 1)) * kJacVals + V0 + v, Num<T>::acc_value(a));
  };
  typename Num<T>::Acc acc{};
  int cur = keys[i0];
#pragma unroll 4
  for (int i = i0; i < i1; ++i) {
    const int k = keys[i];
    if (k != cur) {
      if (cur >= 0) emit(cur, acc);
      acc = typename Num<T>::Acc();
      cur = k;
    }
    Num<T>::acc(acc, col[i]);
  }
  if (cur >= 0) emit(cur, acc);
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_jacobian(PlanView pv, WorkView wv, Params prm,
                                                                         const double *__restrict__ alpha_state,
                                                                         int gate) {
  grid_enter();
  using M = Num<T>;
  using V = typename M::V;
  constexpr bool kMixed = std::is_same<T, float>::value;
  constexpr int kRow = kJacRow<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int2 cb = pv.ch_sched[blockIdx.x];
  const int c = cb.x, b = cb.y;
  if (!problem_active(wv.lm, b, gate)) return;
  const int tid = threadIdx.x, lane = tid & 31;
  const int f0 = pv.ch_f0[c], nb = pv.ch_nb[c], lm0 = pv.ch_lm0[c], cnt = pv.ch_cnt[c];
  const int fo = pv.p_frame_off[b];
  const float *intr = pv.p_intr + 8 * b;
  JacSmem<T> &sm = *reinterpret_cast<JacSmem<T> *>(smem_raw);
  const JacLayout<T> lay(pv.max_nb, blockDim.x >> 5);
  V *dc = reinterpret_cast<V *>(smem_raw + lay.d);
  V *stage = reinterpret_cast<V *>(smem_raw + lay.stage);
  V *rows = reinterpret_cast<V *>(smem_raw + lay.rows);
  auto row_at = [&](int f, int k, int slot) { return rows + ((size_t)f * kRow + k) * SPGO_CHUNK + slot; };
  const int host = pv.lm_host[lm0];  // every landmark of the chunk has this host
  const int64_t ob = pv.lm_obs[lm0], oe = pv.lm_obs[lm0 + cnt];

  // phase A: the chunk's anchor points, its windows, the centre differences
  if (tid < cnt) {
    const int li = lm0 + tid;
    if constexpr (kMixed) {  // as the cost pass at this state formed them
      const float4 *xa = reinterpret_cast<const float4 *>(wv.xanc + ((size_t)wv.lm[b].res_sel * pv.L + li) * 8);
      const float4 x0 = xa[0], x1 = xa[1];
      sm.X[tid][0] = x0.x, sm.X[tid][1] = x0.y, sm.X[tid][2] = x0.z;
      sm.dX[tid][0] = x0.w, sm.dX[tid][1] = x1.x, sm.dX[tid][2] = x1.y;
    } else {
      const double alpha = alpha_state[pv.lm_user[li]];
      const double ua = (double)pv.lm_uv[2 * li], va = (double)pv.lm_uv[2 * li + 1];
      const Vec3<double> ta = v3<double>((ua - (double)intr[2]) / (double)intr[0] / alpha,
                                         (va - (double)intr[3]) / (double)intr[1] / alpha, 1.0 / alpha);
      const Vec3<double> X = mul(FramesT<double>::R(wv, fo + host, 0), ta);
      sm.X[tid][0] = X.x, sm.X[tid][1] = X.y, sm.X[tid][2] = X.z;
      sm.dX[tid][0] = -X.x / alpha, sm.dX[tid][1] = -X.y / alpha, sm.dX[tid][2] = -X.z / alpha;
    }
    sm.lo[tid] = pv.lm_lo[li];
    sm.hi[tid] = pv.lm_hi[li];
  }
  if (tid < 32) {  // per window row, the landmarks whose window [lo, hi) holds its frame
    const int lo = tid < cnt ? pv.lm_lo[lm0 + tid] : 0, hi = tid < cnt ? pv.lm_hi[lm0 + tid] : 0;
    int run = 0;
    for (int i = 0; i < nb; ++i) {
      const unsigned m = __ballot_sync(0xffffffffu, lo <= f0 + i && f0 + i < hi);
      if (tid == 0) {
        sm.rmask[i] = m;
        sm.rsp[i] = run;
      }
      run += __popc(m);
    }
    if (tid == 0) sm.rsp[nb] = run;
  }
  for (int idx = tid; idx < (nb + 1) * 6; idx += blockDim.x) {
    const int f = idx / 6, cam = (idx / 3) & 1, k = idx % 3;
    const size_t fh = (size_t)(fo + host), fn = (size_t)(fo + f0 + f);
    if constexpr (kMixed) {
      df d = df_sub(wv.fr_ch[fh * 6 + k], wv.fr_ch[fn * 6 + cam * 3 + k]);
      dc[idx] = d + df_make(wv.fr_cl[fh * 6 + k] - wv.fr_cl[fn * 6 + cam * 3 + k]);
    } else {
      dc[idx] = wv.fr_c[fh * 6 + k] - wv.fr_c[fn * 6 + cam * 3 + k];
    }
  }
  {
    float4 *r4 = reinterpret_cast<float4 *>(rows);
    for (int i = tid; i < (nb + 1) * kRow * SPGO_CHUNK / 2; i += blockDim.x) r4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();

  // phase B: thread per observation
  const int D = pv.p_pair_D[b];
  double *pair_base = reinterpret_cast<double *>(wv.pair_acc) + (size_t)pv.p_pair_off[b] * kJacVals;
  const T lscale = (T)prm.loss_scale;
  const float *res_buf = nullptr, *tcam_buf = nullptr;
  if constexpr (kMixed) {  // the state's residuals and camera-frame points
    res_buf = wv.res + (size_t)wv.lm[b].res_sel * (size_t)pv.O * 4;
    tcam_buf = wv.tcam + (size_t)wv.lm[b].res_sel * (size_t)pv.O * 6;
  }
  for (int64_t base = ob + (tid & ~31); base < oe; base += blockDim.x) {
    const int64_t o = base + lane;
    V H[6], h[3], Xp[3];  // about the pair origin: Xp = X + (c_a - c_lo)
    int key = -1;
#pragma unroll
    for (int k = 0; k < 6; ++k) H[k] = M::zero();
#pragma unroll
    for (int k = 0; k < 3; ++k) h[k] = Xp[k] = M::zero();
    if (o < oe) {
      const int slot = pv.obs_slot[o], n = pv.obs_frame[o], fw = n - f0;
      const T *X = sm.X[slot], *dX = sm.dX[slot];
      const T boost = (prm.near_boost && abs(n - host) < 2) ? T(16) : T(1);
      // rows of both cameras, (left factor) x (right factor) = w^2 u u^T: FP32 weights each by
      // w, FP64 one of them by w^2 (no square root)
      T U[4][3], W[4][3], Rr[4];
      if constexpr (kMixed) {
        const float4 z4 = reinterpret_cast<const float4 *>(res_buf)[o];
        const float2 *tp = reinterpret_cast<const float2 *>(tcam_buf + (size_t)o * 6);
        const float2 a0 = tp[0], a1 = tp[1], a2 = tp[2];
        const float *Rn = FramesT<float>::R(wv, fo + n, 0);
        weighted_rows(prm.loss, lscale, boost, intr[0], intr[1], Rn, a0.x, a0.y, a1.x, z4.x, z4.y, W, Rr);
        weighted_rows(prm.loss, lscale, boost, intr[4], intr[5], Rn + 9, a1.y, a2.x, a2.y, z4.z, z4.w, W + 2, Rr + 2);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < 3; ++k) U[q][k] = W[q][k];
      } else {
        const float4 z4 = reinterpret_cast<const float4 *>(pv.obs_uv)[o];
#pragma unroll
        for (int cam = 0; cam < 2; ++cam) {
          const double *Rn = FramesT<double>::R(wv, fo + n, cam);
          const double fx = (double)intr[4 * cam], fy = (double)intr[4 * cam + 1];
          const double *d = reinterpret_cast<const double *>(dc) + fw * 6 + cam * 3;
          const Vec3<double> t = mulT(Rn, v3<double>(X[0] + d[0], X[1] + d[1], X[2] + d[2]));
          const double iz = 1.0 / t.z;
          const double r0 = (double)(cam ? z4.z : z4.x) - (fx * t.x * iz + (double)intr[4 * cam + 2]);
          const double r1 = (double)(cam ? z4.w : z4.y) - (fy * t.y * iz + (double)intr[4 * cam + 3]);
          double rho;
          const double w2 = boost * robust<double>(prm.loss, lscale, r0 * r0 + r1 * r1, rho);
          const double j00 = fx * iz, j02 = -j00 * t.x * iz, j11 = fy * iz, j12 = -j11 * t.y * iz;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            U[2 * cam][k] = j00 * Rn[3 * k] + j02 * Rn[3 * k + 2];
            U[2 * cam + 1][k] = j11 * Rn[3 * k + 1] + j12 * Rn[3 * k + 2];
            W[2 * cam][k] = w2 * U[2 * cam][k];
            W[2 * cam + 1][k] = w2 * U[2 * cam + 1][k];
          }
          Rr[2 * cam] = r0;
          Rr[2 * cam + 1] = r1;
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = i; j < 3; ++j)
          H[sym3(i, j)] = M::sum4(W[0][i], U[0][j], W[1][i], U[1][j], W[2][i], U[2][j], W[3][i], U[3][j]);
        h[i] = M::sum4(W[0][i], Rr[0], W[1][i], Rr[1], W[2][i], Rr[2], W[3][i], Rr[3]);
      }
      // the landmark's row of this frame: q = H dX and dX . h
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *row_at(fw, k, slot) = M::dot(H[sym3(k, 0)], H[sym3(k, 1)], H[sym3(k, 2)], dX[0], dX[1], dX[2]);
      *row_at(fw, 3, slot) = M::dot(h[0], h[1], h[2], dX[0], dX[1], dX[2]);
      if (n != host) {
        key = n;
        const T sgn = n > host ? T(1) : T(-1);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          h[k] = M::scale(sgn, h[k]);
          Xp[k] = n < host ? M::shift(X[k], dc[fw * 6 + k]) : M::of(X[k]);
        }
      }
    }
    // the 27 pair values in three rounds of 9, staged and summed over the runs of equal
    // target frame into the FP64 pair records
    int *keys = sm.key[tid >> 5];
    keys[lane] = key;
    if (__any_sync(0xffffffffu, key >= 0)) {
      V *st = stage + (size_t)(tid >> 5) * kJacRound * kJacPitch;
      auto wv_at = [&](int i, int j) {  // (X x H[:, j])_i
        return M::cross(Xp[(i + 1) % 3], H[sym3((i + 2) % 3, j)], Xp[(i + 2) % 3], H[sym3((i + 1) % 3, j)]);
      };
      V G[3][3];  // [X]x H
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) G[i][j] = wv_at(i, j);
      auto put = [&](auto v0) {
        constexpr int V0 = decltype(v0)::value;
        auto store = [&](int v, V x) {
          if (v >= V0 && v < V0 + kJacRound) st[(v - V0) * kJacPitch + lane] = x;
        };
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
          for (int j = i; j < 3; ++j)  // [X]x H [X]x^T: row i of G crossed with X
            if (tri6(i, j) >= V0 && tri6(i, j) < V0 + kJacRound)
              store(tri6(i, j), M::cross(Xp[(j + 1) % 3], G[i][(j + 2) % 3], Xp[(j + 2) % 3], G[i][(j + 1) % 3]));
#pragma unroll
          for (int j = 0; j < 3; ++j) store(tri6(i, 3 + j), G[i][j]);
#pragma unroll
          for (int j = i; j < 3; ++j) store(tri6(3 + i, 3 + j), H[sym3(i, j)]);
          if (21 + i >= V0 && 21 + i < V0 + kJacRound)
            store(21 + i, M::cross(Xp[(i + 1) % 3], h[(i + 2) % 3], Xp[(i + 2) % 3], h[(i + 1) % 3]));
          store(24 + i, h[i]);
        }
      };
      put(std::integral_constant<int, 0>{});
      __syncwarp();
      jac_runs<T, 0>(st, keys, lane, host, D, pair_base);
      __syncwarp();
      put(std::integral_constant<int, kJacRound>{});
      __syncwarp();
      jac_runs<T, kJacRound>(st, keys, lane, host, D, pair_base);
      __syncwarp();
      put(std::integral_constant<int, 2 * kJacRound>{});
      __syncwarp();
      jac_runs<T, 2 * kJacRound>(st, keys, lane, host, D, pair_base);
    }
    __syncwarp();
  }
  __syncthreads();

  // phase C.1: thread (landmark, component).  q: the suffix sums over the frames after the
  // host (row i takes the frames beyond i) and the negated prefix sums over those before it
  // (row i takes the frames up to i), in place, and the total; row hi, which belongs to no
  // pose of the window, ends as zero.  Component 3: the total of dX . h is g_a.
  for (int idx = tid; idx < cnt * 4; idx += blockDim.x) {
    const int slot = idx % cnt, k = idx / cnt;
    const int a = host - f0, lo = sm.lo[slot] - f0, hi = sm.hi[slot] - f0;
    V after = M::zero(), before = M::zero();
    V own = *row_at(hi, k, slot);
    *row_at(hi, k, slot) = M::zero();
    for (int i = hi - 1; i >= a; --i) {
      V *p = row_at(i, k, slot);
      after = M::add(after, own);
      own = *p;
      *p = after;
    }
    for (int i = lo; i < a; ++i) {
      V *p = row_at(i, k, slot);
      before = M::add(before, *p);
      *p = M::neg(before);
    }
    const V total = M::add(M::add(after, own), before);  // own: the host's row
    if (k < 3) {
      sm.tot[k][slot] = total;
    } else {
      reinterpret_cast<T *>(wv.ga)[lm0 + slot] = M::round(total);
      if (wv.gaacc) wv.gaacc[lm0 + slot] = M::value(total);
    }
  }
  __syncthreads();
  if (tid < cnt) {
    const T *dX = sm.dX[tid];
    reinterpret_cast<T *>(wv.C)[lm0 + tid] =
        M::round(M::dot(sm.tot[0][tid], sm.tot[1][tid], sm.tot[2][tid], dX[0], dX[1], dX[2]));
  }
  // phase C.2: B_l(i) = [R_i^T (X_i x b) ; R_i^T b], b = the row's sum, X_i = X - (c_i - c_a),
  // for the (landmark, frame) pairs inside the landmark's window [lo, hi) only (about 60 % of
  // the chunk window's pairs), enumerated row by row so that a warp's lanes take different
  // landmarks; each result takes the place of its own b, the other entries are zero
  const int n_in = sm.rsp[nb];
  for (int j = tid; j < n_in; j += blockDim.x) {
    int row = 0;  // the last window row whose pairs start at or before pair j
#pragma unroll
    for (int step = 64; step >= 1; step >>= 1)
      if (row + step < nb && sm.rsp[row + step] <= j) row += step;
    // the landmark: the (j - rsp[row])-th set bit of the row's mask
    unsigned m = sm.rmask[row];
    int r = j - sm.rsp[row], slot = 0;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
      const int n = __popc(m & ((1u << w) - 1u));
      if (r >= n) {
        r -= n;
        m >>= w;
        slot += w;
      }
    }
    V q[3], Xi[3], t[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      q[k] = *row_at(row, k, slot);
      Xi[k] = M::shift(sm.X[slot][k], dc[row * 6 + k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) t[k] = M::cross(Xi[(k + 1) % 3], q[(k + 2) % 3], Xi[(k + 2) % 3], q[(k + 1) % 3]);
    const int fi = fo + f0 + row;
    if constexpr (kMixed) {
      const float *Rh = wv.fr_Rf + (size_t)fi * 18, *Rl = wv.fr_Rl + (size_t)fi * 18;
#pragma unroll
      for (int k = 0; k < 3; ++k) {  // (R^T v)_k, in double-float, rounded once
        const df Bw = df_dot3(Rh[k], Rl[k], Rh[3 + k], Rl[3 + k], Rh[6 + k], Rl[6 + k], t[0], t[1], t[2]);
        const df Bv = df_dot3(Rh[k], Rl[k], Rh[3 + k], Rl[3 + k], Rh[6 + k], Rl[6 + k], q[0], q[1], q[2]);
        *row_at(row, k, slot) = df{Bw.h + Bw.l, Bv.h + Bv.l};  // the pair of FP32 entries k and 3 + k
      }
    } else {
      const double *R = FramesT<double>::R(wv, fi, 0);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        *row_at(row, k, slot) = R[k] * t[0] + R[3 + k] * t[1] + R[6 + k] * t[2];
        *row_at(row, 3 + k, slot) = R[k] * q[0] + R[3 + k] * q[1] + R[6 + k] * q[2];
      }
    }
  }
  __syncthreads();
  // the chunk's slab, every row and all 32 columns (the Schur pass reads them all)
  if constexpr (kMixed) {
    float4 *g4 = reinterpret_cast<float4 *>(reinterpret_cast<float *>(wv.slab) + pv.ch_slab[c]);
    for (int idx = tid; idx < nb * 3 * (SPGO_CHUNK / 4); idx += blockDim.x) {
      const int s = idx % (SPGO_CHUNK / 4), k = (idx / (SPGO_CHUNK / 4)) % 3, i = idx / (3 * SPGO_CHUNK / 4);
      const float4 *p = reinterpret_cast<const float4 *>(row_at(i, k, 4 * s));
      const float4 x = p[0], y = p[1];
      g4[(size_t)(6 * i + k) * (SPGO_CHUNK / 4) + s] = make_float4(x.x, x.z, y.x, y.z);
      g4[(size_t)(6 * i + 3 + k) * (SPGO_CHUNK / 4) + s] = make_float4(x.y, x.w, y.y, y.w);
    }
  } else {
    double *g = reinterpret_cast<double *>(wv.slab) + pv.ch_slab[c];
    const double *s = reinterpret_cast<const double *>(rows);
    for (int idx = tid; idx < 6 * nb * SPGO_CHUNK; idx += blockDim.x) g[idx] = s[idx];
  }
}

template <typename T>
int launch_jacobian(const PlanView &pv, const WorkView &wv, const Params &prm, const double *alpha, int gate,
                    void *stream) {
  if (pv.n_chunks == 0) return 0;
  const int nt = prm.lin_block > 0 ? prm.lin_block : 256;
  const size_t sm = JacLayout<T>(pv.max_nb, nt / 32).total;
  cudaFuncSetAttribute(k_jacobian<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  // all of the unified L1 / shared memory as shared: the resident CTAs fill it
  cudaFuncSetAttribute(k_jacobian<T>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  launch(k_jacobian<T>, pv.n_chunks, nt, sm, (cudaStream_t)stream, pv, wv, prm, alpha, gate);
  ++g_launches;
  return (int)cudaGetLastError();
}

template int launch_jacobian<float>(const PlanView &, const WorkView &, const Params &, const double *, int, void *);
template int launch_jacobian<double>(const PlanView &, const WorkView &, const Params &, const double *, int, void *);

}  // namespace spgo
