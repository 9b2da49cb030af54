// Large reduced camera systems: problems whose packed factor does not fit in one
// CTA's shared memory (P beyond ~300 in FP32; config 1's 600 and config 2's 3000).
//
// On the mixed path, problems whose windows give S a band of at most 16 SPGO_BAND_MAX_H
// (windows of 45 poses) go to k_chol_band.cu instead; what is below serves the FP64 path and
// the wider bands.
//
// Same mathematics as k_factor_solve (S = A + lam diag(A) - S_L, Cholesky, one
// refinement step with an exact residual), spread over the GPU instead of one CTA:
//   k_lg_assemble  row per CTA: the FP32/T copy of S into the factor storage
//                  (column-major, lower), the exact S (double-float / FP64,
//                  full, row-major) for the residual, g0 = g - g_L; clears S_L, g_L
//   per 64-column panel kb (FP32), as far down as the band of S reaches:
//     k_lg_potrf_rows  one CTA factors the 64x64 diagonal block, one thread per row
//     k_lg_trsm    thread per row below it: L(i, kb:) = S(i, kb:) L_kk^-T
//     k_lg_syrk    one CTA per 64x64 tile of the trailing lower triangle,
//                  C -= L_i L_j^T from shared-memory tiles, 4x4 outputs per thread;
//                  the next panel's tile column first, then (with the solver's second
//                  stream) the next diagonal block beside the rest of the update
//   per 32-column panel (FP64):
//     k_lg_panel   every CTA factors the 32x32 diagonal block, a warp of it solves one
//                  row below
//     k_lg_syrk    one CTA per 16x16 tile of the trailing lower triangle
//   k_lg_fwd/bwd   forward / backward substitution with one CTA per 64-row block,
//                  chained by per-block flags (32-unknown shuffle chains inside each
//                  diagonal block, staged in shared memory while the CTA waits its
//                  turn), x += solution
//   k_lg_resid     warp per row: g0 - S x from the exact S (between two solves)
// Replaces, for such problems, the reference's libtorch Cholesky of the dense
// reduced system (src/Optimization/linear_solvers.cu:195-218).
#include "kernels.cuh"
#include "dfloat.cuh"
#include "chol_subst.cuh"

#include <algorithm>
#include <type_traits>

namespace spgo {

constexpr int kLgNB = 64;  // rows per block of the substitutions

// Panel width and trailing-update tile.  FP64 issues at 1/64 of the FP32 rate, so one warp
// instruction holds its quarter of an SM for 64 cycles: FP64 panels are narrow and their work is
// spread so that a quarter SM has one or two warps of it.
template <typename T> struct LgShape;
template <> struct LgShape<float> { static constexpr int NB = 64, TS = 64; };
template <> struct LgShape<double> { static constexpr int NB = 32, TS = 16; };
constexpr int kLgPanelRows = 4;  // rows (warps) per CTA of k_lg_panel: a whole 32-byte sector of each column

template <typename T> struct ExactS;
template <> struct ExactS<float> { using type = float2; };  // (hi, lo) double-float
template <> struct ExactS<double> { using type = double; };

template <typename T>
__global__ void __launch_bounds__(256) k_lg_assemble(PlanView pv, WorkView wv, int b) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  const int P = 6 * pv.p_npose[b], r = blockIdx.x;
  if (r >= P) return;
  const size_t off = pv.p_S_off[b];
  const T *A = reinterpret_cast<const T *>(wv.A) + off;
  T *SL = reinterpret_cast<T *>(wv.SL) + off;
  T *fac = reinterpret_cast<T *>(wv.fac) + off;
  auto *Sx = reinterpret_cast<typename ExactS<T>::type *>(wv.Sx) + off;
  const double lam = wv.lm[b].lam;
  // S_L may hold entries up to the end of the row's 48-wide SIMT tile (both Schur paths clear here)
  constexpr int TR = 6 * SPGO_TILE_BLOCKS;
  const int cmax = min(P, (r / TR + 1) * TR);
  for (int c = threadIdx.x; c < cmax; c += blockDim.x) {
    if (c <= r) {
      const T a = A[(size_t)r * P + c], sl = SL[(size_t)r * P + c];
      T v = a - sl;
      if (c == r) v += (T)lam * a;
      fac[(size_t)c * P + r] = v;
      if constexpr (std::is_same<T, float>::value) {
        df e = df_sub(a, sl);
        if (c == r) e = e + df_from_double(lam * (double)a);
        Sx[(size_t)r * P + c] = make_float2(e.h, e.l);
        if (c < r) Sx[(size_t)c * P + r] = make_float2(e.h, e.l);
      } else {
        const double e = (double)a - (double)sl + (c == r ? lam * (double)a : 0.0);
        Sx[(size_t)r * P + c] = e;
        if (c < r) Sx[(size_t)c * P + r] = e;
      }
    }
    SL[(size_t)r * P + c] = T(0);
  }
  if (threadIdx.x == 0) {
    const int po = pv.p_param_off[b];
    T *gL = reinterpret_cast<T *>(wv.gL) + po;
    wv.lg_g0[po + r] = (double)reinterpret_cast<const T *>(wv.g)[po + r] - (double)gL[r];
    gL[r] = T(0);
  }
}

// FP64: one 32-column panel.  Every CTA factors the diagonal block for itself (the chain is the
// same length for one CTA or for all, and it saves a launch and the block's way through memory),
// then each warp solves one row below it, lane = column.  Bound by the FP64 pipe of a quarter SM
// (64 cycles per warp instruction), so the chain is counted in such instructions: column k costs
// three for 1 / d_k, one for the column of the unit factor U = a(:, k) / d_k and one per column of
// this warp (j = warp, warp + 4, ..) still to update: 8 on average.  The row solve runs on U too,
// one FMA per column; 1 / sqrt(d) comes in at the end, for all columns at once.  Measured on a 600-wide system with a band of 245:
// diagonal blocks and row solves 1354 us in 32-column panels with one CTA and one row per thread
// (1643 in 64-column ones), 417 us so.
// The diagonal block is kept as U, which the substitutions read, and 1 / L(k, k); U goes to the
// transposed place (the upper triangle: other CTAs may still read S_kk).
__global__ void __launch_bounds__(32 * kLgPanelRows) k_lg_panel(PlanView pv, WorkView wv, int b, int kb) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  constexpr int NB = LgShape<double>::NB, W = kLgPanelRows, C = NB / W;
  static_assert(NB == 32, "lane = row of the diagonal block");
  __shared__ double col[2][NB], U[NB][NB], dd[NB];
  const int P = 6 * pv.p_npose[b], nb = min(NB, P - kb), ke = kb + nb;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *fac = reinterpret_cast<double *>(wv.fac) + pv.p_S_off[b];
  const int row = ke + blockIdx.x * W + warp;
  // (rows below exist only under a full panel)
  double u = row < P ? fac[(size_t)(kb + lane) * P + row] : 0.0;
  double a[C];  // row `lane` of the block, columns warp + W c (narrow last panel: the identity's beyond nb)
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = warp + W * c;
    a[c] = (lane < nb && j <= lane) ? fac[(size_t)(kb + j) * P + kb + lane] : (lane == j ? 1.0 : 0.0);
  }
  bool bad = false;
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    double *ck = col[k & 1];  // (double-buffered: one barrier per column)
    if (warp == k % W) ck[lane] = a[k / W];
    __syncthreads();
    const double d = ck[k];
    bad = bad || !pivot_ok(d);
    const double t = ck[lane] * rcp_pivot(d);  // rows above k: values nobody reads
    if (warp == k % W) {
      U[k][lane] = t;
      if (lane == 0) dd[k] = d;
    }
#pragma unroll
    for (int c = k / W; c < C; ++c)
      if (warp + W * c > k) a[c] = fma(-t, ck[warp + W * c], a[c]);
  }
  __syncthreads();
  const double y = rsqrt_pivot(dd[lane]);
#pragma unroll
  for (int j = 0; j < NB - 1; ++j) {
    const double uj = __shfl_sync(0xffffffffu, u, j);
    if (lane > j) u = fma(-uj, U[j][lane], u);
  }
  if (row < P) fac[(size_t)(kb + lane) * P + row] = u * y;
  if (blockIdx.x != 0) return;
  for (int i = warp; i < nb; i += W)
    if (lane < i) fac[(size_t)(kb + i) * P + kb + lane] = U[lane][i];
  if (warp == 0 && lane < nb) reinterpret_cast<double *>(wv.lg_dinv)[pv.p_param_off[b] + kb + lane] = y;
  if (threadIdx.x == 0 && bad) atomicOr(&wv.lm[b].fail, FAIL_PIVOT);
}

// entry i > j of a diagonal block of the substitutions: of the unit factor U(i, j) =
// L(i, j) / L(j, j) within its 32-wide diagonal parts, of L outside them
template <typename T>
__device__ __forceinline__ T lg_diag(const T *L, const T *dinv, int P, int i, int j) {
  if (i / 32 != j / 32) return L[(size_t)j * P + i];
  if (std::is_same<T, double>::value) return L[(size_t)i * P + j];  // where k_lg_panel put it
  return L[(size_t)j * P + i] * dinv[j];
}

// FP32 path: one CTA of 64 threads factors the 64x64 diagonal block, thread i holding row i of
// the block in registers.  Column k: the threads of rows i >= k put their entry of
// column k into a shared column (double-buffered: one barrier per column), then each
// reads the pivot, and row i > k forms L(i, k) = a(i, k) / L(k, k) and updates its own
// entries j in (k, i]: a(i, j) -= L(i, k) L(j, k), with L(j, k) taken as a(j, k) from
// the shared column times 1 / L(k, k).  The serial part per column is one barrier,
// one square root and one reciprocal; the update is spread over the rows.
__global__ void __launch_bounds__(kLgNB) k_lg_potrf_rows(PlanView pv, WorkView wv, int b, int kb) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  __shared__ float col[2][kLgNB];
  const int P = 6 * pv.p_npose[b], nb = min(kLgNB, P - kb), i = threadIdx.x;
  float *fac = reinterpret_cast<float *>(wv.fac) + pv.p_S_off[b];
  float *dinv = reinterpret_cast<float *>(wv.lg_dinv) + pv.p_param_off[b];
  float a[kLgNB];
#pragma unroll
  for (int j = 0; j < kLgNB; ++j) a[j] = (i < nb && j <= i) ? fac[(size_t)(kb + j) * P + kb + i] : 0.f;
  bool bad = false;
  float rdiag = 0.f;  // 1 / L(i, i)
#pragma unroll
  for (int k = 0; k < kLgNB; ++k) {
    if (k >= nb) break;  // (uniform: a narrow last panel)
    float *c = col[k & 1];
    if (i >= k) c[i] = a[k];
    __syncthreads();
    const float d = c[k];
    bad = bad || !(d > 0.f) || !(d < INFINITY);
    const float lkk = sqrtf(d), rinv = 1.f / lkk;  // correctly rounded
    if (i == k) {
      a[k] = lkk;
      rdiag = rinv;
    } else if (i > k) {
      const float lik = a[k] * rinv;
      a[k] = lik;
      const float s = lik * rinv;  // L(i, k) / L(k, k): times a(j, k) gives L(i, k) L(j, k)
#pragma unroll
      for (int j = k + 1; j < kLgNB; ++j)
        if (j <= i) a[j] -= s * c[j];
    }
  }
  if (i < nb) {
#pragma unroll
    for (int j = 0; j < kLgNB; ++j)
      if (j <= i) fac[(size_t)(kb + j) * P + kb + i] = a[j];
    dinv[kb + i] = rdiag;
  }
  if (bad && i == 0) atomicOr(&wv.lm[b].fail, FAIL_PIVOT);
}

// thread per row below the panel: L(i, kb:ke) = S(i, kb:ke) L_kk^-T, right-looking
// (once x_j is final it is removed from every later column: independent updates
// instead of one dependent chain per column)
__global__ void __launch_bounds__(128) k_lg_trsm(PlanView pv, WorkView wv, int b, int kb) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  __shared__ float D[kLgNB][kLgNB + 1];
  __shared__ float di[kLgNB];
  const int P = 6 * pv.p_npose[b], nb = min(kLgNB, P - kb), ke = kb + nb, tid = threadIdx.x;
  const float *fac_c = reinterpret_cast<const float *>(wv.fac) + pv.p_S_off[b];
  float *fac = reinterpret_cast<float *>(wv.fac) + pv.p_S_off[b];
  const float *dinv = reinterpret_cast<const float *>(wv.lg_dinv) + pv.p_param_off[b];
  for (int idx0 = tid; idx0 < kLgNB * kLgNB; idx0 += 8 * blockDim.x) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {  // loads first
      const int idx = idx0 + q * blockDim.x, i = idx % kLgNB, j = idx / kLgNB;
      v[q] = (idx < kLgNB * kLgNB && i > j && i < nb) ? fac_c[(size_t)(kb + j) * P + kb + i] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int idx = idx0 + q * blockDim.x;
      if (idx < kLgNB * kLgNB) D[idx % kLgNB][idx / kLgNB] = v[q];
    }
  }
  for (int j = tid; j < kLgNB; j += blockDim.x) di[j] = j < nb ? dinv[kb + j] : 0.f;
  __syncthreads();
  const int i = ke + blockIdx.x * blockDim.x + tid;
  if (i >= P) return;
  float x[kLgNB];
#pragma unroll
  for (int j = 0; j < kLgNB; ++j) x[j] = j < nb ? fac_c[(size_t)(kb + j) * P + i] : 0.f;
#pragma unroll
  for (int j = 0; j < kLgNB; ++j) {
    x[j] *= di[j];
#pragma unroll
    for (int m = j + 1; m < kLgNB; ++m) x[m] -= x[j] * D[m][j];
  }
#pragma unroll
  for (int j = 0; j < kLgNB; ++j)
    if (j < nb) fac[(size_t)(kb + j) * P + i] = x[j];
}

// tiles of the trailing lower triangle: mode 0 all of them, mode 1 the first tile column
// (the next panel's columns), mode 2 the others
template <typename T>
__global__ void __launch_bounds__(256) k_lg_syrk(PlanView pv, WorkView wv, int b, int kb, int mode) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  constexpr int NB = LgShape<T>::NB, TS = LgShape<T>::TS, R = TS / 16;
  __shared__ T LR[NB][TS + 1];
  __shared__ T LC[NB][TS + 1];
  const int P = 6 * pv.p_npose[b], nb = min(NB, P - kb), ke = kb + nb, tid = threadIdx.x;
  // tile t -> (ti >= tj)
  int t = blockIdx.x, ti = t, tj = 0;
  if (mode != 1) {
    ti = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    while (ti * (ti + 1) / 2 > t) --ti;
    tj = t - ti * (ti + 1) / 2;
    if (mode == 2) {
      ++ti;
      ++tj;
    }
  }
  const int R0 = ke + TS * ti, C0 = ke + TS * tj;
  T *fac = reinterpret_cast<T *>(wv.fac) + pv.p_S_off[b];
  for (int idx = tid; idx < nb * TS; idx += blockDim.x) {
    const int r = idx % TS, k = idx / TS;
    LR[k][r] = R0 + r < P ? fac[(size_t)(kb + k) * P + R0 + r] : T(0);
    LC[k][r] = C0 + r < P ? fac[(size_t)(kb + k) * P + C0 + r] : T(0);
  }
  __syncthreads();
  const int tx = tid % 16, ty = tid / 16;
  T acc[R][R];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[i][j] = T(0);
  for (int k = 0; k < nb; ++k) {
    T a[R], c[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      a[i] = LR[k][tx + 16 * i];
      c[i] = LC[k][ty + 16 * i];
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < R; ++j) acc[i][j] += a[i] * c[j];
  }
#pragma unroll
  for (int j = 0; j < R; ++j)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = R0 + tx + 16 * i, c = C0 + ty + 16 * j;
      if (r < P && c < P && r >= c) fac[(size_t)c * P + r] -= acc[i][j];
    }
}

// ---- substitutions spread over the GPU: one CTA per 64-row block ----
// Forward L z = r: the CTA of block k adds up L(k, j) z_j for every earlier block j
// as soon as that block's flag is up, then solves its diagonal block and raises its
// own flag; backward L^T x = z the same from the bottom (the CTA of block k waits
// only for blocks finished by lower-numbered CTAs, so the chain never waits on a CTA
// that has not started).  Thread (r, q) handles unknown r of the block and a 16-wide
// quarter q of each other block.  Every wait is bounded (the parameter's limit,
// 2 s by default); a timeout marks the problem failed (the step is rejected and
// counted as a timeout, not as a factorisation failure) and the CTA carries on.

__device__ __forceinline__ uint64_t lg_clock_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool lg_wait_flag(const int *flag, uint64_t deadline) {
  for (int it = 0;; ++it) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v) return true;
    if ((it & 7) == 7 && lg_clock_ns() > deadline) return false;  // (~1 us between looks at the clock)
    __nanosleep(100);
  }
}

__device__ __forceinline__ void lg_set_flag(int *flag) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(flag), "r"(1) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(256) k_lg_fwd(PlanView pv, WorkView wv, int b, int first, uint64_t wait_ns) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  __shared__ T part[4][kLgNB];
  __shared__ T zs[kLgNB];
  // staged while the earlier blocks are still being solved: the diagonal block (strictly lower, its
  // two 32-wide diagonal parts of the unit factor, so that the chain is one shuffle and one FMA per
  // unknown) and the pivots' reciprocals
  __shared__ T Ld[kLgNB][kLgNB + 1];
  __shared__ T ds[kLgNB];
  __shared__ int timed_out;
  const int P = 6 * pv.p_npose[b], po = pv.p_param_off[b];
  const int k = blockIdx.x, kb = k * kLgNB, nb = min(kLgNB, P - kb);
  const int tid = threadIdx.x, r = tid & 63, q = tid >> 6, warp = tid >> 5, lane = tid & 31;
  const T *L = reinterpret_cast<const T *>(wv.fac) + pv.p_S_off[b];
  auto Lat = [&](int i, int j) { return L[(size_t)j * P + i]; };  // L(i, j), i >= j
  const T *dinv = reinterpret_cast<const T *>(wv.lg_dinv) + po;
  T *z = reinterpret_cast<T *>(wv.lg_y) + po;  // in place: this block's right-hand side in, z out
  int *flag = wv.lg_flag + po;
  const uint64_t deadline = lg_clock_ns() + wait_ns;
  if (tid == 0) timed_out = 0;
  for (int idx = tid; idx < kLgNB * kLgNB; idx += blockDim.x) {
    const int i = idx % kLgNB, j = idx / kLgNB;
    Ld[i][j] = (i < nb && j < i) ? lg_diag(L, dinv, P, kb + i, kb + j) : T(0);
  }
  if (tid < kLgNB) ds[tid] = tid < nb ? dinv[kb + tid] : T(0);
  __syncthreads();
  T acc = T(0);
  const int bw = 6 * pv.p_pair_D[b] - 1;  // L(i, j) = 0 for i - j > bw
  for (int j = max(0, kb - bw) / kLgNB; j < k; ++j) {  // earlier blocks are full 64-wide
    // this block's part of L is loaded before the wait for block j's solution
    const int c0 = j * kLgNB + 16 * q;
    T lv[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) lv[c] = r < nb ? Lat(kb + r, c0 + c) : T(0);
    if (tid == 0 && !timed_out && !lg_wait_flag(flag + j, deadline)) timed_out = 1;
    __syncthreads();
    if (r < nb) {
      T zv[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) zv[c] = __ldcg(z + c0 + c);
#pragma unroll
      for (int c = 0; c < 16; ++c) acc += lv[c] * zv[c];
    }
  }
  part[q][r] = acc;
  __syncthreads();
  if (tid < nb) {
    const T rhs = first ? (T)wv.lg_g0[po + kb + tid] : z[kb + tid];
    zs[tid] = rhs - ((part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]));
  }
  __syncthreads();
  if (warp == 0) {  // L_kk z_k = zs: two 32-unknown halves, lane = unknown
    for (int h = 0; h < nb; h += 32) {
      const int w = min(32, nb - h);
      T v = lane < w ? zs[h + lane] : T(0);
      if (h > 0) {  // the first half is final: loads first, four chains
        T lq[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) lq[c] = lane < w ? Ld[h + lane][c] : T(0);
        T v1 = T(0), v2 = T(0), v3 = T(0);
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          v -= lq[c] * zs[c];
          v1 -= lq[c + 1] * zs[c + 1];
          v2 -= lq[c + 2] * zs[c + 2];
          v3 -= lq[c + 3] * zs[c + 3];
        }
        v += (v1 + v2) + v3;
      }
      T lr[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) lr[c] = Ld[h + lane][h + c];
#pragma unroll
      for (int c = 0; c < 31; ++c) v -= lr[c] * __shfl_sync(0xffffffffu, v, c);
      if (lane < w) zs[h + lane] = v * ds[h + lane];
      __syncwarp();
    }
  }
  __syncthreads();
  if (tid < nb) z[kb + tid] = zs[tid];
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    lg_set_flag(flag + k);
    if (timed_out) atomicOr(&wv.lm[b].fail, FAIL_TIMEOUT);
  }
}

// backward L^T x = z (z in place in lg_y); then x is added to the solution so far
// (first: x itself) and written to delta (last) or to lg_x and its split; accum
// (a refinement correction of the mixed path): delta += x and ddelta = x
template <typename T>
__global__ void __launch_bounds__(256) k_lg_bwd(PlanView pv, WorkView wv, int b, int first, int last, int accum,
                                                 uint64_t wait_ns) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  __shared__ T part[4][kLgNB];
  __shared__ T zs[kLgNB];
  // staged while the later blocks are still being solved: the diagonal block (strictly lower, its
  // two 32-wide diagonal parts of the unit factor, so that the chain is one shuffle and one FMA per
  // unknown) and the pivots' reciprocals
  __shared__ T Ld[kLgNB][kLgNB + 1];
  __shared__ T ds[kLgNB];
  __shared__ int timed_out;
  const int P = 6 * pv.p_npose[b], po = pv.p_param_off[b];
  const int nblk = (P + kLgNB - 1) / kLgNB, k = nblk - 1 - (int)blockIdx.x;
  const int kb = k * kLgNB, nb = min(kLgNB, P - kb);
  const int tid = threadIdx.x, r = tid & 63, q = tid >> 6, warp = tid >> 5, lane = tid & 31;
  const T *L = reinterpret_cast<const T *>(wv.fac) + pv.p_S_off[b];
  auto Lat = [&](int i, int j) { return L[(size_t)j * P + i]; };
  const T *dinv = reinterpret_cast<const T *>(wv.lg_dinv) + po;
  T *x = reinterpret_cast<T *>(wv.lg_y) + po;
  int *flag = wv.lg_flag + pv.total_params + po;
  const uint64_t deadline = lg_clock_ns() + wait_ns;
  if (tid == 0) timed_out = 0;
  for (int idx = tid; idx < kLgNB * kLgNB; idx += blockDim.x) {
    const int i = idx % kLgNB, j = idx / kLgNB;
    Ld[i][j] = (i < nb && j < i) ? lg_diag(L, dinv, P, kb + i, kb + j) : T(0);
  }
  if (tid < kLgNB) ds[tid] = tid < nb ? dinv[kb + tid] : T(0);
  __syncthreads();
  T acc = T(0);
  const int bw = 6 * pv.p_pair_D[b] - 1;
  for (int j = min(nblk - 1, (kb + nb - 1 + bw) / kLgNB); j > k; --j) {  // later blocks, finished by lower-numbered CTAs
    // this block's part of L is loaded before the wait for block j's solution
    const int jb = j * kLgNB, nbj = min(kLgNB, P - jb);
    T lv[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int i = 16 * q + c;
      lv[c] = (r < nb && i < nbj) ? Lat(jb + i, kb + r) : T(0);  // column kb + r: contiguous per thread
    }
    if (tid == 0 && !timed_out && !lg_wait_flag(flag + j, deadline)) timed_out = 1;
    __syncthreads();
    if (r < nb) {
      T xv[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const int i = 16 * q + c;
        xv[c] = i < nbj ? __ldcg(x + jb + i) : T(0);
      }
#pragma unroll
      for (int c = 0; c < 16; ++c) acc += lv[c] * xv[c];
    }
  }
  part[q][r] = acc;
  __syncthreads();
  if (tid < nb) zs[tid] = x[kb + tid] - ((part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]));
  __syncthreads();
  if (warp == 0) {  // L_kk^T x_k = zs, halves from the bottom
    for (int h = ((nb - 1) / 32) * 32; h >= 0; h -= 32) {
      const int w = min(32, nb - h);
      T v = lane < w ? zs[h + lane] : T(0);
      if (h + w < nb) {  // the later half is final (h = 0): loads first
        T lq[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) lq[c] = (lane < w && 32 + c < nb) ? Ld[32 + c][h + lane] : T(0);
        T v1 = T(0), v2 = T(0), v3 = T(0);
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          v -= lq[c] * (32 + c < nb ? zs[32 + c] : T(0));
          v1 -= lq[c + 1] * (33 + c < nb ? zs[33 + c] : T(0));
          v2 -= lq[c + 2] * (34 + c < nb ? zs[34 + c] : T(0));
          v3 -= lq[c + 3] * (35 + c < nb ? zs[35 + c] : T(0));
        }
        v += (v1 + v2) + v3;
      }
      T lc[32];  // column `lane` of the diagonal block
#pragma unroll
      for (int c = 0; c < 32; ++c) lc[c] = Ld[h + c][h + lane];
      v *= ds[h + lane];  // U^T x = L_jj^-1 (..)
#pragma unroll
      for (int c = 31; c > 0; --c) v -= lc[c] * __shfl_sync(0xffffffffu, v, c);
      if (lane < w) zs[h + lane] = v;
      __syncwarp();
    }
  }
  __syncthreads();
  if (tid < nb) x[kb + tid] = zs[tid];
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    lg_set_flag(flag + k);
    if (timed_out) atomicOr(&wv.lm[b].fail, FAIL_TIMEOUT);
  }
  if (tid < nb && accum) {
    const int i = kb + tid;
    wv.delta[po + i] += (double)zs[tid];
    wv.ddelta[po + i] = (double)zs[tid];
  } else if (tid < nb) {
    const int i = kb + tid;
    const double xi = (first ? 0.0 : wv.lg_x[po + i]) + (double)zs[tid];
    if (last) {
      wv.delta[po + i] = xi;  // (a failed factorisation zeroes delta after the solve)
    } else {
      wv.lg_x[po + i] = xi;
      const df sp = df_from_double(xi);
      wv.lg_xs[2 * (po + i)] = sp.h;
      wv.lg_xs[2 * (po + i) + 1] = sp.l;
    }
  }
}

// a failed factorisation (or a timed-out substitution) leaves no step.  band: the banded
// assembly cleared S_L inside the band only; what a non-finite 1 / D may have spread beyond
// it (such an S always fails the factor) goes here.
__global__ void k_lg_zero_failed(PlanView pv, WorkView wv, int b, int band) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  if (!wv.lm[b].fail) return;
  const int P = 6 * pv.p_npose[b], po = pv.p_param_off[b];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) wv.delta[po + i] = 0.0;
  if (!band) return;
  float *SL = reinterpret_cast<float *>(wv.SL) + pv.p_S_off[b];
  const size_t n = (size_t)P * P, step = (size_t)gridDim.x * blockDim.x;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) SL[k] = 0.f;
}

// residual y = g0 - S x from the exact S, warp per row
template <typename T>
__global__ void __launch_bounds__(256) k_lg_resid(PlanView pv, WorkView wv, int b) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  const int P = 6 * pv.p_npose[b], po = pv.p_param_off[b];
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= P) return;
  const auto *Sx = reinterpret_cast<const typename ExactS<T>::type *>(wv.Sx) + pv.p_S_off[b] + (size_t)i * P;
  const int bw = 6 * pv.p_pair_D[b] - 1, j0 = max(0, i - bw), j1 = min(P, i + bw + 1);  // S's band
  double r;
  if constexpr (std::is_same<T, float>::value) {
    const float *xs = wv.lg_xs + 2 * (size_t)po;
    df acc = df_make(0.f);
    for (int j = j0 + lane; j < j1; j += 32) {
      const float2 s = Sx[j];
      acc = acc + df{s.x, s.y} * df{xs[2 * j], xs[2 * j + 1]};
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const df other{__shfl_xor_sync(0xffffffffu, acc.h, o), __shfl_xor_sync(0xffffffffu, acc.l, o)};
      acc = acc + other;
    }
    r = (double)acc.h + (double)acc.l;
  } else {
    double acc = 0.0;
    for (int j = j0 + lane; j < j1; j += 32) acc += Sx[j] * wv.lg_x[po + j];
    r = warp_sum(acc);
  }
  if (lane == 0) reinterpret_cast<T *>(wv.lg_y)[po + i] = (T)(wv.lg_g0[po + i] - r);
}

template <typename T>
int launch_factor_large(const PlanView &pv, const WorkView &wv, const Params &prm, int b, int N, int D, int param_off,
                        int refine, void *stream, void *side, void *ev_a, void *ev_b) {
  cudaStream_t st = (cudaStream_t)stream;
  const int P = 6 * N;
  if (std::is_same<T, float>::value && band_route(N, D)) {
    int rc = launch_band_factor(pv, wv, prm, b, N, D, refine > 0, stream);
    for (int it = 0; rc == 0 && it <= refine; ++it) {
      if (it > 0) {
        launch(k_lg_resid<T>, (P + 7) / 8, 256, 0, st, pv, wv, b);
        ++g_launches;
      }
      rc = launch_band_solve(pv, wv, prm, b, N, D, it == 0, it == refine, 0, stream);
    }
    launch(k_lg_zero_failed, grid_for(P, 256), 256, 0, st, pv, wv, b, 1);
    ++g_launches;
    return rc ? rc : (int)cudaGetLastError();
  }
  const uint64_t wait_ns = wait_limit_ns(prm);
  launch(k_lg_assemble<T>, P, 256, 0, st, pv, wv, b);
  int n = 1;
  // (the panels' kernels are launched plainly: CTAs that come in while the kernel before still
  // fills most SMs share the others', and a 600-wide FP64 system took 1.74 ms instead of 1.64)
  constexpr int NB = LgShape<T>::NB, TS = LgShape<T>::TS;
  const int bw = 6 * D - 1;  // S and L are zero beyond it: a panel reaches bw rows down
  if constexpr (std::is_same<T, double>::value) {
    for (int kb = 0; kb < P; kb += NB) {
      const int M = std::min(std::max(P - kb - NB, 0), bw), nt = (M + TS - 1) / TS;
      k_lg_panel<<<std::max(1, (M + kLgPanelRows - 1) / kLgPanelRows), 32 * kLgPanelRows, 0, st>>>(pv, wv, b, kb);
      ++n;
      if (nt > 0) {
        k_lg_syrk<T><<<nt * (nt + 1) / 2, 256, 0, st>>>(pv, wv, b, kb, 0);
        ++n;
      }
    }
  } else {
    // one panel of look-ahead: once panel kb's rows are solved, the next panel's columns take
    // its update first and the next diagonal block is factored on the side stream while the
    // rest of the trailing matrix is updated; every element takes the same updates in the
    // same order as without it
    cudaStream_t sd = (cudaStream_t)side;
    cudaEvent_t ea = (cudaEvent_t)ev_a, eb = (cudaEvent_t)ev_b;
    const bool ahead = sd && ea && eb;
    k_lg_potrf_rows<<<1, kLgNB, 0, st>>>(pv, wv, b, 0);
    ++n;
    for (int kb = 0; kb + NB < P; kb += NB) {
      const int ke = kb + NB, M = std::min(P - ke, bw), nt = (M + TS - 1) / TS;
      k_lg_trsm<<<(M + 127) / 128, 128, 0, st>>>(pv, wv, b, kb);
      n += 3;
      if (!ahead) {
        k_lg_syrk<T><<<nt * (nt + 1) / 2, 256, 0, st>>>(pv, wv, b, kb, 0);
        k_lg_potrf_rows<<<1, kLgNB, 0, st>>>(pv, wv, b, ke);
        continue;
      }
      k_lg_syrk<T><<<nt, 256, 0, st>>>(pv, wv, b, kb, 1);
      cudaError_t e = cudaEventRecord(ea, st);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(sd, ea, 0);
      if (e != cudaSuccess) return (int)e;
      k_lg_potrf_rows<<<1, kLgNB, 0, sd>>>(pv, wv, b, ke);
      if ((e = cudaEventRecord(eb, sd)) != cudaSuccess) return (int)e;
      if (nt > 1) {
        k_lg_syrk<T><<<nt * (nt - 1) / 2, 256, 0, st>>>(pv, wv, b, kb, 2);
        ++n;
      }
      if ((e = cudaStreamWaitEvent(st, eb, 0)) != cudaSuccess) return (int)e;
    }
  }
  const int nblk = (P + kLgNB - 1) / kLgNB;
  int *ff = wv.lg_flag + param_off, *fb = wv.lg_flag + pv.total_params + param_off;
  for (int it = 0; it <= refine; ++it) {
    if (it > 0) {
      launch(k_lg_resid<T>, (P + 7) / 8, 256, 0, st, pv, wv, b);
      ++n;
    }
    cudaError_t e = cudaMemsetAsync(ff, 0, sizeof(int) * (size_t)nblk, st);
    if (e != cudaSuccess) return (int)e;
    launch(k_lg_fwd<T>, nblk, 256, 0, st, pv, wv, b, it == 0, wait_ns);
    e = cudaMemsetAsync(fb, 0, sizeof(int) * (size_t)nblk, st);
    if (e != cudaSuccess) return (int)e;
    launch(k_lg_bwd<T>, nblk, 256, 0, st, pv, wv, b, it == 0, it == refine, 0, wait_ns);
    n += 2;
  }
  launch(k_lg_zero_failed, grid_for(P, 256), 256, 0, st, pv, wv, b, 0);
  ++n;
  g_launches += n;
  return (int)cudaGetLastError();
}

// one refinement correction of the mixed path: the right-hand side is in lg_y
// (k_resid_solve); delta += S^-1 lg_y with the factor of this iteration
int launch_refine_large(const PlanView &pv, const WorkView &wv, const Params &prm, int b, int N, int D, int param_off,
                        void *stream) {
  if (band_route(N, D)) return launch_band_solve(pv, wv, prm, b, N, D, 0, 0, 1, stream);
  cudaStream_t st = (cudaStream_t)stream;
  const int P = 6 * N;
  const uint64_t wait_ns = wait_limit_ns(prm);
  const int nblk = (P + kLgNB - 1) / kLgNB;
  int *ff = wv.lg_flag + param_off, *fb = wv.lg_flag + pv.total_params + param_off;
  cudaError_t e = cudaMemsetAsync(ff, 0, sizeof(int) * (size_t)nblk, st);
  if (e != cudaSuccess) return (int)e;
  launch(k_lg_fwd<float>, nblk, 256, 0, st, pv, wv, b, 0, wait_ns);
  e = cudaMemsetAsync(fb, 0, sizeof(int) * (size_t)nblk, st);
  if (e != cudaSuccess) return (int)e;
  launch(k_lg_bwd<float>, nblk, 256, 0, st, pv, wv, b, 0, 0, 1, wait_ns);
  g_launches += 2;
  return (int)cudaGetLastError();
}

template int launch_factor_large<float>(const PlanView &, const WorkView &, const Params &, int, int, int, int, int,
                                        void *, void *, void *, void *);
template int launch_factor_large<double>(const PlanView &, const WorkView &, const Params &, int, int, int, int, int,
                                         void *, void *, void *, void *);

}  // namespace spgo
