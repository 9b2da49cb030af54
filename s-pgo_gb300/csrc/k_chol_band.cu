// Banded Cholesky and substitutions for large reduced camera systems (mixed path).
//
// A landmark's window spans at most D = p_pair_D pose blocks, so S(i, j) = 0 for
// |i - j| > 6 D - 1 and the Cholesky factor keeps that band.  For the wide problems (500
// poses, windows of 20) that is a band of 119 in a 3000-wide matrix: 43 MFLOP instead of
// 9 GFLOP, and what is left is the serial chain of 3000 pivots.  So one problem takes two
// CTAs (a cluster) that eliminate from both ends towards a middle of h 16-wide blocks,
// h = the band's width in blocks (two ends that far apart do not couple, and neither adds
// fill), and the first CTA adds the second's middle to its own and factors it.
//
//   k_band_assemble  S = A + lam diag(A) - S_L inside the band as 16x16 blocks, block column
//                  by block column for each end (the place its factor takes later); clears
//                  what it read of S_L, and g_L after g0 = g - g_L
//   k_band_factor  right-looking on the blocks.  The h + 2 live block rows sit in shared
//                  memory as packed unordered pairs of (row mod C, column mod C), so a new
//                  block row (cp.async, straight into place) replaces the one that retired
//                  without moving anything.  Warp 0 runs the chain: it factors the 32x16
//                  panel of a diagonal block and the block below it (lane = row) and applies
//                  it to the next diagonal block; the other warps solve the remaining rows,
//                  update the rest and invert the diagonal blocks (for the substitutions).
//                  Two barriers per block column.
//   k_band_solve   forward from both ends, the middle, backward to both ends; a block
//                  column of L is one contiguous stretch (cp.async, four columns ahead),
//                  the diagonal blocks act through their inverses.  Warp 0 carries the
//                  solution from block to block in registers, the other warps apply it
//                  to the blocks further away: one barrier per block.
//
// The second CTA works on the reversed problem: local scalar s stands for global scalar
// 16 nB - 1 - s, nB = ceil(P / 16); the scalars from P on are padded with the identity.
// Bound by the serial chain (a 32x16 panel alone takes 1350 cycles, 85 a pivot) and, beside
// it, by shared-memory reads of the updates.  Measured on one GB300 against the dense
// multi-CTA path it replaces: factor of a 3000-wide system with a band of 119, 3.1 ms ->
// 0.31 ms; its solves, 390 -> 109 us; 600 wide with a band of 245, 540 -> 178 us and 81 -> 38 us.
// (Shuffles instead of xs in the panel, 4x4 and 8x8 update tiles, and rows brought in
// through registers were slower.)
#include "kernels.cuh"
#include "dfloat.cuh"

namespace spgo {

constexpr int kBb = 16;                    // block width
constexpr int kBandSlot = kBb * kBb + 16;  // floats per shared block: consecutive slots half a bank row apart
constexpr int kBandThreads = 384;
constexpr int kBandWarps = kBandThreads / 32;
constexpr int kBandTri = SPGO_BAND_MAX_H * (SPGO_BAND_MAX_H + 1) / 2;
constexpr int kBandSolveThreads = 320;     // warp 0 the diagonal blocks, 18 x 16 row threads
constexpr int kBandStages = 5;
// h + 2 = 19 block rows: 190 slots, 207 KB
static_assert((SPGO_BAND_MAX_H + 2) * (SPGO_BAND_MAX_H + 3) / 2 * kBandSlot * 4 <= 220 * 1024, "shared memory");
static_assert((SPGO_BAND_MAX_H + 1) * kBb + 32 <= kBandSolveThreads, "blocks 2..h below the diagonal, and the next");

// the two ends' block counts: [0, mL) from the first, [mR, nB) from the second
struct BandGeo {
  int P, bw, nB, h, mL, mR, nR;
  __host__ __device__ BandGeo(int N, int D) {
    P = 6 * N;
    bw = 6 * D - 1;
    nB = (P + kBb - 1) / kBb;
    h = (bw + kBb - 1) / kBb;
    if (nB > h + 1) {
      mL = (nB - h + 1) / 2;
      mR = mL + h;
    } else {  // one end alone, for a caller with narrow systems: those that come here today have at
              // least 19 block rows, and h is at most 17
      mL = mR = nB;
    }
    nR = nB - mR;
  }
  // first block column of the CTA's factor storage and its step count
  __device__ int base(int e) const { return e ? mR : 0; }
  __device__ int steps(int e) const { return e ? nR : mR; }
  __device__ int last_row(int e) const { return e ? nR + h - 1 : mR - 1; }
  __device__ int global(int e, int s) const { return e ? kBb * nB - 1 - s : s; }
};

size_t band_factor_floats(int N, int D) {
  const BandGeo g(N, D);
  return (size_t)g.nB * (g.h + 1) * kBb * kBb;
}

__device__ __forceinline__ uint32_t bd_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ int bd_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ void bd_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t bd_peer(const void *p, int rank) {  // the peer CTA's copy of a shared address
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(bd_smem(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float bd_peer_load(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void bd_peer_raise(const int *flag, int rank) {
  asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(bd_peer(flag, rank)), "r"(1) : "memory");
}
__device__ __forceinline__ uint64_t bd_clock_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// waits for the peer's flag in this CTA's shared memory, at most until the deadline
__device__ __forceinline__ bool bd_wait(const int *flag, uint64_t deadline) {
  for (;;) {
    int v;
    asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(bd_smem(flag)) : "memory");
    if (v) return true;
    if (bd_clock_ns() > deadline) return false;
    __nanosleep(40);
  }
}

// shared slot of the block of rows and columns a, b (block indices mod C): distinct for
// every pair of live rows
__device__ __forceinline__ int bd_slot(int a, int b) {
  const int hi = max(a, b), lo = min(a, b);
  return (hi * (hi + 1) / 2 + lo) * kBandSlot;
}

// C -= L_r L_c^T on a 16x16 block, TM x TN outputs a thread (t = 0 .. 256 / (TM TN) - 1);
// blocks are column-major, 16 rows a column
template <int TM, int TN>
__device__ __forceinline__ void bd_update(float *Cb, const float *Lr, const float *Lc, int t) {
  const int ty = TM * (t % (kBb / TM)), tx = TN * (t / (kBb / TM));
  float acc[TN][TM];
#pragma unroll
  for (int j = 0; j < TN; ++j)
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[j][i] = 0.f;
#pragma unroll
  for (int k = 0; k < kBb; ++k) {
    float av[TM], cv[TN];
#pragma unroll
    for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4 *>(av + i) = *reinterpret_cast<const float4 *>(Lr + k * kBb + ty + i);
    if constexpr (TN == 2) {
      *reinterpret_cast<float2 *>(cv) = *reinterpret_cast<const float2 *>(Lc + k * kBb + tx);
    } else {
#pragma unroll
      for (int j = 0; j < TN; j += 4) *reinterpret_cast<float4 *>(cv + j) = *reinterpret_cast<const float4 *>(Lc + k * kBb + tx + j);
    }
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int i = 0; i < TM; ++i) acc[j][i] = fmaf(av[i], cv[j], acc[j][i]);
  }
#pragma unroll
  for (int j = 0; j < TN; ++j)
#pragma unroll
    for (int i = 0; i < TM; i += 4) {
      float4 *p = reinterpret_cast<float4 *>(Cb + (tx + j) * kBb + ty + i);
      float4 v = *p;
      v.x -= acc[j][i];
      v.y -= acc[j][i + 1];
      v.z -= acc[j][i + 2];
      v.w -= acc[j][i + 3];
      *p = v;
    }
}

// one warp: the 32x16 panel of a diagonal block B (Cholesky, lanes 0..15 = its rows) and the
// block X below it (X L^-T, lanes 16..31, when `below`).  Four columns at a time: every lane
// takes the 4x4 pivot block by shuffles and factors it redundantly, so the serial chain per
// column is a reciprocal square root and a few FMAs with no shuffle in it; the rows' entries
// and the rank-4 update (the other rows' entries through xs) follow.  Returns whether every
// pivot was positive.
__device__ __forceinline__ bool bd_panel(float *B, float *X, bool below, float *rinv_out, float *xs, int lane) {
  const int i = lane & 15;
  float *mine = (lane < kBb ? B : X) + i;
  float a[kBb];
#pragma unroll
  for (int j = 0; j < kBb; ++j) a[j] = lane < kBb || below ? mine[j * kBb] : 0.f;
  bool ok = true;
  auto rsq = [&](float d) {  // 1 / sqrt(d): the hardware estimate and one Newton step (NaN unless 0 < d < inf)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float t = d * r;
    r = fmaf(0.5f * r, fmaf(-t, r, 1.f), r);
    ok = ok && r > 0.f;
    return r;
  };
#pragma unroll
  for (int k = 0; k < kBb; k += 4) {
    float g[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int s = 0; s <= q; ++s) g[q][s] = __shfl_sync(0xffffffffu, a[k + s], k + q);
    const float r0 = rsq(g[0][0]);
    const float l10 = g[1][0] * r0, l20 = g[2][0] * r0, l30 = g[3][0] * r0;
    const float r1 = rsq(fmaf(-l10, l10, g[1][1]));
    const float l21 = fmaf(-l20, l10, g[2][1]) * r1, l31 = fmaf(-l30, l10, g[3][1]) * r1;
    const float r2 = rsq(fmaf(-l21, l21, fmaf(-l20, l20, g[2][2])));
    const float l32 = fmaf(-l31, l21, fmaf(-l30, l20, g[3][2])) * r2;
    const float r3 = rsq(fmaf(-l32, l32, fmaf(-l31, l31, fmaf(-l30, l30, g[3][3]))));
    // this row's entries of the four columns (rows above them compute values nobody reads)
    const float x0 = a[k] * r0;
    const float x1 = fmaf(-x0, l10, a[k + 1]) * r1;
    const float x2 = fmaf(-x1, l21, fmaf(-x0, l20, a[k + 2])) * r2;
    const float x3 = fmaf(-x2, l32, fmaf(-x1, l31, fmaf(-x0, l30, a[k + 3]))) * r3;
    a[k] = x0;
    a[k + 1] = x1;
    a[k + 2] = x2;
    a[k + 3] = x3;
    if (lane < 4) rinv_out[k + lane] = lane == 0 ? r0 : lane == 1 ? r1 : lane == 2 ? r2 : r3;
    if (k + 4 < kBb) {
      float *xk = xs + (k & 4) * 16;  // (double-buffered: one warp barrier per four columns)
      if (lane < kBb) *reinterpret_cast<float4 *>(xk + 4 * lane) = make_float4(x0, x1, x2, x3);
      __syncwarp();
#pragma unroll
      for (int j = k + 4; j < kBb; ++j) {
        const float4 y = *reinterpret_cast<const float4 *>(xk + 4 * j);
        a[j] = fmaf(-x3, y.w, fmaf(-x2, y.z, fmaf(-x1, y.y, fmaf(-x0, y.x, a[j]))));
      }
    }
  }
  if (lane < kBb || below) {
#pragma unroll
    for (int j = 0; j < kBb; ++j) mine[j * kBb] = a[j];
  }
  return ok;
}

// one warp: column j = lane (< 16) of the inverse of the 16x16 lower factor, to global
__device__ __forceinline__ void bd_invert_diag(const float *B, const float *rinv, float *dst, int lane) {
  if (lane >= kBb) return;
  float x[kBb];
#pragma unroll
  for (int i = 0; i < kBb; ++i) x[i] = i == lane ? 1.f : 0.f;
#pragma unroll
  for (int m = 0; m < kBb; ++m) {
    x[m] *= rinv[m];
#pragma unroll
    for (int i = m + 1; i < kBb; ++i) x[i] = fmaf(-x[m], B[m * kBb + i], x[i]);
  }
#pragma unroll
  for (int i = 0; i < kBb; i += 4)
    *reinterpret_cast<float4 *>(dst + lane * kBb + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
}

// one CTA per block column of each end.  sx: also the exact S (hi, lo), both triangles, for
// the residual of the reduced solve's own refinement.
__global__ void __launch_bounds__(256) k_band_assemble(PlanView pv, WorkView wv, int b, int sx) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  const BandGeo geo(pv.p_npose[b], pv.p_pair_D[b]);
  const int e = (int)blockIdx.x >= geo.mR, c = (int)blockIdx.x - geo.base(e);
  const int P = geo.P, h = geo.h, po = pv.p_param_off[b];
  const size_t off = pv.p_S_off[b];
  const float *A = reinterpret_cast<const float *>(wv.A) + off;
  float *SL = reinterpret_cast<float *>(wv.SL) + off;
  float *dst = reinterpret_cast<float *>(wv.fac) + off + (size_t)blockIdx.x * (h + 1) * kBb * kBb;
  float2 *Sx = reinterpret_cast<float2 *>(wv.Sx) + off;
  const double lam = wv.lm[b].lam;
  for (int t = threadIdx.x; t < (h + 1) * kBb * kBb; t += blockDim.x) {
    // the contiguous direction of the row-major A: columns for the first end, rows (reversed) for the second
    const int d = t / (kBb * kBb), u = (t / kBb) % kBb, v = t % kBb, i = e ? v : u, j = e ? u : v;
    const int sr = geo.global(e, kBb * (c + d) + i), sc = geo.global(e, kBb * c + j);
    const int hi = max(sr, sc), lo = min(sr, sc);
    float val = sr == sc ? 1.f : 0.f;  // the padding
    if (sr >= 0 && sc >= 0 && hi < P) {
      val = 0.f;
      // every element of S has one owner, which clears it: not the upper triangle of a diagonal
      // block, nor what couples the middle to the second end, which that end's columns hold
      const bool other = (d == 0 && i < j) || (!e && c + d >= geo.mR);
      if (hi - lo <= geo.bw && !other) {
        const size_t k = (size_t)hi * P + lo;
        const float a = A[k], sl = SL[k];
        SL[k] = 0.f;
        val = a - sl;
        if (hi == lo) val += (float)lam * a;
        if (sx) {
          df x = df_sub(a, sl);
          if (hi == lo) x = x + df_from_double(lam * (double)a);
          Sx[k] = Sx[(size_t)lo * P + hi] = make_float2(x.h, x.l);
        }
      }
    }
    dst[d * kBb * kBb + j * kBb + i] = val;
  }
  if (threadIdx.x < kBb) {
    const int g = geo.global(e, kBb * c + threadIdx.x);
    if (g < P) {
      float *gL = reinterpret_cast<float *>(wv.gL) + po;
      wv.lg_g0[po + g] = (double)reinterpret_cast<const float *>(wv.g)[po + g] - (double)gL[g];
      gL[g] = 0.f;
    }
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBandThreads) k_band_factor(PlanView pv, WorkView wv, int b,
                                                                                        uint64_t wait_ns) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  extern __shared__ __align__(16) float blocks[];
  __shared__ float rinv[2][kBb];
  __shared__ __align__(16) float xs[4 * 2 * kBb];
  __shared__ unsigned char tri_r[kBandTri], tri_c[kBandTri];
  __shared__ int peer_done, bad, timed_out;
  const BandGeo geo(pv.p_npose[b], pv.p_pair_D[b]);
  const int e = bd_rank();
  const int h = geo.h, C = h + 2, K = geo.steps(e), last = geo.last_row(e);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col = (h + 1) * kBb * kBb;  // one block column in global memory
  float *fac = reinterpret_cast<float *>(wv.fac) + pv.p_S_off[b] + (size_t)geo.base(e) * col;
  const uint64_t deadline = bd_clock_ns() + wait_ns;
  if (tid == 0) peer_done = bad = timed_out = 0;
  // what the second CTA adds to the middle, h (h + 1) / 2 blocks (a wide problem has no other
  // use for its part of facs)
  float *middle = wv.facs + pv.p_S_off[b];
  // S(r, c), absolute block indices, into its slot: by 64 threads, 16 bytes each.  The second
  // CTA's middle-middle blocks start from zero (they only collect its updates).
  auto bring = [&](int r, int c, int t) {
    float *dst = blocks + bd_slot(r % C, c % C) + 4 * t;
    if (e && c >= geo.nR)
      *reinterpret_cast<float4 *>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    else
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(bd_smem(dst)),
                   "l"(fac + (size_t)c * col + (r - c) * kBb * kBb + 4 * t)
                   : "memory");
  };
  for (int r = 0; r <= min(h, last); ++r)
    for (int t = tid; t < 64 * (r + 1); t += kBandThreads) bring(r, t >> 6, t & 63);
  asm volatile("cp.async.wait_all;" ::: "memory");
  for (int t = tid; t < kBandTri; t += kBandThreads) {  // t -> (r >= c) of a lower triangle
    int r = 0;
    while ((r + 1) * (r + 2) / 2 <= t) ++r;
    tri_r[t] = (unsigned char)r;
    tri_c[t] = (unsigned char)(t - r * (r + 1) / 2);
  }
  bd_cluster_sync();  // (also before the peer may raise a flag here)
  if (K > 0 && warp == 0 &&
      !bd_panel(blocks + bd_slot(0, 0), blocks + bd_slot(1, 0), last >= 1, rinv[0], xs, lane))
    bad = 1;
  __syncthreads();

  int km = 0;  // k mod C
  for (int k = 0; k < K; ++k, km = km + 1 == C ? 0 : km + 1) {
    const int nr = min(h, last - k);
    auto at = [&](int r, int c) {  // block (k + r, k + c)
      const int a = km + r, d = km + c;
      return blocks + bd_slot(a >= C ? a - C : a, d >= C ? d - C : d);
    };
    const float *Ld = at(0, 0);
    const float *ri = rinv[k & 1];
    float *fk = fac + (size_t)k * col;
    if (warp == 0) {
      if (nr >= 1) bd_update<4, 2>(at(1, 1), at(1, 0), at(1, 0), lane);  // the next diagonal block
    } else {
      if (k + 1 + h <= last)  // the block row that enters at the next step (its slots: row k - 1's, retired a step ago)
        for (int t = tid - 32; t < 64 * (h + 1); t += kBandThreads - 32) bring(k + 1 + h, k + 1 + (t >> 6), t & 63);
      // the rows of blocks 2.. below: L(r, k) = S(r, k) L_kk^-T, right-looking
      const int d = 2 + (tid - 32) / kBb, i = tid % kBb;
      if (d <= nr) {
        float *B = at(d, 0) + i;
        float x[kBb];
#pragma unroll
        for (int c = 0; c < kBb; ++c) x[c] = B[c * kBb];
#pragma unroll
        for (int c = 0; c < kBb; ++c) {
          x[c] *= ri[c];
#pragma unroll
          for (int q = (c + 1) / 4; q < kBb / 4; ++q) {
            const float4 l = *reinterpret_cast<const float4 *>(Ld + c * kBb + 4 * q);
            const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
            for (int m = 0; m < 4; ++m)
              if (4 * q + m > c) x[4 * q + m] = fmaf(-x[c], lv[m], x[4 * q + m]);
          }
        }
#pragma unroll
        for (int c = 0; c < kBb; ++c) {
          B[c * kBb] = x[c];
          fk[(size_t)d * kBb * kBb + c * kBb + i] = x[c];
        }
      }
    }
    if (h == 1) asm volatile("cp.async.wait_all;" ::: "memory");  // (then warp 0 reads the new row right away)
    __syncthreads();
    const bool merge = e == 0 && geo.nR > 0 && k == geo.mL - 1;  // the next column is the middle's first
    if (warp == 0) {
      if (nr >= 2) bd_update<4, 2>(at(2, 1), at(2, 0), at(1, 0), lane);
      __syncwarp();
      if (!merge && k + 1 < K &&
          !bd_panel(at(1, 1), at(2, 1), k + 2 <= last, rinv[(k + 1) & 1], xs, lane))
        bad = 1;
    } else {
      // blocks (r, c), 1 <= c <= r <= nr, without the two warp 0 updated, 8 threads a block (a
      // quarter-warp reads one block: no bank conflicts).  Warps 4 and 8 share warp 0's
      // scheduler: they only join where the updates, not the chain, set the pace.
      const bool light = (warp & 3) == 0;
      if (warp == 8) bd_invert_diag(Ld, ri, fk, lane);
      if (warp == 4 && nr >= 1)  // the block warp 0 solved, to global memory
        for (int t = lane; t < kBb * kBb / 4; t += 32)
          reinterpret_cast<float4 *>(fk + kBb * kBb)[t] = reinterpret_cast<const float4 *>(at(1, 0))[t];
      const int nt = nr * (nr + 1) / 2;
      const bool all = nt > 72;
      if (!light || all) {
        const int w = all ? warp - 1 : warp - 1 - (warp >> 2), nw = all ? kBandWarps - 1 : 9;
        for (int t = 2 + 4 * w + (lane >> 3); t < nt; t += 4 * nw) {
          const int r = 1 + tri_r[t], c = 1 + tri_c[t];
          bd_update<8, 4>(at(r, c), at(r, 0), at(c, 0), lane & 7);
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (merge) {
      if (tid == 0 && !bd_wait(&peer_done, deadline)) timed_out = 1;
      __syncthreads();
      if (!timed_out)
        for (int t = tid; t < h * (h + 1) / 2 * (kBb * kBb / 4); t += kBandThreads) {
          const int q = t / (kBb * kBb / 4);
          float4 *p = reinterpret_cast<float4 *>(at(1 + tri_r[q], 1 + tri_c[q])) + t % (kBb * kBb / 4);
          const float4 m = __ldcg(reinterpret_cast<const float4 *>(middle) + t);
          float4 v = *p;
          v.x += m.x;
          v.y += m.y;
          v.z += m.z;
          v.w += m.w;
          *p = v;
        }
      __syncthreads();
      if (warp == 0 && !bd_panel(at(1, 1), at(2, 1), k + 2 <= last, rinv[(k + 1) & 1], xs, lane))
        bad = 1;
      __syncthreads();
    }
  }
  if (e == 1 && K > 0) {
    // the middle blocks in the first CTA's order and orientation: its block (u, v), element
    // (i, j) is this one's (v', u'), (15 - j, 15 - i)
    for (int t = tid; t < h * (h + 1) / 2 * kBb * kBb; t += kBandThreads) {
      const int q = t / (kBb * kBb), j = (t / kBb) % kBb, i = t % kBb;
      const int u = geo.nR + h - 1 - tri_r[q], v = geo.nR + h - 1 - tri_c[q];
      middle[t] = blocks[bd_slot(v % C, u % C) + (kBb - 1 - i) * kBb + (kBb - 1 - j)];
    }
    __threadfence();
    __syncthreads();
  }
  if (e == 1 && tid == 0) bd_peer_raise(&peer_done, 0);
  if (tid == 0) {
    if (bad) atomicOr(&wv.lm[b].fail, FAIL_PIVOT);
    if (timed_out) atomicOr(&wv.lm[b].fail, FAIL_TIMEOUT);
  }
  bd_cluster_sync();  // (no flag is raised in a CTA that has left)
}

// shared memory of k_band_solve per stage: h + 1 blocks, the stride half a bank row off
constexpr int kBandBlk = kBb * kBb + 16;

// element (i, c) of a staged block: 16-byte pieces of a column rotated by the column pair,
// so that 16 lanes reading the same piece of 16 columns meet distinct banks
__device__ __forceinline__ int bd_at(int c, int i) { return c * kBb + 4 * ((i >> 2) ^ ((c >> 1) & 3)) + (i & 3); }

// L L^T x = rhs with the factor of k_band_factor; rhs: lg_g0 (first) or lg_y.  Then, as the
// multi-CTA substitutions: accum: delta += x, ddelta = x (a refinement correction); else x is
// added to the solution so far (first: x itself), to delta (last) or lg_x and its split.
// Warp 0: c = lane & 15 is an unknown of the block, and the two half-warps take half of each
// 16-term sum; it forms the next block's value from its own registers while the other warps
// (thread = (block further away, unknown)) apply the block before it.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBandSolveThreads)
    k_band_solve(PlanView pv, WorkView wv, int b, int first, int last, int accum, uint64_t wait_ns) {
  grid_enter();
  if (!problem_active(wv.lm, b, GATE_RUNNING)) return;
  extern __shared__ __align__(16) float stage[];               // [kBandStages][h + 1][kBandBlk]
  __shared__ __align__(16) float ring[(SPGO_BAND_MAX_H + 2) * kBb];  // running right-hand sides, then solutions
  __shared__ float mid[SPGO_BAND_MAX_H * kBb];                 // first CTA: the middle's solution
  __shared__ float part[2][SPGO_BAND_MAX_H * kBb];
  __shared__ __align__(16) float zs[2][kBb];
  __shared__ int peer_done, timed_out;
  const BandGeo geo(pv.p_npose[b], pv.p_pair_D[b]);
  const int e = bd_rank();
  const int P = geo.P, h = geo.h, C = h + 2, K = geo.steps(e), lastr = geo.last_row(e), po = pv.p_param_off[b];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col = (h + 1) * kBb * kBb, stage_len = (h + 1) * kBandBlk;  // one block column, in global and staged
  const float *fac = reinterpret_cast<const float *>(wv.fac) + pv.p_S_off[b] + (size_t)geo.base(e) * col;
  float *z = reinterpret_cast<float *>(wv.lg_y) + po;
  const uint64_t deadline = bd_clock_ns() + wait_ns;
  if (tid == 0) peer_done = timed_out = 0;

  // block column k into its stage: the thread's 16-byte pieces keep their places
  constexpr int kPieces = ((SPGO_BAND_MAX_H + 1) * kBb * kBb / 4 + kBandSolveThreads - 1) / kBandSolveThreads;
  int to[kPieces];
#pragma unroll
  for (int q = 0; q < kPieces; ++q) {
    const int t = tid + q * kBandSolveThreads, d = t / (kBb * kBb / 4), c = (t / 4) % kBb;
    to[q] = d * kBandBlk + bd_at(c, 4 * (t % 4));
  }
  auto fetch = [&](int k, int s) {  // s = k mod kBandStages; every thread commits one group
    if (k >= 0 && k < K) {
      const uint32_t dst = bd_smem(stage + s * stage_len);
      const float *src = fac + (size_t)k * col + 4 * tid;
#pragma unroll
      for (int q = 0; q < kPieces; ++q)
        if (tid + q * kBandSolveThreads < col / 4)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4 * to[q]),
                       "l"(src + 4 * q * kBandSolveThreads)
                       : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto rhs_at = [&](int s) -> float {  // right-hand side at local scalar s (the second CTA's middle starts at zero)
    const int g = geo.global(e, s);
    if (g >= P || (e && s >= kBb * geo.nR)) return 0.f;
    return first ? (float)wv.lg_g0[po + g] : z[g];
  };
  const int hf = lane >> 4, cl = lane & 15;                  // warp 0: half and unknown
  const int d = tid >= 32 ? 1 + (tid - 32) / kBb : 0, i = tid % kBb;  // warps 1..: block 1 + d below the diagonal
  // half of sum_c M(c, unknown) v_c over a staged block M, the v_c of the lanes 0..15; both halves end with the sum
  auto half_rows = [&](const float *M, float v) {  // M's row `cl`
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
      const int c = 8 * hf + q;
      s0 = fmaf(M[bd_at(c, cl)], __shfl_sync(0xffffffffu, v, c), s0);
      s1 = fmaf(M[bd_at(c + 1, cl)], __shfl_sync(0xffffffffu, v, c + 1), s1);
    }
    return s0 + s1;
  };
  auto half_cols = [&](const float *M, float v) {  // M's column `cl`
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = 8 * hf + 4 * q;
      const float4 m = *reinterpret_cast<const float4 *>(M + bd_at(cl, r));
      s0 = fmaf(m.x, __shfl_sync(0xffffffffu, v, r), s0);
      s1 = fmaf(m.y, __shfl_sync(0xffffffffu, v, r + 1), s1);
      s0 = fmaf(m.z, __shfl_sync(0xffffffffu, v, r + 2), s0);
      s1 = fmaf(m.w, __shfl_sync(0xffffffffu, v, r + 3), s1);
    }
    return s0 + s1;
  };
  auto both = [&](float v) { return v + __shfl_xor_sync(0xffffffffu, v, 16); };
  auto keep_z = [&](int k, float v) {  // warp 0: unknown cl of block k
    const int g = geo.global(e, kBb * k + cl);
    if (hf == 0 && g < P) z[g] = v;
  };

  // ---- forward ----
  for (int k = 0; k < kBandStages - 1; ++k) fetch(k, k);
  for (int s = tid; s < kBb * (min(h, lastr) + 1); s += kBandSolveThreads) ring[s] = rhs_at(s);
  float rhs_next = d == h + 1 && h + 1 <= lastr ? rhs_at(kBb * (h + 1) + i) : 0.f;  // the block entering at step 0
  bd_cluster_sync();
  float zk = 0.f;
  int km = 0, ks = 0;  // k mod C, k mod kBandStages
  auto wrap = [&](int a) { return a >= C ? a - C : a; };
  for (int k = 0; k < K; ++k) {
    if (e == 0 && geo.nR > 0 && k == geo.mL - 1) {  // the second end's share of the middle
      __syncthreads();
      if (tid == 0 && !bd_wait(&peer_done, deadline)) timed_out = 1;
      __syncthreads();
      if (!timed_out)
        for (int s = tid; s < h * kBb; s += kBandSolveThreads) {
          const int sp = kBb * geo.nB - 1 - (kBb * geo.mL + s);  // the peer's local scalar
          ring[wrap(km + 1 + s / kBb) * kBb + s % kBb] += bd_peer_load(bd_peer(ring + ((sp / kBb) % C) * kBb + sp % kBb, 1));
        }
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(kBandStages - 3) : "memory");
    __syncthreads();  // columns k and k + 1 staged, z_k and ring[k + 1] final
    fetch(k + kBandStages - 1, ks == 0 ? kBandStages - 1 : ks - 1);
    const float *Lk = stage + ks * stage_len;
    if (warp == 0) {
      if (k == 0) {
        zk = both(half_rows(Lk, ring[cl]));
        if (hf == 0) zs[0][cl] = zk;
        keep_z(0, zk);
      }
    }
    if (k == 0) __syncthreads();
    if (warp == 0) {
      if (k + 1 < K) {
        const float *Ln = stage + (ks + 1 == kBandStages ? 0 : ks + 1) * stage_len;
        const float y = ring[wrap(km + 1) * kBb + cl] - both(half_rows(Lk + kBandBlk, zk));
        zk = both(half_rows(Ln, y));
        if (hf == 0) zs[(k + 1) & 1][cl] = zk;
        keep_z(k + 1, zk);
      } else if (k + 1 <= lastr) {  // the second CTA's last column: the middle's first block
        const float v = both(half_rows(Lk + kBandBlk, zk));
        if (hf == 0) ring[wrap(km + 1) * kBb + cl] -= v;
      }
    } else if (d < h) {
      if (k + 1 + d <= lastr) {
        const float *B = Lk + (1 + d) * kBandBlk;
        const float4 *zp = reinterpret_cast<const float4 *>(zs[k & 1]);
        float v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 zv = zp[q];
          v0 = fmaf(B[bd_at(4 * q, i)], zv.x, v0);
          v1 = fmaf(B[bd_at(4 * q + 1, i)], zv.y, v1);
          v0 = fmaf(B[bd_at(4 * q + 2, i)], zv.z, v0);
          v1 = fmaf(B[bd_at(4 * q + 3, i)], zv.w, v1);
        }
        ring[wrap(km + 1 + d) * kBb + i] -= v0 + v1;
      }
    } else if (d == h + 1) {  // the block that enters now, and the load of the next one
      if (k + 1 + h <= lastr) ring[wrap(km + 1 + h) * kBb + i] = rhs_next;
      rhs_next = k + 2 + h <= lastr ? rhs_at(kBb * (k + 2 + h) + i) : 0.f;
    }
    km = wrap(km + 1);
    ks = ks + 1 == kBandStages ? 0 : ks + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (e == 1 && tid == 0) bd_peer_raise(&peer_done, 0);

  // ---- backward ----
  ks = K > 0 ? (K - 1) % kBandStages : 0;
  km = K > 0 ? (K - 1) % C : 0;
  for (int q = 0; q < kBandStages - 1; ++q) fetch(K - 1 - q, ks >= q ? ks - q : ks - q + kBandStages);
  float xk = 0.f;  // warp 0: the block after k
  if (e == 1 && K > 0) {  // the middle's solution from the first CTA
    if (tid == 0 && !bd_wait(&peer_done, deadline)) timed_out = 1;
    __syncthreads();
    if (!timed_out)
      for (int s = tid; s < h * kBb; s += kBandSolveThreads) {
        const int sm = kBb * geo.nB - 1 - (kBb * geo.nR + s) - kBb * geo.mL;  // its place in the middle
        ring[wrap(km + 1 + s / kBb) * kBb + s % kBb] = bd_peer_load(bd_peer(mid + sm, 0));
      }
    __syncthreads();
    if (warp == 0) xk = ring[wrap(km + 1) * kBb + cl];
  }
  // what the blocks beyond k + 1 contribute to column k (m = k mod C): thread (block, column)
  auto further = [&](int k, int m, const float *Lk) {
    if (d >= 1 && d < h && k >= 0 && k + 1 + d <= lastr) {
      const float *B = Lk + (1 + d) * kBandBlk;
      const float *x = ring + wrap(m + 1 + d) * kBb;
      float v0 = 0.f, v1 = 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 l = *reinterpret_cast<const float4 *>(B + bd_at(i, 4 * q));
        const float4 xv = *reinterpret_cast<const float4 *>(x + 4 * q);
        v0 = fmaf(l.x, xv.x, fmaf(l.z, xv.z, v0));
        v1 = fmaf(l.y, xv.y, fmaf(l.w, xv.w, v1));
      }
      part[k & 1][(d - 1) * kBb + i] = v0 + v1;
    }
  };
  auto load_z = [&](int k) {  // (written by this lane in the forward sweep)
    const int g = k >= 0 ? geo.global(e, kBb * k + cl) : P;
    return warp == 0 && hf == 0 && g < P ? z[g] : 0.f;
  };
  float zn = load_z(K - 1);
  asm volatile("cp.async.wait_group %0;" ::"n"(kBandStages - 2) : "memory");
  __syncthreads();
  further(K - 1, km, stage + ks * stage_len);
  for (int k = K - 1; k >= 0; --k) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kBandStages - 3) : "memory");
    __syncthreads();  // columns k and k - 1 staged, ring[k + 1] and part_k final
    fetch(k - (kBandStages - 1), ks + 1 == kBandStages ? 0 : ks + 1);
    const float *Lk = stage + ks * stage_len;
    const int sp = ks == 0 ? kBandStages - 1 : ks - 1, mp = km == 0 ? C - 1 : km - 1;
    if (warp == 0) {
      const int n = min(h, lastr - k) - 1;  // blocks beyond k + 1
      const float z0 = zn;
      zn = load_z(k - 1);
      float t = z0 - (k + 1 <= lastr ? half_cols(Lk + kBandBlk, xk) : 0.f);
      for (int q = hf; q < n; q += 2) t -= part[k & 1][q * kBb + cl];
      t = both(t);
      xk = both(half_cols(Lk, t));  // x_k = L_kk^-T t
      if (hf == 0) {
        ring[km * kBb + cl] = xk;
        if (e == 0 && geo.nR > 0 && k >= geo.mL) mid[(k - geo.mL) * kBb + cl] = xk;
      }
      keep_z(k, xk);
    } else {
      further(k - 1, mp, stage + sp * stage_len);
    }
    if (e == 0 && geo.nR > 0 && k == geo.mL) {  // the middle is solved: the second end may go on
      __syncthreads();
      if (tid == 0) bd_peer_raise(&peer_done, 1);
    }
    km = mp;
    ks = sp;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int s = tid; s < kBb * K; s += kBandSolveThreads) {
    const int g = geo.global(e, s);
    if (g >= P) continue;
    const double x = (double)z[g];
    if (accum) {
      wv.delta[po + g] += x;
      wv.ddelta[po + g] = x;
    } else {
      const double xi = (first ? 0.0 : wv.lg_x[po + g]) + x;
      if (last) {
        wv.delta[po + g] = xi;
      } else {
        wv.lg_x[po + g] = xi;
        const df sp = df_from_double(xi);
        wv.lg_xs[2 * (po + g)] = sp.h;
        wv.lg_xs[2 * (po + g) + 1] = sp.l;
      }
    }
  }
  if (tid == 0 && timed_out) atomicOr(&wv.lm[b].fail, FAIL_TIMEOUT);
  bd_cluster_sync();  // neither CTA leaves while the other may read its shared memory
}

bool band_route(int N, int D) {
  const BandGeo g(N, D);
  return D >= 1 && g.h <= SPGO_BAND_MAX_H && band_factor_floats(N, D) <= (size_t)g.P * g.P;
}

int launch_band_factor(const PlanView &pv, const WorkView &wv, const Params &prm, int b, int N, int D, int sx,
                       void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const BandGeo g(N, D);
  const size_t sm = (size_t)(g.h + 2) * (g.h + 3) / 2 * kBandSlot * sizeof(float);
  cudaFuncSetAttribute(k_band_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_band_assemble<<<g.nB, 256, 0, st>>>(pv, wv, b, sx);
  k_band_factor<<<2, kBandThreads, sm, st>>>(pv, wv, b, wait_limit_ns(prm));
  g_launches += 2;
  return (int)cudaGetLastError();
}

int launch_band_solve(const PlanView &pv, const WorkView &wv, const Params &prm, int b, int N, int D, int first,
                      int last, int accum, void *stream) {
  const BandGeo g(N, D);
  const size_t sm = (size_t)kBandStages * (g.h + 1) * kBandBlk * sizeof(float);
  cudaFuncSetAttribute(k_band_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_band_solve<<<2, kBandSolveThreads, sm, (cudaStream_t)stream>>>(pv, wv, b, first, last, accum, wait_limit_ns(prm));
  ++g_launches;
  return (int)cudaGetLastError();
}

}  // namespace spgo
