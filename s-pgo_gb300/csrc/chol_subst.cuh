// Blocked forward / backward substitution with a packed Cholesky factor held in
// shared memory, shared by the batched factorisation (k_solve.cu) and the
// refinement solves of the mixed path (k_refine.cu).
//
// Storage: element (i, j), i >= j, of L at Lm[cb[j] + i] (packed lower triangle,
// column-major: cb[j] = j P - j (j + 1) / 2), but for the 16x16 diagonal blocks: their inverses
// in FP32, their unit factors U(i, j) = L(i, j) / L(j, j) in FP64 (where an inverse would cost
// more than it saves, and with dinv[k] = 1 / L(k, k) besides).
#pragma once
#include "kernels.cuh"
#include "subst_index.h"

namespace spgo {

// 1 / d and 1 / sqrt(d) for an FP64 pivot.  The pivots are the serial chain of a factorisation,
// and one FP64 instruction of a warp, a comparison or a conversion too, holds its quarter of an
// SM for 64 cycles: one third-order Newton step from the FP32 estimate (2^-21 -> 2^-63, then the
// rounding of the step) takes three and five of them, the estimate's argument and result are
// converted by their bits and the pivots tested by their high words.  Pivots out of the
// estimate's range, and those that are no pivots, take the library's functions.
__device__ __forceinline__ bool pivot_ok(double d) {  // 0 < d < inf
  const int h = __double2hiint(d);
  return (h < 0x7ff00000) & ((h > 0) | ((h == 0) & (__double2loint(d) != 0)));
}
__device__ __forceinline__ bool pivot_in_range(double d) {  // 2^-100 <= d < 2^100
  return (unsigned)(__double2hiint(d) - 0x39b00000) < 0x0c800000u;
}
// d truncated to FP32, and back, for values of the pivot range and their (inverse) roots
__device__ __forceinline__ float pivot_float(double d) {
  const unsigned h = (unsigned)(__double2hiint(d) - (896 << 20)), l = (unsigned)__double2loint(d);
  return __uint_as_float((h << 3) | (l >> 29));
}
__device__ __forceinline__ double pivot_double(float f) {
  const unsigned u = __float_as_uint(f);
  return __hiloint2double((int)((u >> 3) + (896u << 20)), (int)(u << 29));
}
__device__ __forceinline__ double rcp_estimate(double d) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(pivot_float(d)));
  return pivot_double(y);
}
__device__ __forceinline__ double rcp_pivot(double d) {
  if (!pivot_in_range(d)) return 1.0 / d;
  const double y = rcp_estimate(d), e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt_pivot(double d) {
  if (!pivot_in_range(d)) return 1.0 / sqrt(d);
  const double y = pivot_double(rsqrtf(pivot_float(d))), e = fma(-(d * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// Solves L L^T w = y in place (y in shared memory) in 16-unknown blocks, one barrier each:
// warp 0 solves a block and then, while the other warps take it out of the unknowns further on,
// takes it out of the next block's itself.  A block costs warp 0 a 16x16 product (FP32, with the
// block's inverse) or a chain of 16 FMAs (FP64, with its unit factor), the barrier and another
// 16x16 product; everything it reads of L is loaded before the barrier it would wait at anyway.
// Bound by that chain (60 unknowns, FP32: 17.2k cycles with a chain through 1 / L(k, k) per unknown
// and two barriers per block, 7.4k so, 2k of them the first pass through the code).  Every thread of the CTA must call it, with y and
// the factor visible to all.
template <typename T>
__device__ void chol_substitute(const T *Lm, const int *cb, T *y, const T *dinv, int P) {
#define ix(i, j) (cb[(j)] + (i))
  constexpr bool kUnit = sizeof(T) == 8;
  constexpr int kHalf = kPanel / 2, kD = kUnit ? kPanel : kHalf;
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int i = lane & 15, h = (lane >> 4) * kHalf;  // lanes (i, h): unknown i, terms h .. h + 7
  const unsigned all = 0xffffffffu;
  // (loads are unconditional, their values selected: a predicated load costs a branch.  Rows past a
  // narrow last block reach up to kPanel elements behind the factor and y; columns past it are
  // its last column's, subst_index.h.)
  T d[kD], s[kHalf], v = T(0);  // warp 0: the block to solve, the block between it and the next, its right-hand side
  // sum over the 16 lanes' u of the coefficients c
  auto product = [&](const T (&c)[kHalf], T u) {
    T acc = T(0);
#pragma unroll
    for (int q = 0; q < kHalf; ++q) acc += c[q] * __shfl_sync(all, u, h + q);
    return acc + __shfl_xor_sync(all, acc, 16);
  };
  // forward L z = y
  auto load_fwd = [&](int kb, int w) {
    const int c0 = kUnit ? 0 : h;
    const T *B = Lm + ix(kb + i, kb) + subst_fwd_first(P, kb, c0);
#pragma unroll
    for (int q = 0; q < kD; ++q) {
      const T x = *B;
      d[q] = i < w && c0 + q < i + (kUnit ? 0 : 1) ? x : T(0);
      B += subst_fwd_step(P, kb, c0 + q);
    }
  };
  if (warp == 0) {
    load_fwd(0, min(kPanel, P));
    v = i < P ? y[i] : T(0);
  }
  for (int kb = 0; kb < P; kb += kPanel) {
    const int ke = min(kb + kPanel, P), w = ke - kb;
    if (warp == 0) {
      if constexpr (kUnit) {
#pragma unroll
        for (int c = 0; c < kPanel - 1; ++c) v -= d[c] * __shfl_sync(all, v, c);
        v *= i < w ? dinv[kb + i] : T(0);
      } else {
        v = product(d, v);
      }
      if (lane < w) y[kb + lane] = v;
      if (ke < P) {
        load_fwd(ke, min(kPanel, P - ke));
        const T *B = Lm + ix(ke + i, kb) + subst_col(P, kb, h);
#pragma unroll
        for (int q = 0; q < kHalf; ++q) {
          const T x = *B;
          s[q] = ke + i < P ? x : T(0);
          B += P - kb - 1 - h - q;
        }
      }
    }
    __syncthreads();
    if (ke >= P) break;
    if (warp == 0) {
      const T yn = ke + i < P ? y[ke + i] : T(0);
      v = yn - product(s, v);
    } else {
      for (int r = ke + kPanel + tid - 32; r < P; r += nt - 32) {
        const T *B = Lm + ix(r, kb);
        T a0 = T(0), a1 = T(0);
#pragma unroll
        for (int c = 0; c < kPanel; c += 2) {
          a0 += B[0] * y[kb + c];
          a1 += B[P - kb - 1 - c] * y[kb + c + 1];
          B += 2 * (P - kb - c) - 3;
        }
        y[r] -= a0 + a1;
      }
    }
  }
  // backward L^T w = z, blocks from the bottom (warp 0 still holds the last one's z)
  auto load_bwd = [&](int kb, int w) {
    const T *B = Lm + (i < w ? ix(kb, kb + i) : 0);
#pragma unroll
    for (int q = 0; q < kD; ++q) {
      const int r = kUnit ? q : h + q;
      const T x = B[r];
      d[q] = r < w && r + (kUnit ? 0 : 1) > i ? x : T(0);
    }
  };
  const int last = ((P - 1) / kPanel) * kPanel;
  if (warp == 0) load_bwd(last, P - last);
  for (int kb = last;; kb -= kPanel) {
    const int w = min(kPanel, P - kb);
    if (warp == 0) {
      if constexpr (kUnit) {
        v *= i < w ? dinv[kb + i] : T(0);
#pragma unroll
        for (int r = kPanel - 1; r > 0; --r) v -= d[r] * __shfl_sync(all, v, r);
      } else {
        v = product(d, v);
      }
      if (lane < w) y[kb + lane] = v;
      if (kb > 0) {
        load_bwd(kb - kPanel, kPanel);
        const T *B = Lm + ix(kb + h, kb - kPanel + i);
#pragma unroll
        for (int q = 0; q < kHalf; ++q) {
          const T x = B[q];
          s[q] = h + q < w ? x : T(0);
        }
      }
    }
    __syncthreads();
    if (kb == 0) break;
    if (warp == 0) {
      v = y[kb - kPanel + i] - product(s, v);
    } else {
      for (int c = tid - 32; c < kb - kPanel; c += nt - 32) {
        const T *B = Lm + ix(kb, c);
        T a0 = T(0), a1 = T(0);
#pragma unroll
        for (int r = 0; r < kPanel; r += 2) {
          const T x0 = B[r], x1 = B[r + 1], y0 = y[kb + r], y1 = y[kb + r + 1];
          a0 += r < w ? x0 * y0 : T(0);
          a1 += r + 1 < w ? x1 * y1 : T(0);
        }
        y[c] -= a0 + a1;
      }
    }
  }
#undef ix
}

}  // namespace spgo
