// What the Jacobian pass and the refinement's residual pass share: the arithmetic of their
// sums, and the rounded, weighted rows of an observation, which both must form alike (see
// k_jacobian.cu).
#pragma once
#include "kernels.cuh"
#include "dfloat.cuh"

namespace spgo {

// ---- arithmetic of the two paths: V is double, or a double-float (not always normalised:
// the low part may reach a few units in the last place of the high one) ----
template <typename T> struct Num;
template <> struct Num<double> {
  using V = double;
  using Acc = double;
  __device__ static V zero() { return 0.0; }
  __device__ static V of(double x) { return x; }
  __device__ static V sum4(double a0, double b0, double a1, double b1, double a2, double b2, double a3, double b3) {
    return a0 * b0 + a1 * b1 + a2 * b2 + a3 * b3;
  }
  __device__ static V cross(V xa, V a, V xb, V b) { return xa * a - xb * b; }  // xa a - xb b
  __device__ static V dot(V a0, V a1, V a2, double b0, double b1, double b2) { return a0 * b0 + a1 * b1 + a2 * b2; }
  __device__ static V shift(double x, V d) { return x + d; }
  __device__ static V add(V a, V b) { return a + b; }
  __device__ static V sub(V a, V b) { return a - b; }
  __device__ static V neg(V a) { return -a; }
  __device__ static V scale(double s, V a) { return s * a; }
  __device__ static double value(V a) { return a; }
  __device__ static double round(V a) { return a; }
  __device__ static void acc(Acc &s, V a) { s += a; }
  __device__ static double acc_value(Acc s) { return s; }
};
template <> struct Num<float> {
  using V = df;
  using Acc = df_acc;
  __device__ static V zero() { return df{0.f, 0.f}; }
  __device__ static V of(float x) { return df{x, 0.f}; }
  __device__ static V sum4(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
    return sum4_prod(a0, b0, a1, b1, a2, b2, a3, b3);
  }
  __device__ static V cross(V xa, V a, V xb, V b) {
    const df p = two_prod(xa.h, a.h), q = two_prod(xb.h, b.h);
    const df s = two_sum(p.h, -q.h);
    float l = (p.l - q.l) + s.l;
    l = fmaf(xa.h, a.l, l);
    l = fmaf(xa.l, a.h, l);
    l = fmaf(-xb.h, b.l, l);
    l = fmaf(-xb.l, b.h, l);
    return df{s.h, l};
  }
  __device__ static V dot(V a0, V a1, V a2, float b0, float b1, float b2) {
    const df p0 = two_prod(a0.h, b0), p1 = two_prod(a1.h, b1), p2 = two_prod(a2.h, b2);
    const df s01 = two_sum(p0.h, p1.h);
    const df s = two_sum(s01.h, p2.h);
    float l = ((p0.l + p1.l) + (p2.l + s01.l)) + s.l;
    l = fmaf(a0.l, b0, l);
    l = fmaf(a1.l, b1, l);
    l = fmaf(a2.l, b2, l);
    return df{s.h, l};
  }
  __device__ static V shift(float x, V d) {  // x + d, normalised
    const df s = two_sum(x, d.h);
    return fast_two_sum(s.h, s.l + d.l);
  }
  __device__ static V add(V a, V b) { return a + b; }
  __device__ static V sub(V a, V b) { return a - b; }
  __device__ static V neg(V a) { return df{-a.h, -a.l}; }
  __device__ static V scale(float s, V a) { return df{s * a.h, s * a.l}; }  // s = +-1
  __device__ static double value(V a) { return df_to_double(a); }
  __device__ static float round(V a) { return a.h + a.l; }
  __device__ static void acc(Acc &s, V a) { s.add(a.h, a.l); }
  __device__ static double acc_value(const Acc &s) { return df_acc_value(s); }
};

// FP32, one camera: the rows w u (u = dpi/dt R^T, w^2 the robust weight times boost) and the
// weighted residuals w r of the camera-frame point (tx, ty, tz) with residual (r0, r1).  The
// products and sums are spelled out so that every caller rounds alike.
__device__ __forceinline__ void weighted_rows(int loss, float scale, float boost, float fx, float fy, const float *R,
                                              float tx, float ty, float tz, float r0, float r1, float (*W)[3],
                                              float *wr) {
  float rho;
  const float s = fmaf(r1, r1, __fmul_rn(r0, r0));
  const float w = sqrtf(boost * robust<float>(loss, scale, s, rho));
  const float iz = 1.f / tz;
  const float j00 = __fmul_rn(fx, iz), j11 = __fmul_rn(fy, iz);
  const float j02 = -__fmul_rn(__fmul_rn(j00, tx), iz), j12 = -__fmul_rn(__fmul_rn(j11, ty), iz);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    W[0][k] = __fmul_rn(w, fmaf(j02, R[3 * k + 2], __fmul_rn(j00, R[3 * k])));
    W[1][k] = __fmul_rn(w, fmaf(j12, R[3 * k + 2], __fmul_rn(j11, R[3 * k + 1])));
  }
  wr[0] = __fmul_rn(w, r0);
  wr[1] = __fmul_rn(w, r1);
}

}  // namespace spgo
