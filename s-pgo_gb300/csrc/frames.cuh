// Frame-table access shared by the linearisation and the pair reduction.
//
// Per frame f and camera (0 left, 1 right) the pose chain writes the
// camera-to-world rotation (FP32 and FP64 copies) and the camera centre (FP64,
// plus a (hi, lo) float pair, from which the mixed path forms relative centres
// without FP64 arithmetic per observation).
#pragma once
#include "kernels.cuh"

namespace spgo {

template <typename T> struct FramesT;
template <> struct FramesT<float> {
  __device__ static const float *R(const WorkView &wv, int f, int cam) { return wv.fr_Rf + (size_t)f * 18 + cam * 9; }
};
template <> struct FramesT<double> {
  __device__ static const double *R(const WorkView &wv, int f, int cam) { return wv.fr_Rd + (size_t)f * 18 + cam * 9; }
  // c(fx, camx) - c(fy, camy)
  __device__ static Vec3<double> rel(const WorkView &wv, int fx, int camx, int fy, int camy) {
    const double *x = wv.fr_c + (size_t)fx * 6 + camx * 3, *y = wv.fr_c + (size_t)fy * 6 + camy * 3;
    return v3<double>(x[0] - y[0], x[1] - y[1], x[2] - y[2]);
  }
};

}  // namespace spgo
