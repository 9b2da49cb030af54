// Addresses of the packed factor that the substitutions (chol_subst.cuh) load without a
// predicate, in plain C++ so that they can be walked on a CPU.
#pragma once

#ifdef __CUDACC__
#define SPGO_HD __host__ __device__ __forceinline__
#else
#define SPGO_HD inline
#endif

namespace spgo {

constexpr int kPanel = 16;  // block width of the factorisation and the substitutions

// offset of column c of the block at kb from the block's first column, same row (packed lower
// triangle, column-major: column j holds rows j..P-1)
SPGO_HD int subst_col(int P, int kb, int c) { return c * (P - kb) - c * (c + 1) / 2; }

// The forward sweep walks kPanel columns whatever the block's width.  Past the last column of a
// narrow block it stays on that column: going on would turn back in front of the block (P = 6:
// element -30 of the factor).
SPGO_HD int subst_fwd_first(int P, int kb, int c0) {
  const int last = P - kb - 1;
  return subst_col(P, kb, c0 < last ? c0 : last);
}
SPGO_HD int subst_fwd_step(int P, int kb, int c) {  // from column c to the next
  const int d = P - kb - 1 - c;
  return d > 0 ? d : 0;
}

}  // namespace spgo
