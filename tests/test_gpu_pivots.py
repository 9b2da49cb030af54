"""The FP64 pivots' reciprocal and inverse root (chol_subst.cuh) against 60-digit arithmetic, over
the range of their Newton step, at its two ends and beyond them (the library's functions).
Bound: the step's own remainder is below 2^-60 (a third-order step from an estimate of 2^-20 or
better), so the roundings are what is left: one of 2^-53 in the reciprocal's last FMA; in the
root the error of d y^2 (2^-53, halved) and the last FMA.  Both stay below 2^-52."""
import ctypes as C
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest
import torch

from spgo_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "chol_subst.cuh"
__global__ void pivots(const double *d, double *r, double *s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = spgo::rcp_pivot(d[i]), s[i] = spgo::rsqrt_pivot(d[i]);
}
extern "C" int run(const double *d, double *r, double *s, int n) {
  pivots<<<(n + 255) / 256, 256>>>(d, r, s, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_pivot_reciprocal_and_root(built_lib, cuda_device, tmp_path):
    src, lib = tmp_path / "pivots.cu", tmp_path / "pivots.so"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, *build.FLAGS, "-shared", str(src), "-o", str(lib)], check=True)
    rng = np.random.Generator(np.random.PCG64(31))
    edge = [2.0 ** e * m for e in (-100, 0, 1, 99, 100, -101, 101) for m in (1.0, 1.0 + 2.0 ** -52, 1.5, 2.0 - 2.0 ** -52)]
    d = np.concatenate([edge, [np.nextafter(2.0 ** -100, 0.0), np.nextafter(2.0 ** 100, 0.0), 1e-300, 1e300],
                        np.ldexp(rng.uniform(1.0, 2.0, 8000), rng.integers(-105, 105, 8000))])
    x = torch.from_numpy(d).to(cuda_device)
    r, s = torch.zeros_like(x), torch.zeros_like(x)
    rc = C.CDLL(str(lib)).run(C.c_void_p(x.data_ptr()), C.c_void_p(r.data_ptr()), C.c_void_p(s.data_ptr()), len(d))
    assert rc == 0
    getcontext().prec = 60
    one, bound = Decimal(1), Decimal(2) ** -52
    for v, a, b in zip(d.tolist(), r.cpu().tolist(), s.cpu().tolist()):
        assert abs(Decimal(a) * Decimal(v) - one) <= bound, (v, a)
        assert abs(Decimal(b) * Decimal(v).sqrt() - one) <= bound, (v, b)
