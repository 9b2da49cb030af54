"""The Jacobian pass builds every record from the per-observation sums H = sum w^2 u u^T and
h = sum w^2 u r.  Checked where that can go wrong: a landmark next to a camera's image plane
(rows of 1e9 to 1e12 along one direction, whose cross products have to cancel), and CTAs of
every shape (observations split over one, three or eight warps), both precisions."""
import numpy as np
import pytest

import spgo_gb300.scenes as scenes
from spgo_gb300.solver import BatchSolver
from oracle import solver as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", [82, 90, 250])
def test_graded_rows_keep_the_reduced_system_consistent(built_lib, cuda_device, index):
    """A, B and C must come from one Jacobian: however it is rounded, S = A - B D^-1 B^T of the
    exported blocks is positive semidefinite up to the FP32 rounding of A, B and C themselves
    (2^-24 an entry; A once, B twice and C once, in the scaling of diag A: 4 P 2^-24)."""
    s, n, l = scenes.config3_specs(3)[index]
    p = scenes.round_pixels_f32(scenes.circle_scene(s, n, l))
    bs = BatchSolver([p], precision="mixed")
    bs.set_params(loss="l2")
    e = bs.export_system(0)
    bs.close()
    sc = 1.0 / np.sqrt(np.diag(e["A"]))
    Sm = (e["A"] - (e["B"] / (e["C"] * (1.0 + 1e-6) + 1e-4)) @ e["B"].T) * np.outer(sc, sc)
    assert np.linalg.eigvalsh((Sm + Sm.T) / 2)[0] > -4.0 * 6 * n * 2.0 ** -24


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("mixed", 2e-6)])
@pytest.mark.parametrize("block", [32, 96, 256])
def test_every_cta_shape_builds_the_same_system(built_lib, cuda_device, prec, tol, block):
    # windows on both sides of the host, one landmark seen by its host alone
    p = scenes.round_pixels_f32(scenes.circle_scene(77, 13, 210))
    o = np.arange(p.obs_ptr[4], p.obs_ptr[5])
    drop = o[p.obs_frame[o] != p.host[4]]
    p.obs_frame, p.obs_uv = np.delete(p.obs_frame, drop), np.delete(p.obs_uv, drop, 0)
    p.obs_ptr = np.concatenate([p.obs_ptr[:5], p.obs_ptr[5:] - len(drop)])
    bs = BatchSolver([p], precision=prec)
    bs.set_params(loss="huber", loss_scale=2.0, lin_block=block)
    e = bs.export_system(0)
    bs.close()
    lin = S.linearize(p, S.Loss(S.LOSS_HUBER, 2.0))
    for key, ref in (("A", lin.A), ("g", lin.g_T), ("B", lin.B), ("C", lin.C), ("g_a", lin.g_a)):
        assert np.abs(e[key] - ref).max() < tol * np.abs(ref).max(), key
