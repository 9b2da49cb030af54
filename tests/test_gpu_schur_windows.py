"""The FP64 Schur complement multiplies only the landmarks whose window of pose blocks
meets a warp's rows and columns, and splits short work lists over more CTAs: the reduced
system at the edges of its 8-block tiles and 2 x 4 block warps, with landmarks whose
window is empty (seen by their host alone) or one block wide, against the FP64 oracle.
Tolerance: the FP64 path's 1e-10 of max|A| (its other reduced-system test's bound)."""
import numpy as np
import pytest

import spgo_gb300.scenes as scenes
from spgo_gb300.solver import BatchSolver
from oracle import solver as S

pytestmark = pytest.mark.gpu


def narrowed(p, rng):
    """p with every third landmark reduced to its host's observation and every third to
    its host and one neighbour."""
    keep = np.ones(p.n_obs, bool)
    for l in range(p.n_landmarks):
        o = np.arange(p.obs_ptr[l], p.obs_ptr[l + 1])
        other = o[p.obs_frame[o] != p.host[l]]
        if l % 3 == 0:
            keep[other] = False
        elif l % 3 == 1 and len(other) > 1:
            keep[other] = False
            keep[rng.choice(other)] = True
    cnt = np.add.reduceat(keep.astype(np.int64), p.obs_ptr[:-1])
    q = p.copy()
    q.obs_ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    q.obs_frame, q.obs_uv = p.obs_frame[keep], p.obs_uv[keep]
    return q


@pytest.mark.parametrize("n_poses,n_landmarks", [(1, 33), (2, 40), (7, 150), (8, 160), (9, 200), (16, 330), (17, 350),
                                                 (36, 900)])
def test_fp64_reduced_system_at_tile_edges(built_lib, cuda_device, n_poses, n_landmarks):
    rng = np.random.default_rng(n_poses)
    p = narrowed(scenes.round_pixels_f32(scenes.corridor_scene(500 + n_poses, n_poses, n_landmarks)), rng)
    bs = BatchSolver([p], precision="fp64")
    bs.set_params(loss="l2")
    lin = S.linearize(p, S.Loss())
    for lam in (1e-4, 2.0):
        D = lin.C * (1.0 + lam) + float(np.float32(1e-4))
        BD = lin.B / D[None, :]
        Sm = lin.A + np.diag(lam * np.diag(lin.A)) - BD @ lin.B.T
        got = bs.export_reduced(0, lam)
        assert np.abs(got["S"] - Sm).max() < 1e-10 * np.abs(lin.A).max()
        assert np.abs(got["gS"] - (lin.g_T - BD @ lin.g_a)).max() < 1e-10 * np.abs(lin.g_T).max()
    bs.close()
