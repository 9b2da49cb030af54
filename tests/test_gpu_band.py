"""The banded factorisation of wide reduced systems (mixed path): windows of D poses give a
band of 6 D - 1, eliminated from both ends in 16-wide blocks.  Bands of one block to the 17 it
takes and one wider (the multi-CTA path), seven of the eight residues P mod 16, systems barely
wider than the band (``test_gpu_band_edges.py``: the eighth, the smallest system and both sides
of the route's line).  The refined mixed step must match the
FP64 path's step from the same state.  Tolerance: the mixed step's stated accuracy, 1e-5 of
the step (its refinement's floor is the FP32 rounding of the Jacobian, 1e-7 to 2e-6)."""
import numpy as np
import pytest

import spgo_gb300.scenes as scenes
from spgo_gb300.solver import BatchSolver

pytestmark = pytest.mark.gpu


def corridor(seed, n_poses, window):
    """Frames 0.1 m apart looking sideways, so that a landmark is in view for about 100 of
    them; the covisibility window sets the band."""
    rng = np.random.Generator(np.random.PCG64(seed))
    W = np.tile(np.eye(4), (n_poses + 1, 1, 1))
    W[:, 0, 3] = 0.1 * np.arange(n_poses + 1)
    n = 40 * n_poses
    pts = np.stack([rng.uniform(-1.0, 0.1 * n_poses + 1.0, 2 * n), rng.uniform(-1.5, 1.5, 2 * n),
                    rng.uniform(4.0, 8.0, 2 * n)], 1)
    cand = np.broadcast_to(np.arange(n_poses + 1), (2 * n, n_poses + 1)).copy()
    return scenes.round_pixels_f32(scenes._build(rng, W, pts, cand, n, window=window))


def step(p, precision, **params):
    bs = BatchSolver([p], precision=precision)
    bs.set_params(loss="l2", max_iters=1, tol=0.0, use_graph=0, **params)
    p0, a0 = bs.poses.clone(), bs.alpha.clone()
    bs.reset()
    bs.iterate(1)
    st = bs.status()[0]
    d = (bs.poses - p0).cpu().numpy(), (bs.alpha - a0).cpu().numpy()
    bs.close()
    return d, st


@pytest.mark.parametrize("n_poses,window", [(52, 2), (54, 6), (55, 10), (61, 16), (62, 20), (63, 24), (67, 32), (54, 44),
                                            (57, 44), (80, 44), (96, 60)])
def test_banded_step_matches_fp64(built_lib, cuda_device, n_poses, window):
    p = corridor(900 + n_poses, n_poses, window)
    # near the optimum of the scene's truth, so that the step is well conditioned
    p.poses, p.alpha = p.gt_poses.copy(), p.gt_alpha.copy()
    (dp, da), st = step(p, "mixed")
    (rp, ra), rt = step(p, "fp64")
    assert st["accepted"] == rt["accepted"] == 1 and st["factor_failures"] == 0 and st["wait_timeouts"] == 0
    assert np.abs(dp - rp).max() < 1e-5 * np.abs(rp).max()
    assert np.abs(da - ra).max() < 1e-5 * np.abs(ra).max()
