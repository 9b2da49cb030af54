"""The FP64 factorisation and substitutions against the oracle's dense solve, at the edges of
their shapes: one CTA with the packed factor (16-wide blocks: one narrow block, an exact
multiple, every kind of remainder, the largest number of rows left), and 32-column panels
spread over CTAs (an exact multiple, narrow last panels, bands below one panel, below the
substitutions' 64-row blocks, and as wide as the matrix); the last three also at the edges of
the pose chain's passes of 128 frames.  One damped step near the optimum;
tolerance 1e-8 of the step, the one the FP64 GN steps are held to elsewhere."""
import numpy as np
import pytest

from oracle import solver as S
from spgo_gb300.solver import BatchSolver
from test_gpu_band import corridor, step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_poses,window", [(1, 2), (2, 2), (3, 3), (8, 4), (11, 6), (16, 8), (21, 9), (27, 27), (34, 12),
                                            (38, 2), (43, 4), (48, 6), (53, 11), (58, 16), (64, 44), (41, 41),
                                            (128, 3), (129, 5), (300, 2)])
def test_fp64_step_matches_dense_solve(built_lib, cuda_device, n_poses, window):
    p = corridor(700 + n_poses, n_poses, window)
    p.poses, p.alpha = p.gt_poses.copy(), p.gt_alpha.copy()
    bs = BatchSolver([p.copy()], precision="fp64")
    bs.set_params(loss="l2", max_iters=1, tol=0.0, lambda0=1e-4, eps=1e-4, use_graph=0)
    bs.reset()
    bs.iterate(1)
    st = bs.status()[0]
    poses, alpha = np.asarray(bs.get_poses(0)), np.asarray(bs.get_alpha(0))
    bs.close()
    ref = S.solve_damped(S.linearize(p, S.Loss()), 1e-4, 1e-4)
    ref_p, ref_a = S.apply_update(p.poses, p.alpha, ref.delta, ref.delta_a)
    assert st["accepted"] == 1 and st["factor_failures"] == 0 and st["wait_timeouts"] == 0
    assert np.abs(poses - ref_p).max() < 1e-8 * np.abs(ref_p - p.poses).max()
    assert np.abs(alpha - ref_a).max() < 1e-8 * np.abs(ref_a - p.alpha).max()


@pytest.mark.parametrize("n_poses", [11, 48])
def test_fp64_pivots_beyond_fp32_range(built_lib, cuda_device, n_poses):
    """Pixels and focal lengths times 2^54: pivots of 2^115 and more, beyond the range whose
    reciprocals start from an FP32 estimate.  Same step, same tolerance."""
    p = corridor(760 + n_poses, n_poses, 6)
    p.poses, p.alpha = p.gt_poses.copy(), p.gt_alpha.copy()
    s = 2.0 ** 54
    p.intrinsics, p.anchor_uv, p.obs_uv = p.intrinsics * s, p.anchor_uv * s, p.obs_uv * s
    bs = BatchSolver([p.copy()], precision="fp64")
    bs.set_params(loss="l2", max_iters=1, tol=0.0, lambda0=1e-4, eps=1e-4, use_graph=0)
    bs.reset()
    bs.iterate(1)
    st = bs.status()[0]
    poses = np.asarray(bs.get_poses(0))
    bs.close()
    ref = S.solve_damped(S.linearize(p, S.Loss()), 1e-4, 1e-4)
    ref_p, _ = S.apply_update(p.poses, p.alpha, ref.delta, ref.delta_a)
    assert st["accepted"] == 1 and st["factor_failures"] == 0
    assert np.abs(poses - ref_p).max() < 1e-8 * np.abs(ref_p - p.poses).max()


@pytest.mark.parametrize("n_poses,window", [(1, 2), (2, 2), (3, 3), (8, 4), (11, 6), (16, 8), (21, 9), (27, 27), (37, 12), (48, 20)])
def test_mixed_step_matches_fp64(built_lib, cuda_device, n_poses, window):
    """The FP32 factorisation of one CTA (inverted diagonal blocks) at the same edges: the refined
    mixed step within its stated accuracy, 1e-5 of the step, of the FP64 path's."""
    p = corridor(800 + n_poses, n_poses, window)
    p.poses, p.alpha = p.gt_poses.copy(), p.gt_alpha.copy()
    (dp, da), st = step(p, "mixed")
    (rp, ra), rt = step(p, "fp64")
    assert st["accepted"] == rt["accepted"] == 1 and st["factor_failures"] == 0
    assert np.abs(dp - rp).max() < 1e-5 * np.abs(rp).max()
    assert np.abs(da - ra).max() < 1e-5 * np.abs(ra).max()
