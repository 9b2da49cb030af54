"""Both sides of the banded factorisation's route (bands of up to 17 16-wide blocks: windows of
45 poses) and its smallest system: 50 poses with windows of 44 (h = 17 of 19 block rows, one of
them at the second end; P mod 16 = 12), 45 poses (the widest band it takes), 46 (the multi-CTA
path)."""
import numpy as np
import pytest

from oracle import lie
from spgo_gb300.solver import BatchSolver
from test_gpu_band import corridor, step

pytestmark = pytest.mark.gpu


def scene(n_poses, span):
    """A corridor near the optimum whose widest landmark spans exactly `span` poses."""
    p = corridor(900 + n_poses, n_poses, span + span % 2)
    lo = p.span()[0]
    lm = np.repeat(np.arange(p.n_landmarks), np.diff(p.obs_ptr))
    keep = p.obs_frame - lo[lm] <= span
    p.obs_frame, p.obs_uv = p.obs_frame[keep], p.obs_uv[keep]
    p.obs_ptr = np.concatenate([[0], np.cumsum(np.bincount(lm[keep], minlength=p.n_landmarks))]).astype(np.int64)
    lo, hi = p.span()
    assert (hi - lo).max() == span
    p.poses, p.alpha = p.gt_poses.copy(), p.gt_alpha.copy()
    return p


# tolerance: as test_gpu_band.py, the refined mixed step's stated accuracy, 1e-5 of the step
@pytest.mark.parametrize("n_poses,span", [(50, 44), (60, 45), (60, 46)])
def test_refined_step_at_the_route_s_edges(built_lib, cuda_device, n_poses, span):
    p = scene(n_poses, span)
    (dp, da), st = step(p, "mixed")
    (rp, ra), rt = step(p, "fp64")
    assert st["accepted"] == rt["accepted"] == 1 and st["factor_failures"] == 0 and st["wait_timeouts"] == 0
    assert np.abs(dp - rp).max() < 1e-5 * np.abs(rp).max()
    assert np.abs(da - ra).max() < 1e-5 * np.abs(ra).max()


@pytest.mark.parametrize("n_poses,span", [(50, 44), (52, 8), (60, 46)])
def test_reduced_solve_s_own_refinement(built_lib, cuda_device, n_poses, span):
    """Without the refinement of the whole step (outer_steps 0) the reduced solve is refined
    against the exact S of the assembly.  What is left is the rounding of A and S_L to FP32
    (2^-24 each, and of their sums: 8 in all), seen through the scaled system's inverse:
    a bound on the step's error in the norm of diag(S)."""
    p, lam = scene(n_poses, span), 1e-4
    bs = BatchSolver([p.copy()], precision="fp64")
    bs.set_params(loss="l2")
    S = bs.export_reduced(0, lam)["S"]
    A = bs.export_system(0)["A"]
    A = A + lam * np.diag(np.diag(A))
    bs.close()
    d = 1.0 / np.sqrt(np.diag(S))
    scaled = lambda M: M * d[:, None] * d
    tol = 8.0 * 2.0 ** -24 * np.linalg.norm(scaled(np.abs(A) + np.abs(A - S)), 2) / np.linalg.eigvalsh(scaled(S))[0]

    def delta(precision, **params):
        s = BatchSolver([p.copy()], precision=precision)
        s.set_params(loss="l2", max_iters=1, tol=0.0, lambda0=lam, use_graph=0, **params)
        s.reset()
        s.iterate(1)
        st, poses = s.status()[0], s.get_poses(0)
        s.close()
        assert st["accepted"] == 1 and st["factor_failures"] == 0 and st["wait_timeouts"] == 0
        return np.concatenate([lie.log_se3(lie.inv_se3(a) @ b) for a, b in zip(p.poses, poses)]) / d

    ref, got = delta("fp64"), delta("mixed", outer_steps=0, refine_steps=2)
    assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref), (np.linalg.norm(got - ref) / np.linalg.norm(ref), tol)
