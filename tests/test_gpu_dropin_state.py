"""State of the drop-in class between steps: single poses and depths written after a step, reads
in between, more observations (which rebuild the solver).  A second object that gets every pose
and depth written before every step must arrive at the same state.  Tolerance: float32 readback
of FP64 sums whose order varies, 1e-6."""
import numpy as np
import pytest

import spgo_gb300.scenes as scenes
from spgo_gb300.solver import CudaSolver

pytestmark = pytest.mark.gpu


def make(p, M, last):
    cs = CudaSolver(p.n_poses, M, precision="fp64")
    cs.loadCalibration(p.intrinsics.reshape(4, 2), p.T_rl)
    cs.setStepSize(0.5)
    observe(cs, p, 0, last)
    return cs


def observe(cs, p, first, last):
    lm = np.repeat(np.arange(p.n_landmarks), np.diff(p.obs_ptr))
    for o in range(p.n_obs):
        if first <= lm[o] < last:
            z = p.obs_uv[o]
            cs.writeObservations(p.host[lm[o]], p.obs_frame[o], lm[o], [z[0], z[1], 1.0], [z[2], z[3], 1.0])


def state(cs, N):
    return np.stack([cs.getIncrementalPose(k) for k in range(N)]), cs.getInverseDepths()


def test_state_written_and_read_between_steps(built_lib, cuda_device):
    p = scenes.corridor_scene(77, 6, 90)
    N, L, M = 6, p.n_landmarks, 20
    alpha = np.full(N * M, 0.3, np.float32)
    alpha[:L] = p.alpha
    got = make(p, M, L - 10)
    ref = make(p, M, L - 10)
    model_p, model_a = state(got, N)

    def write(cs, poses, depths):
        for k in poses:
            cs.writeIncrementalPose(k, model_p[k])
        if depths:
            cs.loadInverseDepths(model_a)

    model_p, model_a = p.poses.astype(np.float32), alpha
    for poses, depths, observed in ((range(N), True, False), ((2,), False, False), ((), False, False), ((0, N - 1), True, False),
                                    ((), False, True), ((3,), False, False)):
        model_p = model_p.copy()
        for k in poses:  # the written poses differ from the state
            model_p[k, :3, 3] += 0.01 * (k + 1)
        if depths:
            model_a = (model_a * 1.02).astype(np.float32)
        if observed:
            observe(got, p, L - 10, L)
            observe(ref, p, L - 10, L)
        write(got, poses, depths)
        gp, ga = state(got, N)  # read back before the step
        assert np.array_equal(gp, model_p) and np.array_equal(ga, model_a)
        got.step(2)
        write(ref, range(N), True)
        ref.step(2)
        (gp, ga), (rp, ra) = state(got, N), state(ref, N)
        assert np.abs(gp - rp).max() < 1e-6 and np.abs(ga - ra).max() < 1e-6
        model_p, model_a = gp, ga
        # the reference object continues from what was read (float32), so does this one
        write(got, range(N), True)
