"""One pose or the depths written between two steps of the drop-in class with nothing read in
between: the rest of the state has to stay what the step left on the device.  The reference
object is read back and gets everything written.  Tolerance: float32 readback of FP64 sums whose
order varies, and the reference's restart from float32, 1e-6."""
import numpy as np
import pytest

import spgo_gb300.scenes as scenes
from test_gpu_dropin_state import make, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["pose", "depths", "both"])
def test_write_between_steps_without_a_read(built_lib, cuda_device, what):
    p = scenes.corridor_scene(78, 6, 90)
    N, L, M = 6, p.n_landmarks, 20
    alpha = np.full(N * M, 0.3, np.float32)
    alpha[:L] = p.alpha
    poses = p.poses.astype(np.float32)

    def started():
        cs = make(p, M, L)
        for k in range(N):
            cs.writeIncrementalPose(k, poses[k])
        cs.loadInverseDepths(alpha)
        cs.step(2)
        return cs

    new = poses[2].copy()
    new[:3, 3] += 0.03
    got, ref = started(), started()
    if what != "depths":
        got.writeIncrementalPose(2, new)
    if what != "pose":
        got.loadInverseDepths(alpha)
    got.step(2)
    rp, ra = state(ref, N)
    if what != "depths":
        rp[2] = new
    if what != "pose":
        ra = alpha
    for k in range(N):
        ref.writeIncrementalPose(k, rp[k])
    ref.loadInverseDepths(ra)
    ref.step(2)
    (gp, ga), (rp, ra) = state(got, N), state(ref, N)
    assert np.abs(gp - rp).max() < 1e-6 and np.abs(ga - ra).max() < 1e-6
