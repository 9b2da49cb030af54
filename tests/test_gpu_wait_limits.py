"""Every bounded wait of the wide systems' solves runs out by itself: with a limit of one
microsecond the cluster waits of the banded path and the flag waits of the multi-CTA
substitutions (mixed bands too wide for it, and FP64) give up, the kernels carry on and return,
the step is rejected and counted as a timeout.  The SIMT Schur complement is used, which has no
wait of its own.  With the default limit the same solver then takes the step."""
import numpy as np
import pytest

from spgo_gb300.solver import BatchSolver
from test_gpu_band import corridor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n_poses,window,banded", [("mixed", 60, 20, True), ("mixed", 60, 46, False),
                                                             ("fp64", 60, 20, False)])
def test_wait_runs_out_and_recovers(built_lib, cuda_device, precision, n_poses, window, banded):
    p = corridor(900 + n_poses, n_poses, window)
    bs = BatchSolver([p], precision=precision)
    assert banded == (precision == "mixed" and bs.sizes.pair_records // n_poses <= 45)  # (windows of 45 poses)
    p0, a0 = bs.poses.clone(), bs.alpha.clone()
    bs.set_params(loss="l2", max_iters=1, tol=0.0, use_tc=0, wait_us=1)
    st = bs.solve()[0]
    assert st["wait_timeouts"] == 1 and st["factor_failures"] == 0 and st["accepted"] == 0, st
    assert st["cost"] == st["cost0"] and np.isfinite(st["cost"])
    assert bool((bs.poses == p0).all()) and bool((bs.alpha == a0).all())
    bs.set_params(wait_us=0)
    st = bs.solve()[0]
    assert st["wait_timeouts"] == 0 and st["factor_failures"] == 0 and st["accepted"] == 1, st
    bs.close()
