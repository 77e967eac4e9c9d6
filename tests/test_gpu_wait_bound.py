"""The bounded waits (the kernels never hang on a wait): the cluster launch's for what its CTAs send one another
(32 x 32 nodes, their 16 x 16 coarse ones in the cluster; 16 x 12, the whole V-cycle) and the smoother's for the
staging copies of lines over 131 nodes (200 x 16, whose coarse levels are too long for the cluster). A test hook
sets the waits' first bound to zero tries, so their error flag is raised on every wait while the copies
still land under the second bound. btd_synchronize then reports BTD_E_TIMEOUT exactly once, the next
call returns 0, and the positions equal a run with the default bound bit for bit (the copies did land).
"""
import numpy as np
import pytest

import btd_b200 as btd
from btd_b200 import _abi

pytestmark = pytest.mark.gpu


def run(substeps, shape):
    sc = btd.configs.hanging_patch(shape, 0.15 / 31 * (shape[0] - 1), seed=4)
    g = btd.GpuSolver(sc, btd.configs.solver_params(1 / 60, 4, 1e-6))
    g.substeps(substeps)
    return g


@pytest.mark.parametrize("shape", [(32, 32), (16, 12), (200, 16)])
def test_first_bound_runs_out_and_is_reported_once(shape):
    ref = run(2, shape)
    ref.synchronize()
    x_ref = ref.x.copy()
    ref.close()
    _abi.check("btd_set_wait_bound", 0)
    try:
        g = run(2, shape)
        with pytest.raises(_abi.BtdError) as e:
            g.synchronize()
        assert e.value.rc == -5, e.value
        assert "bounded device-side wait" in str(e.value)
        g.synchronize()  # reported once: the flag was cleared
        assert np.array_equal(g.x, x_ref)
        g.close()
    finally:
        _abi.check("btd_set_wait_bound", -1)
    g = run(1, shape)
    g.synchronize()  # the default bound again: nothing to report
    g.close()
