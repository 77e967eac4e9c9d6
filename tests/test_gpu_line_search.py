"""The line search's energy changes against the oracle's on both sides of its change of kernel (37,888 nodes: four
threads a node up to there, one past it), at a lattice of a few nodes and with a last warp that is partly empty.

Tolerance: the changes are sums of FP32 terms of one node each (about 40 operations, 1e-5 of the terms' own size
at worst) that partly cancel: at every step length 1e-5 of the sum of its own terms' sizes, and that sum to 1e-5 of
itself (it decides whether a step is taken, and is formed by the same threads).
"""
import numpy as np
import pytest

import btd_b200 as btd
from helpers import MG
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny", [(5, 5), (33, 7), (256, 148), (199, 191)])
def test_energy_changes_match_the_oracle(nx, ny):
    sc = btd.configs.hanging_patch((nx, ny), 0.3 / 63 * (nx - 1), seed=3, jitter=2e-5)
    x0 = sc.position.reshape(-1, 3).astype(np.float32).astype(np.float64)
    cpu = Oracle(sc, h=1 / 60, newton_iterations=2, pcg_iterations=2, **MG)
    gpu = btd.GpuSolver(sc, btd.configs.solver_params(1 / 60, 4, 1e-6))
    cpu.set_state(x0)
    gpu.set_state(x0)
    cpu.predict()
    gpu.encode_predict()
    d = 2e-4 * np.random.default_rng(nx).standard_normal((sc.N, 3)).astype(np.float32).astype(np.float64)
    d[sc.pinned != 0] = 0.0
    gpu.write_vector("delta", d)
    e, m = gpu.encode_line_search()
    want, size = cpu.energy_change(d)
    assert (np.abs(e - want) < 1e-5 * size).all(), (e - want) / size
    assert (np.abs(m - size) < 1e-5 * size).all(), (m - size) / size
