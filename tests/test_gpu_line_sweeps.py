"""The yarn-line sweeps and the V-cycle against the oracle's on the GPU's own operator, at the lattice sizes
where the line kernels change over: lines that fill their last chunk or leave one node of it (a chunk and its
separator hold six nodes), a line without a separator, the longest line of the compact sweep (131 nodes) and the
first one past it, alone in its family (132, 256, 257), and levels with the most lines a colour that the clustered
coarse levels take (48 nodes a side) and with one line more.

Tolerances, from FP32 arithmetic on FP64-formed coefficients: a sweep's right-hand side sums about 50 products
and its solve three dots of up to 64, six colours in sequence, on line systems whose softest modes are 1e3 to 1e5
times softer than their spans - 1e-3 of the sweep's result in the 2-norm, the bound that the sweeps' parity
tests use; a V-cycle of up to five levels 5e-3, as theirs.
"""
import numpy as np
import pytest

import btd_b200 as btd
from helpers import MG
from oracle import Oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nx, ny", [(5, 5), (6, 11), (12, 17), (16, 16), (48, 31), (95, 94), (96, 97), (131, 24), (132, 13),
                                    (256, 9), (257, 133)])
def test_sweeps_and_vcycle_match_the_oracle(nx, ny):
    sc = btd.configs.hanging_patch((nx, ny), 0.3 / 63 * (nx - 1), seed=nx + ny, jitter=2e-5)
    x0 = sc.position.reshape(-1, 3).astype(np.float32).astype(np.float64)
    cpu = Oracle(sc, h=1 / 60, newton_iterations=2, pcg_iterations=2, **MG)
    gpu = btd.GpuSolver(sc, btd.configs.solver_params(1 / 60, 4, 1e-6))
    cpu.set_state(x0)
    gpu.set_state(x0)
    cpu.predict()
    gpu.encode_predict()
    gpu.encode_assemble(True)
    cpu.assemble()
    cpu.build_levels(gpu.read_operator(0)[0])
    assert gpu.level_count() == cpu.level_count()
    rng = np.random.default_rng(7)
    for level in range(gpu.level_count()):
        n = gpu.level_nodes(level)
        x = rng.standard_normal((n, 3)).astype(np.float32).astype(np.float64)
        b = rng.standard_normal((n, 3)).astype(np.float32).astype(np.float64)
        fixed = gpu.read_operator(level)[1] != 0
        x[fixed] = 0.0
        for reverse in (False, True):
            gpu.write_vector("X", x, level)
            gpu.write_vector("B", b, level)
            gpu.encode_smooth(level, reverse)
            assert rel(gpu.read_vector("X", level), cpu.smooth(level, x, b, reverse)) < 1e-3, (level, reverse)
    b = rng.standard_normal((sc.N, 3)).astype(np.float32).astype(np.float64)
    b[sc.pinned != 0] = 0.0
    gpu.write_vector("B", b)
    gpu.encode_vcycle()
    assert rel(gpu.read_vector("X"), cpu.vcycle(b)) < 5e-3
    assert gpu.counters()[20] == 0  # no bounded wait ran out
