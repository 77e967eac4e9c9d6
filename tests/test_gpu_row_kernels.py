"""PCG's kernels on the fine rows at the size where their form changes (37,888 nodes: every load of a row in flight up
to there, a neighbour at a time past it), with the last block of a launch full and partly empty.

Tolerances. On the FP32 rows PCG's operator is the one read back, and its stop is decided on b - A x in FP64 from the
FP64 iterate that is read back: the residual formed here is the same number but for the order of the sums, 1e-6 and one
part in 1e6 of it. On the FP64 rows the operator is the oracle's but for the FP32 rounding of the laws' scalars, 2e-6 as
in the operator's own tests. A V-cycle sums about 50 FP32 products a node and colour on four levels, 5e-3 as the V-cycle's
parity tests.
"""
import numpy as np
import pytest

import btd_b200 as btd
from helpers import MG, operator_apply
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny", [(256, 148), (257, 148)])
def test_solves_on_both_sides_of_the_change_of_form(nx, ny):
    sc = btd.configs.hanging_patch((nx, ny), 0.3 / 63 * (nx - 1), seed=nx, jitter=2e-5)
    x0 = sc.position.reshape(-1, 3).astype(np.float32).astype(np.float64)
    cpu = Oracle(sc, h=1 / 60, newton_iterations=2, pcg_iterations=2, **MG)
    gpu = btd.GpuSolver(sc, btd.configs.solver_params(1 / 60, 4, 1e-6))
    cpu.set_state(x0)
    gpu.set_state(x0)
    cpu.predict()
    gpu.encode_predict()
    gpu.encode_assemble(True)
    A_cpu, _, _ = cpu.assemble()
    A_gpu, fixed = gpu.read_operator(0)
    b = gpu.read_vector("B")
    for fp64, A, bound in ((False, A_gpu, 1e-6 * (1 + 1e-6)), (True, A_cpu, 2e-6)):
        gpu.set_operator_precision(fp64)
        gpu.write_vector("B", b)
        gpu.encode_pcg()
        r = b - operator_apply(A, nx, ny, gpu.delta_f64(), fixed)
        assert gpu.counter_dict()["pcg_missed"] == 0
        assert np.linalg.norm(r) <= bound * np.linalg.norm(b), fp64
    cpu.build_levels(A_gpu)
    rhs = np.random.default_rng(nx).standard_normal((sc.N, 3)).astype(np.float32).astype(np.float64)
    rhs[sc.pinned != 0] = 0.0
    gpu.write_vector("B", rhs)
    gpu.encode_vcycle()
    want = cpu.vcycle(rhs)
    assert np.linalg.norm(gpu.read_vector("X") - want) < 5e-3 * np.linalg.norm(want)
