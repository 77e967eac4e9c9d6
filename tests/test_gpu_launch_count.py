"""The kernels that run against what btd_launch_count and the stages promise, counted by the profiler's trace of the
launches (names of this library's kernels only; a stage or an eager substep, so that every launch is a plain one).
"""
import numpy as np
import pytest
import torch

import btd_b200 as btd

pytestmark = pytest.mark.gpu


def kernels(run, synchronize):
    """Names of the library's kernels that `run` launches."""
    synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        synchronize()
    return [e.name for e in prof.events() if "btd::" in e.name]


def solver(shape, **kw):
    sc = btd.configs.hanging_patch(shape, 0.3 / 63 * (shape[0] - 1), seed=1)
    return btd.GpuSolver(sc, btd.configs.solver_params(1 / 60, 2, 1e-6, **kw))


@pytest.mark.parametrize("shape, launches", [((64, 48), 1), ((160, 150), 1), ((160, 48), 2)])
def test_a_level_is_factored_in_one_launch_unless_its_families_take_different_kernels(shape, launches):
    g = solver(shape)
    g.encode_predict()
    g.encode_assemble(False)
    names = kernels(lambda: g.encode_assemble(False), g.synchronize)
    assert sum("k_assemble" in n for n in names) == 1  # the trace sees the library
    assert sum("k_line_" in n for n in names) == launches, names
    g.close()
