"""The sweep autotuner (btd_autotune): per multigrid level it times the yarn-line sweep's CTA sizes and
staging tiles on the current operator and keeps the fastest. The choice changes only the launch shape,
never the arithmetic, so a run tuned after its first substep ends bit for bit where an untuned run does. Levels whose
lines all take the compact sweep (64 x 64 nodes: every level) have one shape, four threads a node; 200 x 200 has
both kinds, 150 x 60 a level with one family of each.
"""
import numpy as np
import pytest

import btd_b200 as btd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 200, (150, 60)])
def test_autotuned_run_equals_the_untuned_one(n):
    nx, ny = n if isinstance(n, tuple) else (n, n)
    sc = btd.configs.hanging_patch(n, 0.3 * (nx - 1) / 63, seed=2)
    params = btd.configs.solver_params(1 / 60, 4, 1e-6)
    a = btd.GpuSolver(sc, params)
    a.substeps(3)
    a.synchronize()
    xa = a.x.copy()
    b = btd.GpuSolver(sc, params)
    b.substeps(1)
    choice = b.autotune(reps=5)
    assert len(choice) == b.level_count()
    for threads, tile, ms in choice:
        assert threads % 32 == 0 and 64 <= threads <= 256
        assert 0 < tile <= 256
        assert ms > 0
    if n == 200:
        assert any(t in (128, 200) for _, t, _ in choice)
    if nx <= 131:
        assert [t for t, _, _ in choice] == [min(256, (4 * k + 31) // 32 * 32) for k in (64, 33, 17)]
    b.substeps(2)
    b.synchronize()
    assert np.array_equal(b.x, xa)
