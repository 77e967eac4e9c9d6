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


def counted(g):
    c = g.counter_dict()
    return g.launch_count(1, c["newton"], c["pcg_total"])


@pytest.mark.parametrize("kind", ["plain", "mixed", "rebuilt", "learned", "layers"])
def test_launch_count_is_the_kernels_of_a_substep(kind):
    if kind == "learned":  # grips, self-contact and the learned correction
        sc, left, _ = btd.configs.config4(n=64, region=16)
        g = btd.GpuSolver(sc, btd.configs.solver_params(1 / 120, 2, 1e-6, self_contact=1))
        g.set_learned(btd.learned.load(), on=True, guard=0.9)
        g.attach_patch(0, int(left[0]), left, np.ones(len(left)), g.x[left[0]], 500.0, max_lead=1.0)
    elif kind == "layers":  # contact between layers
        m = btd.material_preset(0)
        sc = btd.compile_scene([btd.layer_spec(m, 0.01, 0.01, bundle=(1, 1), z=z, seed=3) for z in (0.0, 3e-4)])
        g = btd.GpuSolver(sc, btd.configs.solver_params(1 / 120, 2, 1e-6, pcg_cap=20, self_contact=1, cross_layer=1))
    else:
        g = solver((160, 48) if kind == "mixed" else (64, 64), lag_coarse=0 if kind == "rebuilt" else 1)
    g.set_graph_mode(False)
    g.substep()
    g.clear_counters()
    names = kernels(g.substep, g.synchronize)
    assert len(names) == counted(g)
    g.close()


def test_launch_count_of_a_batch():
    """In a batch the V-cycle's coarse levels take a launch a colour (six) in place of the one cluster launch: two
    sweeps of each, the coarsest included, and a residual, a restriction and a prolongation between two of them."""
    solvers = [solver((64, 64)), solver((36, 20))]
    assert [g.level_count() for g in solvers] == [3, 2]
    for g in solvers:
        g.substep()
    alone = [g.launch_count(1, 2, 20) for g in solvers]
    batch = btd.Batch(solvers)
    batch.run(1)
    for g in solvers:
        g.synchronize()
    # levels in the cluster launch: 33 x 33 and 17 x 17 nodes; 18 x 10 nodes
    for g, before, own in zip(solvers, alone, (12 + 3 + 12, 12)):
        assert g.launch_count(1, 2, 20) - before == 20 * (own - 1)
    for g in solvers:
        g.substep()
    assert [g.launch_count(1, 2, 20) for g in solvers] == alone
    batch.close()
    for g in solvers:
        g.close()
