"""The batched configuration (configuration 3): independent hanging patches of seeded sizes,
stiffnesses, yarn regions and grips, run as one batch (btd_batch_substeps: every patch on its own
stream, queued round robin). The reference has no batch; parity is the plain path: each patch of
the batch ends bit for bit where it ends when run alone.
"""
import numpy as np
import pytest

import btd_b200 as btd

pytestmark = pytest.mark.gpu


def make(patch):
    sc, g = patch
    c = btd.configs.CONFIG3
    s = btd.GpuSolver(sc, btd.configs.solver_params(c["h"], c["newton_iterations"], c["pcg_rel_tol"]))
    x = s.x
    anchor = x[g["picked"]].astype(np.float32)
    s.attach_patch(0, g["picked"], g["nodes"], g["weights"], anchor, g["stiffness"], max_lead=g["max_lead"])
    return s, anchor


def test_batch_equals_each_patch_alone():
    c = btd.configs.CONFIG3
    patches = btd.configs.config3(count=12, sides=(16, 48))
    steps = 15
    batch = [make(p) for p in patches]
    for k in range(1, steps + 1):
        for (s, anchor), (_, g) in zip(batch, patches):
            s.set_target((anchor + k * c["h"] * g["velocity"]).astype(np.float32))
        btd.batch_substeps([s for s, _ in batch], 1)
    for s, _ in batch:
        s.synchronize()
    for (s, _), p in zip(batch, patches):
        alone, anchor = make(p)
        for k in range(1, steps + 1):
            alone.set_target((anchor + k * c["h"] * p[1]["velocity"]).astype(np.float32))
            alone.substep()
        assert np.array_equal(alone.x, s.x)
        assert np.array_equal(alone.field(), s.field())
        alone.close()
    for s, _ in batch:
        assert np.isfinite(s.x).all()
        s.close()


def test_batch_graph_equals_each_patch_alone():
    """The batch as one graph (btd_batch_create / btd_batch_run): every patch's substep a branch of a
    single graph launch, grip targets queued on each patch's stream before it; each patch ends bit for
    bit where it ends alone, also after the sweeps' launch shapes were autotuned."""
    c = btd.configs.CONFIG3
    patches = btd.configs.config3(count=12, sides=(16, 64))
    steps = 12
    batch = [make(p) for p in patches]
    s0, a0 = batch[0]
    s0.set_target((a0 + c["h"] * patches[0][1]["velocity"]).astype(np.float32))
    s0.substep()  # an assembled system to tune on (patch 0 is one substep ahead)
    batch[0][0].autotune(reps=3)
    first = batch[0][0].x.copy()
    graph = btd.Batch([s for s, _ in batch])
    for k in range(1, steps + 1):
        for i, ((s, anchor), (_, g)) in enumerate(zip(batch, patches)):
            kk = k + 1 if i == 0 else k
            s.set_target((anchor + kk * c["h"] * g["velocity"]).astype(np.float32))
        graph.run(1)
    for s, _ in batch:
        s.synchronize()
    for i, ((s, _), p) in enumerate(zip(batch, patches)):
        alone, anchor = make(p)
        total = steps + 1 if i == 0 else steps
        for k in range(1, total + 1):
            alone.set_target((anchor + k * c["h"] * p[1]["velocity"]).astype(np.float32))
            alone.substep()
            if i == 0 and k == 1:
                assert np.array_equal(alone.x, first)
        assert np.array_equal(alone.x, s.x), i
        alone.close()
    graph.close()
    for s, _ in batch:
        s.close()


@pytest.mark.parametrize("shapes, crowded", [([(128, 128), (96, 131), (73, 112), (131, 97)] + 3 * [(128, 128)], True),
                                             ([(128, 131), (73, 50)], False)])
def test_large_batches_equal_their_patches_alone(shapes, crowded):
    """Batches on both sides of 94,720 nodes side by side (at most eight patches: one a hardware queue), past which the
    kernels that leave one CTA an SM give way to others: the long compact sweeps and the row kernels, the same
    arithmetic bit for bit."""
    assert (sum(a * b for a, b in shapes) > 94720) == crowded
    scenes = [btd.configs.hanging_patch(s, 0.3 / 63 * (s[0] - 1), seed=k) for k, s in enumerate(shapes)]
    batch, alone = ([btd.GpuSolver(sc, btd.configs.solver_params(1 / 60, 4, 1e-6)) for sc in scenes] for _ in range(2))
    graph = btd.Batch(batch)
    graph.run(2)
    btd.batch_substeps(batch, 1)
    for s, a in zip(batch, alone):
        a.substeps(3)
        assert np.array_equal(s.x, a.x)
        assert s.counters()[17] == a.counters()[17]
    graph.close()
    for s in batch + alone:
        s.close()


@pytest.mark.parametrize("sweeps, coarsest", [(2, 400), (1, 400), (3, 30)])
def test_the_learned_correction_between_clustered_levels_equals_the_launches(sweeps, coarsest):
    """The cluster launch of the coarse levels is split around the learned correction, its vectors handed through
    memory; in a batch the levels take a launch a colour: the same bit for bit."""
    c = btd.configs.CONFIG4
    solvers = []
    for _ in range(2):
        sc, left, _ = btd.configs.config4(n=64, region=16)
        s = btd.GpuSolver(sc, btd.configs.solver_params(c["h"], 4, 1e-6, coarse_sweeps=sweeps, max_coarsest_nodes=coarsest))
        s.set_learned(btd.learned.load(), on=True, guard=0.9)
        picked = int(left[len(left) // 2])
        s.attach_patch(0, picked, left, np.ones(len(left)), s.x[picked], c["grip_stiffness"], max_lead=1.0)
        solvers.append(s)
    small = btd.GpuSolver(btd.configs.hanging_patch(16, 0.07, seed=1), btd.configs.solver_params(1 / 60, 2, 1e-6))
    graph = btd.Batch([solvers[0], small])
    graph.run(3)
    solvers[1].substeps(3)
    assert np.array_equal(solvers[0].x, solvers[1].x)
    assert solvers[0].counters()[17] == solvers[1].counters()[17]
    assert solvers[1].learned_stats()["applied"] > 0
    graph.close()
    for s in solvers + [small]:
        s.close()


def test_batch_patches_match_the_oracle():
    """Three patches of the batch (their seeded sizes, stiffness factors, yarn regions and grips), run
    in the batch graph on the GPU and one by one in the oracle from the same float32 state: after 8
    substeps every patch's positions agree to 1 % of its motion (a third of the reference's own bound
    for converged trajectories, correctness.ts:271; 0.16 % measured on the first patch). (The grips'
    lead limit, a GPU-side interaction bound that the reference's CPU grip does not have, is opened
    here.)"""
    from helpers import MG
    from oracle import Oracle

    c = btd.configs.CONFIG3
    patches = btd.configs.config3(count=3, sides=(24, 48))
    steps = 8
    batch = []
    for sc, g in patches:
        sv = btd.GpuSolver(sc, btd.configs.solver_params(c["h"], c["newton_iterations"], c["pcg_rel_tol"]))
        anchor = sv.x[g["picked"]].astype(np.float32)
        sv.attach_patch(0, g["picked"], g["nodes"], g["weights"], anchor, g["stiffness"], max_lead=1.0)
        batch.append((sv, anchor))
    graph = btd.Batch([s for s, _ in batch])
    try:
        for k in range(1, steps + 1):
            for (s, anchor), (_, g) in zip(batch, patches):
                s.set_target((anchor + k * c["h"] * g["velocity"]).astype(np.float32))
            graph.run(1)
        for s, _ in batch:
            s.synchronize()
    finally:
        graph.close()
    for (s, anchor), (sc, g) in zip(batch, patches):
        o = Oracle(sc, h=c["h"], newton_iterations=c["newton_iterations"], pcg_iterations=500, pcg_rel_tol=c["pcg_rel_tol"], **MG)
        x = sc.position.reshape(-1, 3).astype(np.float32).astype(np.float64)
        o.set_state(x)
        nodes = np.asarray(g["nodes"])
        a = anchor.astype(np.float64)
        o.add_grip(nodes, np.asarray(g["weights"], np.float64), (x[nodes] - x[g["picked"]]).reshape(-1), a, g["stiffness"])
        for k in range(1, steps + 1):
            o.set_grip_goal(0, (a + k * c["h"] * g["velocity"]).astype(np.float32).astype(np.float64))
            o.substep()
        moved = np.abs(o.x - x).max()
        err = np.abs(s.x.astype(np.float64) - o.x).max()
        assert moved > 0 and err < 1e-2 * moved, (sc.N, err, moved)
        s.close()
