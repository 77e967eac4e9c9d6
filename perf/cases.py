"""The solve's performance cases: substeps of the scenes that the framework is used for, through GpuSolver.

Every pass replays one substep of a scene from its start - reset_state, then the substep - and hands out
the positions and velocities where a renderer would read them, in the solver's own device buffers (the
`host` cases move the state in from and out to host arrays instead, as a program does that owns the
state). The scenes start as cloth is found in a session, under tension and moving gently; flat and slack
starts are a corner where any implicit step is far from converged. The kinds of scene:

  patch  a sheet hanging from its pinned top row, solved to a relative residual of 1e-6 (the plain
         configuration); `slit` cuts it along a line, as cloth is in a session that has begun to tear;
  panel  the shipped denim panel in its frame at the shipped settings: 2 Newton x 2 PCG iterations,
         self-contact on;
  tear   the yarn lattice that two edge grips pull apart, self-contact on, with or without the learned
         coarse correction;
  batch  many small hanging patches, each with a grip, stepped as one graph;
  train  Adam on the learned correction's network over whitened operators.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The framework's package (its folder's name is no Python identifier)."""
    if "btd_b200" in sys.modules:
        return sys.modules["btd_b200"]
    pkg = os.path.join(os.getcwd(), "break-that-denim_b200")
    if not os.path.isdir(pkg):
        pkg = os.path.join(ROOT, "break-that-denim_b200")
    spec = importlib.util.spec_from_file_location("btd_b200", os.path.join(pkg, "__init__.py"), submodule_search_locations=[pkg])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["btd_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ------------------------------------------------------------------------------------------- cases


def _patch(name, nx, ny, slit=False, host=False):
    return dict(name=name, kind="patch", nx=nx, ny=ny, slit=slit, host=host)


def listed():
    return [
        # the smallest patch of the batched configuration, alone: launches and latency
        _patch("patch-16", 16, 16),
        # the plain configuration
        _patch("patch-64", 64, 64),
        # a ragged strip, its sides no power of two: a ribbon or a sleeve's cut
        _patch("patch-151x83", 151, 83),
        # the state owned by the host program, in and out every substep
        _patch("patch-96-host", 96, 96, host=True),
        # torn cloth: a slit across most of the sheet
        _patch("patch-128-slit", 128, 128, slit=True),
        # the large hanging sheet, five levels
        _patch("patch-256", 256, 256),
        # the product: the shipped panel at the shipped settings
        dict(name="panel-182x115", kind="panel", nx=182, ny=115),
        # the tearing patch at its full size, as the benchmark's learned arm runs it, and scaled down, plain
        dict(name="tear-256-learned", kind="tear", n=256, learned=True),
        dict(name="tear-128-plain", kind="tear", n=128, learned=False),
        # many independent patches of mixed sizes in one graph: throughput
        dict(name="batch-24", kind="batch", count=24, lo=16, hi=128),
        # training the learned correction's network
        dict(name="train-6x200", kind="train", ops=6, nodes=200, calls=64, steps=20),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["patch", "patch", "patch", "panel", "tear", "batch", "train"])
    if kind == "patch":
        return dict(kind="patch", nx=side(16, 256), ny=side(16, 256), slit=rng.random() < 0.25, host=rng.random() < 0.25)
    if kind == "panel":
        return dict(kind="panel", nx=side(96, 182), ny=side(72, 182))
    if kind == "tear":
        return dict(kind="tear", n=side(48, 256), learned=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(4, 24), lo=16, hi=side(24, 128))
    return dict(kind="train", ops=rng.randint(3, 6), nodes=rng.randint(60, 200), calls=rng.randint(16, 64), steps=rng.randint(8, 20))


# ------------------------------------------------------------------------------------------ scenes


def _phases(seed, n):
    return 2 * np.pi * _package().configs.splitmix64(seed, n).astype(np.float64) / 2.0 ** 64


def _relief(sc, seed, sigma):
    """Normal jitter of the free nodes, as the configurations have it."""
    free = sc.pinned == 0
    p = sc.position.reshape(-1, 3)
    p[free] += sigma * _package().configs.normal(seed, 3 * int(free.sum())).reshape(-1, 3)


def _hang(sc, seed):
    """The sheet hanging from its top row along -y, its columns stretched by the weight below them and
    swaying out of the plane by up to a few tenths of a radian."""
    nx, ny = sc.nx, sc.ny
    p = sc.position.reshape(ny, nx, 3)
    below = 9.81 * np.cumsum(sc.mass.reshape(ny, nx), 0)[:-1]
    length = sc.rest_length.reshape(ny, nx, 2)[:-1, :, 1] * (1 + below / sc.layers[0].material.yarns[1].ea_low)
    ph = _phases(seed, 2)
    s = (np.arange(ny - 1)[:, None] + 0.5) / (ny - 1)
    sway = 0.2 * (0.6 + 0.2 * np.sin(ph[0]) + 0.2 * np.sin(2 * np.pi * s + ph[1]))
    p[:-1, :, 0] = p[-1:, :, 0]
    p[:-1, :, 1] = p[-1:, :, 1] - np.cumsum((length * np.cos(sway))[::-1], 0)[::-1]
    p[:-1, :, 2] = p[-1:, :, 2] - np.cumsum((length * np.sin(sway))[::-1], 0)[::-1]
    _relief(sc, seed, 4e-6)


def _ripple(sc, seed, height):
    """A sheet held at its edges, out of its plane by `height` and less."""
    nx, ny = sc.nx, sc.ny
    ph = _phases(seed, 2)
    u, v = np.arange(nx)[None, :] / (nx - 1), np.arange(ny)[:, None] / (ny - 1)
    z = height * np.sin(np.pi * u) * np.sin(np.pi * v) * (0.7 + 0.15 * np.sin(ph[0]) + 0.15 * np.sin(3 * np.pi * u + ph[1]))
    sc.position.reshape(ny, nx, 3)[..., 2] += z * (sc.pinned.reshape(ny, nx) == 0)
    _relief(sc, seed, 4e-6)


def _scene(case, seed):
    """(scene, solver settings, grips) of a case with one sheet; a grip is a dict of attach_patch's
    arguments with the velocity of its handle."""
    btd = _package()
    cf = btd.configs
    if case["kind"] == "patch":
        c = cf.CONFIG0
        nx, ny = case["nx"], case["ny"]
        sc = cf.hanging_patch((nx, ny), size=c["size"] / (c["n"] - 1) * (nx - 1), seed=seed, jitter=0.0)
        _hang(sc, seed)
        if case["slit"]:  # the u spans between two columns are cut over half the height
            i, j0 = nx // 3 + seed % max(1, nx // 3), ny // 8 + seed % max(1, ny // 4)
            cut = 2 * (np.arange(j0, j0 + ny // 2) * nx + i)
            sc.seg_flags[cut] |= btd.SEG_BROKEN
            sc.intact[cut] = 0.0
        return sc, cf.solver_params(c["h"], c["newton_iterations"], c["pcg_rel_tol"], gravity=(0, -9.81, 0)), []
    if case["kind"] == "panel":
        spec = btd.default_spec()
        spec.seed = seed % (1 << 30)
        spec.size_u *= case["nx"] / 182
        spec.size_v *= case["ny"] / 115
        # mounted taut: the shipped mounting is slack along u and wrinkles over hundreds of substeps
        spec.compress_u = spec.compress_v = -0.005
        spec.shear = spec.perturbation = 0.0
        sc = btd.compile_scene(spec)
        _ripple(sc, seed, 4e-3)
        return sc, btd.default_params(), []
    c = cf.CONFIG4
    n = case["n"]
    sc, left, right = cf.config4(seed, n=n, region=max(4, n // 4))
    sc.position.reshape(-1, 3)[:, 0] *= 1.005  # the grips have pulled it taut
    _ripple(sc, seed, 1e-3)
    grips = []
    for nodes, sign in ((left, -1.0), (right, 1.0)):
        grips.append(dict(picked=int(nodes[len(nodes) // 2]), nodes=nodes, weights=np.ones(len(nodes)), stiffness=c["grip_stiffness"],
                          max_lead=1.0, velocity=np.array([0.5 * sign * c["grip_speed"], 0.0, 0.0])))
    return sc, cf.solver_params(c["h"], c["newton_iterations"], c["pcg_rel_tol"], self_contact=1), grips


def _batch_scenes(case, seed):
    """The batch's patches as (scene, settings, grips)."""
    cf = _package().configs
    c = cf.CONFIG3
    prm = cf.solver_params(c["h"], c["newton_iterations"], c["pcg_rel_tol"], gravity=(0, -9.81, 0))
    out = []
    for b, (sc, g) in enumerate(cf.config3(count=case["count"], sides=(case["lo"], case["hi"]))):
        _hang(sc, seed + b)
        out.append((sc, prm, [dict(g, velocity=0.03 * g["velocity"])]))  # the pull begins: its handle starts slowly
    return out


class _View:
    """A solver's device buffer as a CUDA array; it keeps the solver, whose memory it is."""

    def __init__(self, solver, which):
        self.solver = solver
        ptr, size = solver.device_buffer(which)
        self.__cuda_array_interface__ = {"shape": (size // 16, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


class _Sheet:
    """A solver with its grips and the views of its state."""

    def __init__(self, sc, prm, grips):
        btd = _package()
        self.g = btd.GpuSolver(sc, prm)
        self.h = prm.h
        self.pos = sc.position.reshape(-1, 3)
        self.x, self.v = (torch.as_tensor(_View(self.g, w), device="cuda")[:, :3] for w in ("x", "v"))
        self.grips = []
        for slot, q in enumerate(grips):
            a = self.pos[q["picked"]].astype(np.float32)
            self.g.attach_patch(slot, q["picked"], q["nodes"], q["weights"], a, q["stiffness"], max_lead=q["max_lead"])
            self.grips.append((a.astype(np.float64), q["velocity"]))

    def aim(self):
        """The grips' handles at the end of the substep."""
        for slot, (a, vel) in enumerate(self.grips):
            self.g.set_target(a + vel * self.h, slot=slot)


def prepare(case, seed):
    btd = _package()
    if case["kind"] == "train":
        rng = np.random.default_rng(seed)
        tr = btd.learned.Trainer()
        for _ in range(case["ops"]):
            n3 = 3 * case["nodes"]
            # a whitened coarse operator: unit diagonal blocks, a smooth near-null space
            B = rng.standard_normal((n3, 24)) / math.sqrt(24)
            At = np.eye(n3) + 0.5 * (B @ B.T - np.diag((B * B).sum(1)))
            At += max(0.0, 0.02 - np.linalg.eigvalsh(At)[0]) * np.eye(n3)
            R = rng.standard_normal((case["calls"], n3))
            tr.add_op(At, rng.uniform(-1, 1, (case["nodes"], btd.learned.IN)), R, np.linalg.solve(At, R.T).T)
        return dict(kind="train", trainer=tr, weights=btd.learned.init_weights(seed), steps=case["steps"], seed=seed)
    if case["kind"] == "batch":
        sheets = [_Sheet(*s) for s in _batch_scenes(case, seed)]
        return dict(kind="batch", sheets=sheets, batch=btd.Batch([s.g for s in sheets]))
    sheet = _Sheet(*_scene(case, seed))
    if case.get("learned"):
        sheet.g.set_learned(btd.learned.load(), guard=btd.configs.CONFIG4["guard"])
    pos = sheet.pos.astype(np.float32)
    return dict(kind="host" if case.get("host") else "sheet", sheet=sheet, pos=pos, vel=np.zeros_like(pos))


def run(state):
    kind = state["kind"]
    if kind == "train":
        w, loss = state["trainer"].train(state["weights"], steps=state["steps"], seed=state["seed"])
        return dict(weights=w, loss=loss)
    if kind == "batch":
        for s in state["sheets"]:
            s.g.reset_state()
            s.aim()
        state["batch"].run(1)
        for s in state["sheets"]:
            s.g.synchronize()
        return [dict(x=s.x, v=s.v) for s in state["sheets"]]
    s = state["sheet"]
    if kind == "host":
        s.g.set_state(state["pos"], state["vel"])
        s.g.substep()
        x, v = s.g.state()
        return dict(x=x[:, :3], v=v[:, :3])
    s.g.reset_state()
    s.aim()
    s.g.substep()
    s.g.synchronize()  # the solver has a stream of its own: its reader waits for it
    return dict(x=s.x, v=s.v)


def work(case):
    """A substep reads and writes each node's state (x, v: 32 B each way), its two spans (32 B) and its
    static data (16 B) once; each Newton iteration forms one row a node (about 1,500 operations) and
    each PCG iteration applies a V-cycle and the operator (about 2,500). PCG to 1e-6 takes 8 or more
    iterations a Newton step."""
    if case["kind"] == "train":
        n, m = case["ops"] * case["nodes"], case["ops"] * case["calls"] * 3 * case["nodes"]
        return {"bytes": 4.0 * (m * 2 + n * 20 + case["ops"] * (3 * case["nodes"]) ** 2),
                "flops": case["steps"] * (6.0 * n * 7064 + 2.0 * case["ops"] * (3 * case["nodes"]) ** 2 * 8 + 4.0 * m * 8)}
    if case["kind"] == "batch":
        nodes = case["count"] * ((case["lo"] + case["hi"]) / 2) ** 2
    else:
        nodes = case["n"] ** 2 if case["kind"] == "tear" else case["nx"] * case["ny"]
    newton, pcg = (2, 2) if case["kind"] == "panel" else (4, 8)
    return {"bytes": 112.0 * nodes, "flops": nodes * newton * (1500.0 + 2500.0 * pcg)}


# ------------------------------------------------------------------------- the same in 64 bits
#
# A substep is the implicit Euler step: the displacement d at which the gradient of the incremental
# potential (inertia, air drag, grip springs, yarn tension with its viscosity, fold-stiffening bending,
# shear diagonals) vanishes. Newton's method finds it in 64 bits, each system solved directly as a
# block-tridiagonal one of pairs of lattice rows.


def exact(case, seed):
    if case["kind"] == "train":
        return None  # BF16 weights by definition: no 64-bit value
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        return [_Exact(sc, prm, grips, dev).substep() for sc, prm, grips in _batch_scenes(case, seed)]
    return _Exact(*_scene(case, seed), dev).substep()


def _popcount(m):
    return sum((m >> k) & 1 for k in range(32))


class _Exact:
    def __init__(self, sc, prm, grips, dev):
        L = sc.layers[0]
        self.nx, self.ny, self.h, self.dev = L.nx, L.ny, prm.h, dev
        nx, ny = L.nx, L.ny
        at = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device=dev)  # noqa: E731
        f32 = lambda a: at(np.asarray(a, np.float32).astype(np.float64))  # noqa: E731
        self.x = f32(sc.position).reshape(-1, 3)
        self.free = at(sc.pinned == 0, torch.bool)
        self.mass = f32(sc.mass)
        self.grav = at(np.array(list(prm.gravity)))
        m = L.material
        rest, intact = f32(sc.rest_length).reshape(-1, 2), f32(sc.intact).reshape(-1, 2)
        active = at((sc.seg_flags.reshape(-1, 2) & 3) == 1, torch.bool)
        mask = at(sc.cut_mask.reshape(-1, 2).astype(np.int64), torch.int64)
        idx = torch.arange(nx * ny, device=dev).reshape(ny, nx)
        # spans of each family (owner a, next b) and bending triples (a, b, c)
        self.spans, self.triples = [], []
        for f, (a, b) in enumerate(((idx[:, :-1], idx[:, 1:]), (idx[:-1], idx[1:]))):
            a, b = a.reshape(-1), b.reshape(-1)
            on = active[a, f]
            a, b = a[on], b[on]
            self.spans.append((m.yarns[f], a, b, rest[a, f], intact[a, f]))
            step = 1 if f == 0 else nx
            p, q, r = (idx[:, :-2], idx[:, 1:-1], idx[:, 2:]) if f == 0 else (idx[:-2], idx[1:-1], idx[2:])
            p, q, r = p.reshape(-1), q.reshape(-1), r.reshape(-1)
            on = active[p, f] & active[q, f]
            p, q, r = p[on], q[on], r[on]
            assert bool((q - p == step).all())
            La, Lc = rest[p, f], rest[q, f]
            s = La + Lc
            lh = 2 * La * Lc / s
            B = max(1, m.yarns[f].yarns_per_span)
            full = (1 << B) - 1
            cont = _popcount(~(mask[p, f] | mask[q, f]) & full).double()
            ua, uc = _popcount(~mask[p, f] & full).double(), _popcount(~mask[q, f] & full).double()
            ma = torch.where(ua > 0, intact[p, f] * B / ua.clamp(min=1), 0.0 * ua)
            mc = torch.where(uc > 0, intact[q, f] * B / uc.clamp(min=1), 0.0 * uc)
            kb = m.yarns[f].bend_rigidity * (cont / B * torch.minimum(ma, mc)) / (lh * lh * 0.5 * s)
            self.triples.append((p, q, r, 2 * Lc / s, 2 * La / s, 4 * lh * lh, kb, kb * m.yarns[f].bend_viscosity / self.h))
        # shear diagonals of every cell
        c, r, t, rt = (q.reshape(-1) for q in (idx[:-1, :-1], idx[:-1, 1:], idx[1:, :-1], idx[1:, 1:]))
        cu, cv, rv, tu = active[c, 0], active[c, 1], active[r, 1], active[t, 0]
        i_ = lambda on, n, f: torch.where(on, intact[n, f], 0.0 * intact[n, f])  # noqa: E731
        area = torch.maximum(0.5 * (i_(cu, c, 0) + i_(tu, t, 0)), 0.5 * (i_(cv, c, 1) + i_(rv, r, 1)))
        cos0 = math.sqrt(1 - (1 - (1 - 0.16) ** 2) ** 2)
        cc = cos0 * area.clamp(0.02, 1.0).sqrt()
        jam = 1 - (1 - (1 - cc * cc).sqrt()).sqrt()
        ks = m.shear_stiffness * f32(sc.crossing_normal0)[c] / m.crossing_normal0
        Ld = (rest[c, 0] ** 2 + rest[c, 1] ** 2).sqrt()
        self.shear = []
        for a, b, on in ((c, rt, (cu & rv) | (cv & tu)), (r, t, (cu & cv) | (rv & tu))):
            self.shear.append((a[on], b[on], ks[on], jam[on], Ld[on]))
        self.drag = m.air_drag * m.pitch_u * m.pitch_v / self.h
        self.active, self.idx = active, idx
        self.grips = [(at(q["nodes"], torch.int64), at(q["weights"]) * q["stiffness"], at(np.asarray(q["velocity"])), q["max_lead"],
                       int(q["picked"])) for q in grips]

    def substep(self):
        """One substep from rest."""
        d = self.step()
        return dict(x=self.x + d, v=d / self.h)

    def drag_blocks(self):
        """Air drag's 3 x 3 block of every node from the accepted positions: along the normal of the
        cross of the two span tangents."""
        x, act, idx, nx, ny = self.x, self.active, self.idx, self.nx, self.ny
        tan = []
        for f in range(2):
            prev, nxt = idx.clone(), idx.clone()
            p, q = (idx[:, :-1], idx[:, 1:]) if f == 0 else (idx[:-1], idx[1:])
            on = act[p, f]
            (prev[:, 1:] if f == 0 else prev[1:]).copy_(torch.where(on, p, q))
            (nxt[:, :-1] if f == 0 else nxt[:-1]).copy_(torch.where(on, q, p))
            tan.append(x[nxt.reshape(-1)] - x[prev.reshape(-1)])
        lu, lv = tan[0].norm(dim=1), tan[1].norm(dim=1)
        cr = torch.linalg.cross(tan[0], tan[1])
        lc = cr.norm(dim=1)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        e = cr / lc.clamp(min=1e-300)[:, None]
        D = e[:, :, None] * e[:, None, :]
        thin = ~((lu > 0) & (lv > 0) & (lc > 1e-3 * lu * lv))
        t = torch.where((lu >= lv)[:, None], tan[0], tan[1])
        tl = t.norm(dim=1)
        t = t / tl.clamp(min=1e-300)[:, None]
        line = torch.where((tl > 0)[:, None, None], eye - t[:, :, None] * t[:, None, :], eye.expand(len(t), 3, 3))
        return self.drag * torch.where(thin[:, None, None], line, D)

    def terms(self, d, hess):
        """The gradient at step d, and with `hess` the projected second derivatives as (a, b, block)."""
        y, eye = self.x + d, torch.eye(3, dtype=torch.float64, device=self.dev)
        w = self.mass / self.h ** 2
        g = w[:, None] * (d - self.pred) + torch.einsum("nij,nj->ni", self.D, d)
        H = []
        n = torch.arange(len(d), device=self.dev)
        if hess:
            H.append((n, n, w[:, None, None] * eye + self.D))
        for nodes, k, target in self.held:
            g.index_add_(0, nodes, k[:, None] * (y[nodes] - target))
            if hess:
                H.append((nodes, nodes, k[:, None, None] * eye))

        def pair(a, b, e, f, K, kp):
            g.index_add_(0, b, f[:, None] * e)
            g.index_add_(0, a, -f[:, None] * e)
            if hess:
                blk = (K - kp)[:, None, None] * e[:, :, None] * e[:, None, :] + kp[:, None, None] * eye
                H.extend(((a, a, blk), (b, b, blk), (a, b, -blk), (b, a, -blk)))

        for yarn, a, b, L, intact in self.spans:
            en, e = self.x[b] - self.x[a], y[b] - y[a]
            l, ln = e.norm(dim=1), en.norm(dim=1)
            eps, ec, dk = l / L - 1, yarn.crimp_strain, yarn.ea_high - yarn.ea_low
            T = torch.where(eps <= 0, yarn.ea_compress * eps,
                            torch.where(eps <= ec, yarn.ea_low * eps + dk * eps * eps / (2 * ec),
                                        yarn.ea_low * ec + 0.5 * dk * ec + yarn.ea_high * (eps - ec)))
            K = torch.where(eps <= 0, yarn.ea_compress + 0 * eps,
                            torch.where(eps <= ec, yarn.ea_low + dk * eps / ec, yarn.ea_high + 0 * eps))
            c = yarn.axial_viscosity / (L * self.h)
            f = intact * T + c * (l - ln)
            pair(a, b, e / l[:, None], f, intact * K / L + c, f.clamp(min=0) / l)
        for a, b, ks, jam, Ld in self.shear:
            e = y[b] - y[a]
            l = e.norm(dim=1)
            f, K = ks * (l - Ld), ks
            c, ex, ramp = (Ld - l) / Ld - jam, ks * 39.0, 0.08
            f = f - torch.where(c > 0, torch.where(c < ramp, ex * Ld * c * c / (2 * ramp), ex * Ld * (c - 0.5 * ramp)), 0 * c)
            K = K + torch.where(c > 0, torch.where(c < ramp, ex * c / ramp, ex), 0 * c)
            pair(a, b, e / l[:, None], f, K, f.clamp(min=0) / l)
        for a, b, c, wa, wc, fold, kb, kd in self.triples:
            def second(z):
                return wa[:, None] * (z[a] - z[b]) + wc[:, None] * (z[c] - z[b]) + (wa + wc - 2)[:, None] * z[b]

            r, rn = second(y), second(self.x)
            q = (r * r).sum(1)
            lr, lrn = q.sqrt(), rn.norm(dim=1)
            d0, s = 1 - 0.85, q / fold
            inner = s < 0.85
            u = torch.where(inner, 1 - s, d0 + 0 * s)
            p1 = torch.where(inner, 1 / (u * u), 1 / d0 ** 2 + 2 / (fold * d0 ** 3) * (q - 0.85 * fold))
            p2 = 2 / (fold * u ** 3)
            k1 = kb * p1 + kd * (lr - lrn) / lr.clamp(min=1e-12)
            gr = k1[:, None] * r
            for nodes, wgt in ((a, wa), (b, -2 + 0 * wa), (c, wc)):
                g.index_add_(0, nodes, wgt[:, None] * gr)
            if hess:
                k2 = 2 * kb * p2 + kd * lrn / lr.clamp(min=1e-12) ** 3
                blk = k1.clamp(min=0)[:, None, None] * eye + k2[:, None, None] * r[:, :, None] * r[:, None, :]
                ws = ((a, wa), (b, -2 + 0 * wa), (c, wc))
                H.extend((m1, m2, (w1 * w2)[:, None, None] * blk) for m1, w1 in ws for m2, w2 in ws)
        g[~self.free] = 0
        return g, H

    def step(self):
        h = self.h
        self.pred = (h * h * self.grav).expand_as(self.x)
        self.D = self.drag_blocks()
        self.held = []
        for nodes, kw, vel, lead, picked in self.grips:  # attached at the start, the handle moved since
            to = vel * h
            to = to * min(1.0, lead / max(float(to.norm()), 1e-300))
            self.held.append((nodes, kw, self.x[nodes] + to))
        d = torch.zeros_like(self.x)
        first = None
        for it in range(40):
            g, H = self.terms(d, True)
            if first is None:
                first = float(g.norm())
            if float(g.norm()) <= 1e-13 * first:
                break
            s = self.solve(H, -g)
            slope = float((g * s).sum())
            alpha, lo, hi = 1.0, 0.0, None
            for _ in range(6):  # the slope along the step: none above a tenth of its start
                now = float((self.terms(d + alpha * s, False)[0] * s).sum())
                if now > -0.1 * slope:
                    hi = alpha
                    alpha = 0.5 * (lo + hi)
                else:
                    break
            d = d + alpha * s
            if float(s.abs().max()) < 1e-12:
                break
        return d

    def solve(self, H, b):
        """The block-tridiagonal solve: rows along the longer side taken in pairs."""
        nx, ny = self.nx, self.ny
        flip = nx > ny
        long, short = (nx, ny) if flip else (ny, nx)
        pairs = (long + 1) // 2
        m = 6 * short
        dev = self.dev
        D = torch.zeros(pairs * m * m, dtype=torch.float64, device=dev)
        E = torch.zeros(max(1, pairs - 1) * m * m, dtype=torch.float64, device=dev)  # block (p + 1, p)
        q3 = torch.arange(3, device=dev)

        def place(n):
            i, j = n % nx, n // nx
            if flip:
                i, j = j, i
            return j // 2, ((j % 2) * short + i) * 3

        for a, c, blk in H:
            on = self.free[a] & self.free[c]
            a, c, blk = a[on], c[on], blk[on]
            (pa, ra), (pc, rc) = place(a), place(c)
            row = (ra[:, None, None] + q3[None, :, None]) * m + rc[:, None, None] + q3[None, None, :]
            same, low = pa == pc, pa == pc + 1
            D.index_add_(0, (pa[same, None, None] * m * m + row[same]).reshape(-1), blk[same].reshape(-1))
            E.index_add_(0, (pc[low, None, None] * m * m + row[low]).reshape(-1), blk[low].reshape(-1))
        D, E = D.view(pairs, m, m), E.view(-1, m, m)
        n = torch.arange(nx * ny, device=dev)
        p, r = place(n)
        at = (p[:, None] * m + r[:, None] + q3[None, :])
        rhs = torch.zeros(pairs * m, dtype=torch.float64, device=dev)
        rhs[at.reshape(-1)] = (b * self.free[:, None]).reshape(-1)
        rhs = rhs.view(pairs, m, 1)
        dia = torch.diagonal(D, dim1=1, dim2=2)
        dia += (dia == 0).double()  # pinned rows and the padding
        C, W, y = [], [], []
        for q in range(pairs):
            S, t = D[q], rhs[q]
            if q:
                S = S - W[-1].T @ W[-1]
                t = t - W[-1].T @ y[-1]
            C.append(torch.linalg.cholesky(S))
            y.append(torch.linalg.solve_triangular(C[-1], t, upper=False))
            if q + 1 < pairs:
                W.append(torch.linalg.solve_triangular(C[-1], E[q].T, upper=False))
        x = [None] * pairs
        for q in range(pairs - 1, -1, -1):
            t = y[q] if q + 1 == pairs else y[q] - W[q] @ x[q + 1]
            x[q] = torch.linalg.solve_triangular(C[q].T, t, upper=True)
        return torch.cat(x).reshape(-1)[at.reshape(-1)].view(-1, 3)
