"""The work that users have the library do, as cases that can be timed and compared.

listed() names twelve of them, draw() gives more of the same ranges, prepare() makes what a program has
in hand before the call, run() is one pass through the public entry points, work() says what that pass
cannot do without, and exact() gives the same outputs from FP64 direct sums in plain torch.

Accelerations, steps and gradients come back whole, in the FP64 arrays that the entry points fill.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from gravitas_gb300 import abi, ics
from gravitas_gb300.sim import DirectSolver, Params, Simulation, Solver, State

STATE9 = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")
PAIRS_MAX = 1.6e11  # pairs that exact() may sum


def listed() -> list[dict]:
    return [
        # a preview scene of a thousand stars at the reference solver's defaults: launches and copies are what counts
        dict(name="accel_1k", kind="accel", scene="plummer", n=1013, theta=0.0, leaf=24, eps=0.05, walk="mixed", mono=False),
        # the plain method's configuration: Plummer sphere of 16,384, leaf 8, global steps on the resident state
        dict(name="plummer_16k", kind="resident", scene="plummer", n=16384, theta=0.5, leaf=8, eps=0.01, dt=1e-3, steps=10, walk="mixed"),
        # the evolve driver's inner loop at its defaults: 60,000 bodies, one step per call on the caller's arrays
        dict(name="evolve_60k", kind="host", scene="plummer", n=60000, theta=0.5, leaf=24, eps=0.01, dt=1e-3, steps=1, walk="mixed"),
        # the galaxy configuration: 131,072 bodies, block steps of 6 levels
        dict(name="galaxy_131k", kind="block", scene="galaxy", n=131072, theta=0.5, leaf=24, eps=0.02, dt=0.016, steps=1, levels=6, eta=0.025),
        # the headline: the merger of 1,048,576 bodies, resident, a few steps between two looks at the state
        dict(name="merger_1m", kind="resident", scene="merger", n=1048576, theta=0.5, leaf=24, eps=0.02, dt=1e-3, steps=4, walk="mixed"),
        # the batched configuration: 64 systems of 2,048 to 65,536 bodies in one forest, at the autotuner's choice
        dict(name="forest_64", kind="forest", nsys=64, nmin=2048, nmax=65536, layout=1, theta=0.7, leaf=32, eps=0.02, dt=1e-3, steps=2),
        # a scene with black holes, as the reference's own scenes have them: the hole-aware step of a 20,000-star disk
        dict(name="holes_20k", kind="host", scene="disk", n=20000, theta=0.5, leaf=24, eps=0.06, dt=4e-3, steps=1, walk="mixed"),
        # parity runs: the FP64 walk, bit for bit the reference's
        dict(name="fp64_16k", kind="resident", scene="plummer", n=16384, theta=0.5, leaf=8, eps=0.01, dt=1e-3, steps=2, walk="fp64"),
        # the differentiable configuration's gradient, a few of its steps, with the direct sum and with the tree
        dict(name="adjoint_32k", kind="adjoint", n=32768, eps=0.01, dt=1e-3, steps=8, every=4, tree=False, theta=0.5, leaf=16),
        dict(name="adjoint_tree_32k", kind="adjoint", n=32768, eps=0.01, dt=1e-3, steps=8, every=4, tree=True, theta=0.5, leaf=16),
        # the inspector's energy and momenta, exact up to 30,000 bodies
        dict(name="energy_30k", kind="energy", scene="disk", n=29998, theta=0.5, leaf=24, eps=0.06),
        # the force-error check of a run: FP64 direct sums at 4,096 of its bodies
        dict(name="direct_4096", kind="direct", scene="galaxy", n=131072, targets=4096, eps=0.02),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    """One more case of the same kinds, its sizes spread over their whole ranges."""
    kind = rng.choice(("accel", "accel", "resident", "resident", "host", "host", "block", "forest", "adjoint", "energy", "direct"))
    c = dict(kind=kind, theta=rng.choice((0.5, 0.6, 0.7, 0.9)), leaf=rng.choice((8, 16, 24, 32)), eps=rng.choice((0.01, 0.02, 0.05)))
    if kind == "accel":
        walk = rng.choice(("mixed", "mixed", "mixed", "plain"))
        c |= dict(scene=rng.choice(("plummer", "disk", "galaxy")), n=_log(rng, 500, 600_000), walk=walk, mono=walk == "mixed" and rng.random() < 0.2)
    elif kind == "resident":
        walk = rng.choice(("mixed", "mixed", "mixed", "fp64"))
        n = _log(rng, 1000, 1_000_000 if walk == "mixed" else 30_000)
        c |= dict(scene=rng.choice(("plummer", "galaxy")), n=n, dt=1e-3, steps=10 if n < 50_000 and walk == "mixed" else 2, walk=walk)
    elif kind == "host":
        scene = rng.choice(("plummer", "galaxy", "disk", "disk"))
        c |= dict(scene=scene, n=_log(rng, 1000, 250_000 if scene != "disk" else 60_000), dt=rng.choice((1e-3, 2e-3)), steps=1, walk="mixed")
        if scene == "disk":
            c |= dict(eps=0.06, dt=rng.choice((2e-3, 4e-3)))
    elif kind == "block":
        c |= dict(scene=rng.choice(("plummer", "galaxy")), n=_log(rng, 4000, 200_000), eps=0.02, dt=0.016, steps=1, levels=rng.choice((4, 5, 6)), eta=0.025)
    elif kind == "forest":
        nmax = _log(rng, 1000, 40_000)
        c |= dict(nsys=rng.choice((8, 33, 64)), nmin=max(50, nmax // 32), nmax=nmax, layout=rng.randrange(1 << 20), dt=1e-3, steps=2)
    elif kind == "adjoint":
        c |= dict(n=_log(rng, 1000, 32_768), eps=0.01, dt=1e-3, steps=8, every=rng.choice((3, 4, 8)), tree=rng.random() < 0.5)
    elif kind == "energy":
        scene = rng.choice(("plummer", "disk"))
        c |= dict(scene=scene, n=_log(rng, 2000, 300_000 if scene == "plummer" else 29_998), eps=0.06 if scene == "disk" else c["eps"])
    else:
        c |= dict(scene=rng.choice(("plummer", "galaxy")), n=_log(rng, 10_000, 131_072), targets=_log(rng, 256, 4096))
        del c["theta"], c["leaf"]
    return c


# ---- what a program has in hand


def _scene(case: dict, seed: int) -> dict:
    n = case["n"]
    if case["scene"] == "plummer":
        return ics.plummer(n, seed=seed)
    if case["scene"] == "galaxy":
        return ics.galaxy(n, seed=seed)
    if case["scene"] == "merger":
        return ics.merger(n, seed=seed)
    return ics.test_disk(n, seed=seed)  # n stars and two holes


def _forest_sizes(case: dict) -> list[int]:
    rng = random.Random(case["layout"])
    return [_log(rng, case["nmin"], case["nmax"]) for _ in range(case["nsys"])]


def _forest(case: dict, seed: int) -> tuple[dict, np.ndarray]:
    """Plummer spheres and disks of the layout's sizes, scale radii in [0.5, 2]."""
    rng = np.random.default_rng(seed)
    parts = []
    for q, n in enumerate(_forest_sizes(case)):
        a = rng.uniform(0.5, 2.0)
        if q % 2:
            s = ics.test_disk(n, seed=seed * 1000 + q, holes=False)
            for k in ("px", "py", "pz"):
                s[k] *= a
        else:
            s = ics.plummer(n, seed=seed * 1000 + q, a=a)
        parts.append(s)
    off = np.concatenate([[0], np.cumsum([len(p["px"]) for p in parts])]).astype(np.int64)
    return {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}, off


def prepare(case: dict, seed: int) -> dict:
    kind, P = case["kind"], abi.ptr
    ctx = abi.Context(0)
    st = dict(case=case, ctx=ctx)
    if kind in ("accel", "host", "direct"):  # the caller's own arrays
        st["state"] = State.from_dict(_scene(case, seed))
        par = Params(dt=case.get("dt", 0.0), softening=case["eps"])
        if kind == "direct":
            rng = np.random.default_rng(seed + 1)
            st |= dict(solver=DirectSolver(ctx), params=par, targets=np.sort(rng.choice(case["n"], case["targets"], replace=False)))
        else:
            sol = Solver(theta=case["theta"], leaf_size=case["leaf"], walk=case["walk"], monopole_only=case.get("mono", False), ctx=ctx)
            st |= dict(solver=sol, params=par, sim=Simulation(st["state"], sol, par))
        return st
    if kind == "adjoint":
        s, targets = ics.adjoint_problem(case["n"], seed=seed)
        x0, v0 = (np.stack([s[a + b] for b in "xyz"], 1) for a in "pv")
        return st | dict(x0=x0, v0=v0, mass=s["mass"], targets=targets)
    # resident states, with page-locked buffers for what comes back
    s, off = _forest(case, seed) if kind == "forest" else (_scene(case, seed), None)
    st["params"] = abi.make_params(case["theta"], case["eps"], case["leaf"], walk=case.get("walk", "mixed"))
    if off is None:
        ctx.call("gbh_state_upload", len(s["px"]), *[P(s[k]) for k in STATE9[:6]], None, None, None, P(s["mass"]), P(s["kind"]), P(s["alive"]))
    else:
        ctx.forest_upload(off, *[s[k] for k in STATE9[:6]], s["mass"], s["kind"], s["alive"])
    if kind != "energy":
        st["out"] = torch.empty((9, len(s["px"])), dtype=torch.float64, pin_memory=True)
    return st


# ---- one pass


def run(st: dict):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "accel":
        s = st["state"]
        st["solver"].accelerations(s, st["params"])
        return [s.acc_x, s.acc_y, s.acc_z]
    if kind == "host":
        s = st["state"]
        st["sim"].step(case["steps"])
        return [s.pos_x, s.pos_y, s.pos_z, s.vel_x, s.vel_y, s.vel_z, s.acc_x, s.acc_y, s.acc_z]
    if kind == "direct":
        return st["solver"].accelerations(st["state"], st["params"], st["targets"])
    if kind == "energy":
        d = ctx.diagnostics(st["params"])
        return {k: np.array(v) if isinstance(v, list) else v for k, v in d.items()}
    if kind == "adjoint":
        x, v = ctx.fwd_save(st["x0"], st["v0"], st["mass"], case["dt"], case["eps"], case["steps"], case["every"], abi.ADJ_FP32,
                            abi.ADJ_TREE if case["tree"] else abi.ADJ_DIRECT, case["theta"], case["leaf"])
        dx, dv, dm = ctx.bwd(2.0 * (x - st["targets"]) / len(x), None)
        return [x, v, dx, dv, dm]
    if kind == "block":
        ctx.step_block(st["params"], case["dt"], case["eta"], case["levels"], case["steps"])
    else:
        ctx.call("gbh_state_step", st["params"], case["dt"], case["steps"])
    ctx.call("gbh_state_download", *[abi.ptr(row.data_ptr()) for row in st["out"]])
    return st["out"]


# ---- what a pass cannot do without


def _tree_flops(n: float, theta: float) -> float:
    """Node and leaf-pair arithmetic of one force evaluation: 1.03e5 per star on the merger of a million at theta 0.5
    (its interactions as the reference's per-star walk counts them), scaled by log n and about 1 / theta^1.9 (its
    measured walk times at theta 0.3, 0.5 and 0.8), never more than the direct sum."""
    return n * min(1.03e5 * (math.log2(n) / 20) * (0.5 / theta) ** 1.9, 20.0 * n)


def work(case: dict) -> dict:
    kind = case["kind"]
    n = sum(_forest_sizes(case)) if kind == "forest" else case["n"]
    th, steps = case.get("theta") or 0.9, case.get("steps", 1)
    if kind == "accel":
        return dict(bytes=n * 56.0, flops=_tree_flops(n, th))
    if kind == "direct":
        return dict(bytes=n * 33.0 + case["targets"] * 32.0, flops=20.0 * n * case["targets"])
    if kind == "energy":
        return dict(bytes=n * 57.0, flops=20.0 * n * n / 2 if n <= 30_000 else 0.6 * _tree_flops(n, th))
    if kind == "adjoint":
        back = steps + 1
        if case["tree"]:
            f = _tree_flops(n, th)
            return dict(bytes=n * 8.0 * 19, flops=(steps + 1) * f + back * 2.5 * f)
        return dict(bytes=n * 8.0 * 19, flops=n * n * ((steps + 1) * 18.0 + back * 51.0))
    if kind == "forest":
        return dict(bytes=n * 152.0, flops=steps * sum(_tree_flops(k, th) for k in _forest_sizes(case)))
    share = 3.0 if kind == "block" else 1.0  # a block step walks each body about this many times
    return dict(bytes=n * 152.0, flops=steps * share * _tree_flops(n, th))


# ---- the same in FP64, from direct sums


def _t(a) -> torch.Tensor:
    return torch.as_tensor(np.asarray(a, np.float64), device="cuda")


def _forces(x, src, m, eps, at=None):
    """Softened direct sums at the bodies `at` (all) from the sources src with masses m; a body adds nothing to itself."""
    out = torch.empty((x.shape[0] if at is None else len(at), 3), dtype=torch.float64, device=x.device)
    step = max(1, int(4e7 // max(1, len(m))))
    for b in range(0, len(out), step):
        t = x[b:b + step] if at is None else x[at[b:b + step]]
        d = src[None] - t[:, None]
        w = m / ((d * d).sum(-1) + eps * eps) ** 1.5
        out[b:b + step] = (w[..., None] * d).sum(1)
    return out


def _kdk(x, v, m, eps, dt, steps):
    a = _forces(x, x, m, eps)
    for _ in range(steps):
        v = v + 0.5 * dt * a
        x = x + dt * v
        a = _forces(x, x, m, eps)
        v = v + 0.5 * dt * a
    return x, v, a


def _block(x, v, m, case):
    """Block steps: every body on the power-of-two fraction of dt that its acceleration asks for."""
    T, ticks = case["dt"], 1 << (case["levels"] - 1)
    a = _forces(x, x, m, case["eps"])

    def rung(a):
        want = case["eta"] * torch.sqrt(case["eps"] / a.norm(dim=1))
        return torch.ceil(torch.log2(T / want)).clamp(0, case["levels"] - 1).long()

    for _ in range(case["steps"]):
        r = rung(a)
        end, now = ticks >> r, 0
        v = v + (0.5 * T / (1 << r))[:, None] * a
        while now < ticks:
            t = int(end.min())
            x, now = x + (t - now) * T / ticks * v, t
            on = (end == t).nonzero()[:, 0]
            a[on] = _forces(x, x, m, case["eps"], on)
            v[on] += (0.5 * T / (1 << r[on]))[:, None] * a[on]
            if t < ticks:
                q = rung(a[on])
                for _ in range(case["levels"]):  # a step starts at a multiple of its own length
                    q = torch.where(t % (ticks >> q) != 0, q + 1, q)
                r[on], end[on] = q, t + (ticks >> q)
                v[on] += (0.5 * T / (1 << q))[:, None] * a[on]
            else:
                break
    return x, v, a


def _split(x, v, m, hole, eps, dt, steps):
    """The hole-aware step: stars near a hole, and the holes, in power-of-two substeps under the hole pairs."""
    h, e2 = hole.nonzero()[:, 0], eps * eps
    star = (~hole).nonzero()[:, 0]

    def pull(t, s):  # of the bodies s on the bodies t
        return _forces(x[t], x[s], m[s], eps) if len(t) and len(s) else torch.zeros((len(t), 3), dtype=torch.float64, device=x.device)

    def slow():
        a = torch.zeros_like(x)
        a[star] = _forces(x[star], x[star], m[star], eps)
        return a

    a = slow()
    for _ in range(steps):
        r2 = ((x[:, None] - x[h][None]) ** 2).sum(-1)
        re = torch.sqrt(r2 + e2)
        tau = torch.sqrt(re / (m[h] / re ** 3 * torch.sqrt(r2)))  # a body on the hole itself: infinite
        below = tau < 20 * dt
        near = below.any(1) & ~hole
        pair = [float(tau[h[i], j]) for i in range(len(h)) for j in range(i + 1, len(h))]
        least = min([float(tau[~hole].min())] + pair)
        least = least if least < 20 * dt else math.inf
        k = 1
        while math.isfinite(least) and k * least < 20 * dt and k < 256:
            k *= 2
        nr, far = near.nonzero()[:, 0], (~near & ~hole).nonzero()[:, 0]

        def outer():
            f = torch.zeros_like(x)
            f[far], f[h] = pull(far, h), pull(h, far)
            return f

        def fast():
            return pull(nr, h), pull(h, h) + pull(h, nr)

        v = v + 0.5 * dt * (a + outer())
        hs, (fn, fh) = dt / k, fast()
        for _ in range(k):
            v[nr] += 0.5 * hs * fn
            v[h] += 0.5 * hs * fh
            x[nr] += hs * v[nr]
            x[h] += hs * v[h]
            fn, fh = fast()
            v[nr] += 0.5 * hs * fn
            v[h] += 0.5 * hs * fh
        x[far] += dt * v[far]
        a = slow()
        v = v + 0.5 * dt * (a + outer())
    return x, v, a


def _adjoint(case, seed):
    """KDK steps of the softened direct sum and the transposed Jacobian of every kick."""
    s, targets = ics.adjoint_problem(case["n"], seed=seed)
    x, v = (torch.stack([_t(s[a + b]) for b in "xyz"], 1) for a in "pv")
    m, eps, dt = _t(s["mass"]), case["eps"], case["dt"]
    xs, a = [x], _forces(x, x, m, eps)
    for _ in range(case["steps"]):
        v = v + 0.5 * dt * a
        x = x + dt * v
        a = _forces(x, x, m, eps)
        v = v + 0.5 * dt * a
        xs.append(x)

    def vjp(x, w):  # J^T w and (da/dm)^T w
        gx, gm = torch.empty_like(x), torch.empty_like(m)
        step = max(1, int(2e7 // len(m)))
        for b in range(0, len(m), step):
            d = x[None] - x[b:b + step, None]
            s2 = (d * d).sum(-1) + eps * eps
            u = m[b:b + step, None, None] * w[None] - m[None, :, None] * w[b:b + step, None]
            du = (d * u).sum(-1)
            gx[b:b + step] = (u / s2[..., None] ** 1.5).sum(1) - 3 * (d * (du / s2 ** 2.5)[..., None]).sum(1)
            gm[b:b + step] = -((d * w[None]).sum(-1) / s2 ** 1.5).sum(1)
        return gx, gm

    lx, lv, lm = 2 * (x - _t(targets)) / len(m), torch.zeros_like(x), torch.zeros_like(m)
    for q in range(case["steps"], -1, -1):
        gx, gm = vjp(xs[q], lv) if q < case["steps"] else (torch.zeros_like(lx), torch.zeros_like(lm))
        c = dt if 0 < q < case["steps"] else 0.5 * dt
        lx, lm = lx + c * gx, lm + c * gm
        if q:
            lv = lv + dt * lx
    return [x, v, lx, lv, lm]


def _energy(s, eps):
    x, v = (torch.stack([_t(s[a + b]) for b in "xyz"], 1) for a in "pv")
    m = _t(s["mass"])
    u = 0.0
    step = max(1, int(4e7 // len(m)))
    for b in range(0, len(m), step):
        d = x[None] - x[b:b + step, None]
        w = m[b:b + step, None] * m[None] / torch.sqrt((d * d).sum(-1) + eps * eps)
        u -= float(w.sum()) / 2
    u += float((m * m).sum()) / eps / 2  # each body with itself
    ke = float((m * (v * v).sum(1)).sum()) / 2
    mass = float(m.sum())
    host = [q.cpu().numpy() for q in ((m[:, None] * v).sum(0), (m[:, None] * torch.linalg.cross(x, v)).sum(0), (m[:, None] * x).sum(0) / mass)]
    return dict(kinetic=ke, potential=u, total=ke + u, momentum=host[0], angular_momentum=host[1], center_of_mass=host[2], mass=mass, quality=None)


def _columns(*arrays):
    return [c.cpu().numpy() for a in arrays for c in a.T]


def exact(case: dict, seed: int):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "adjoint":
        return None if n * n * 6.0 * case["steps"] > PAIRS_MAX else [q.cpu().numpy() for q in _adjoint(case, seed)]
    if kind == "forest":
        if sum(k * k for k in _forest_sizes(case)) * (case["steps"] + 1.0) > PAIRS_MAX:
            return None
        s, off = _forest(case, seed)
    else:
        pairs = float(n) * case["targets"] if kind == "direct" else float(n) * n * {"accel": 1, "energy": 1, "block": 5 * case.get("steps", 1)}.get(kind, case.get("steps", 1) + 1)
        if pairs > PAIRS_MAX:
            return None
        s, off = _scene(case, seed), None
    if kind == "energy":
        return _energy(s, case["eps"])
    x, v = (torch.stack([_t(s[a + b]) for b in "xyz"], 1) for a in "pv")
    m, hole = _t(s["mass"]), torch.as_tensor(s["kind"] == abi.BLACK_HOLE, device="cuda")
    if kind == "direct":
        at = np.sort(np.random.default_rng(seed + 1).choice(n, case["targets"], replace=False))
        return _forces(x, x, m, case["eps"], torch.as_tensor(at, device="cuda")).cpu().numpy()
    if kind == "accel":
        a, star = torch.zeros_like(x), (~hole).nonzero()[:, 0]
        a[star] = _forces(x[star], x[star], m[star], case["eps"])
        return _columns(a)
    if kind == "forest":
        got = [_kdk(x[a:b], v[a:b], m[a:b], case["eps"], case["dt"], case["steps"]) for a, b in zip(off[:-1], off[1:])]
        out = [torch.cat(q) for q in zip(*got)]
    elif kind == "block":
        out = _block(x, v, m, case)
    elif bool(hole.any()):
        out = _split(x, v, m, hole, case["eps"], case["dt"], case["steps"])
    else:
        out = _kdk(x, v, m, case["eps"], case["dt"], case["steps"])
    return _columns(*out) if kind == "host" else np.stack(_columns(*out))
