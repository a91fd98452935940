"""Tree adjoint against automatic differentiation, in 64 bits, of the force of the same interaction lists:
accepted nodes (centre of mass, mass, quadrupole), leaf pairs, the moments' own dependence on the stars.
Node lists of one entry, of odd and of even counts. A group's list follows from the oracle's tree: a node is
accepted if it passes the opening test of all 32 stars; states are chosen with no test near its line.

Tolerance: a term's some 30 roundings are 2e-6 of it, FP32 sums of up to 56 of them and FP32 moments
another 4e-6, so 1e-5 of the terms; the gradients' sums lose at most a factor of 10 to cancellation."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS, DT, GROUP = 0.05, 0.1, 32


def lists(x, m, theta, leaf):
    """Per group: its bodies, the bodies of each accepted node, those of each opened leaf; the nearest test."""
    t = O.Tree(*(np.ascontiguousarray(x[:, k]) for k in range(3)), m, theta=theta, leaf=leaf).export()
    order, nodes = t["order"].astype(int), t["nodes"]
    com = np.stack([nodes["x"], nodes["y"], nodes["z"]], 1)
    out, margin = [], np.inf
    for g in range(0, len(order), GROUP):
        stars = order[g:g + GROUP]
        acc, near, i = [], [], 0
        while i >= 0:
            nd = nodes[i]
            d2 = ((x[stars] - com[i]) ** 2).sum(1).min()
            margin = min(margin, abs(np.sqrt(d2 / nd["crit2"]) - 1))
            if d2 >= nd["crit2"] or nd["first"] < 0:
                (acc if d2 >= nd["crit2"] else near).append(order[nd["lo"]:nd["hi"]])
                i = nd["next"]
            else:
                i = nd["first"]
        out.append((stars, acc, near))
    return out, margin


def force(torch, x, m, groups):
    rows = [None] * len(m)
    for stars, acc, near in groups:
        xt, a = x[stars], 0.0
        for j in acc:
            M = m[j].sum()
            c = (m[j, None] * x[j]).sum(0) / M
            e = x[j] - c
            Q = 3 * (m[j, None, None] * e[:, :, None] * e[:, None, :]).sum(0) - (m[j] * (e * e).sum(1)).sum() * torch.eye(3, dtype=x.dtype)
            d = c - xt
            inv = 1 / ((d * d).sum(1) + EPS * EPS)
            q = d @ Q
            f = M * inv ** 1.5 + 2.5 * (d * q).sum(1) * inv ** 3.5
            a = a + f[:, None] * d - q * (inv ** 2.5)[:, None]
        for j in near:
            d = x[j][None] - xt[:, None]
            a = a + ((m[j] * ((d * d).sum(2) + EPS * EPS) ** -1.5)[:, :, None] * d).sum(1)
        for k, s in enumerate(stars):
            rows[s] = a[k]
    return torch.stack(rows)


def clusters(k):
    """k clusters of 32 stars in different octants, each accepted by all others at theta 1."""
    rng = np.random.default_rng(k)
    at = np.array([[i >> 2 & 1, i >> 1 & 1, i & 1] for i in range(8)])[[0, 7, 3, 5, 6, 1, 2, 4][:k]] * 2.0 - 1.0
    x = np.repeat(at, 32, 0) + rng.uniform(-0.02, 0.02, (32 * k, 3))
    p = rng.permutation(len(x))
    return x[p], rng.normal(size=x.shape), rng.uniform(0.5, 1.5, len(x)) / len(x)


def plummer(n):
    s, _ = ics.adjoint_problem(n, seed=n)
    return (*(np.stack([s[a + b] for b in "xyz"], 1) for a in "pv"), s["mass"])


CASES = [("clusters", 2, 1.0, 32), ("clusters", 4, 1.0, 32), ("clusters", 7, 1.0, 32), ("clusters", 8, 1.0, 32),
         ("plummer", 33, 0.9, 4), ("plummer", 70, 0.9, 2), ("plummer", 150, 0.7, 8), ("plummer", 401, 0.9, 4),
         ("plummer", 700, 0.5, 3)]


def problem(kind, n, theta, leaf):
    x0, v0, m = clusters(n) if kind == "clusters" else plummer(n)
    groups0, margin0 = lists(x0, m, theta, leaf)
    return x0, v0, m, groups0, margin0


@pytest.mark.parametrize("kind,n,theta,leaf", CASES)
def test_gradient_of_the_same_lists(kind, n, theta, leaf):
    torch = pytest.importorskip("torch")
    x0, v0, m, groups0, margin0 = problem(kind, n, theta, leaf)
    rng = np.random.default_rng(3)
    gx, gv = rng.normal(size=x0.shape), rng.normal(size=x0.shape)
    tx, tv, tm = (torch.tensor(a, requires_grad=True) for a in (x0, v0, m))
    half = tv + 0.5 * DT * force(torch, tx, tm, groups0)
    x1 = tx + DT * half
    groups1, margin1 = lists(x1.detach().numpy(), m, theta, leaf)
    assert min(margin0, margin1) > 1e-5 and any(acc for _, acc, _ in groups0)
    v1 = half + 0.5 * DT * force(torch, x1, tm, groups1)
    ((torch.tensor(gx) * x1).sum() + (torch.tensor(gv) * v1).sum()).backward()
    with abi.Context(0) as ctx:
        ctx.fwd_save(x0, v0, m, DT, EPS, 1, 1, abi.ADJ_FP32, abi.ADJ_TREE, theta, leaf)
        dx, dv, dm = ctx.bwd(gx, gv)
    for got, want in ((dx - gx, tx.grad.numpy() - gx), (dv - gv - DT * gx, tv.grad.numpy() - gv - DT * gx),
                      (dm, tm.grad.numpy())):
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
