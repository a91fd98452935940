"""Stars in the root cube's highest corner, whose keys are all ones or nearly so, in a sort tile that also
holds dead bodies and holes: lattices, coincident stars in the corner, stars within eight cells of it, a
diagonal pair. Keys, order and FP64 forces against the oracle, bit for bit."""
import ctypes

import numpy as np
import pytest

from gravitas_gb300 import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu
P = abi.ptr
EPS, THETA, LEAF = 0.02, 0.5, 8


def lattice(k):
    g = np.arange(float(k))
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)


def scene(name):
    """Positions, with the bodies that are no stars (the first of them before the corner's stars)."""
    cell = 7.0 / 2**21
    if name == "lattice":
        return np.concatenate([[[3.2, 3.1, 3.3]], lattice(8)]), [0]
    if name == "tiles":  # 5 tiles, the corner in the last
        return np.concatenate([lattice(16) * 0.5, [[1.0, 2.0, 3.0]] * 700, [[7.5, 7.5, 7.5]]]), [0, 4100, 4500]
    if name == "coincident":
        return np.concatenate([lattice(8), [[7.0, 7.0, 7.0]] * 40]), [3, 100, 520]
    if name == "near":  # every distance in cells from 0 to 12 on each axis
        d = np.random.default_rng(5).integers(0, 13, (300, 3)) * cell
        return np.concatenate([lattice(8), 7.0 - d]), [0, 5, 511, 600, 700]
    return np.array([[0.5, 0.4, 0.3], [0.0, 0.0, 0.0], [1.0, 1.0, 1.0]]), [0]  # a pair on a diagonal


SCENES = ("lattice", "tiles", "coincident", "near", "pair")


def state(name, how):
    p, off = scene(name)
    n = len(p)
    rng = np.random.default_rng(n)
    s = dict(px=p[:, 0].copy(), py=p[:, 1].copy(), pz=p[:, 2].copy(), mass=rng.uniform(0.5, 1.5, n) / n,
             kind=np.zeros(n, np.uint8), alive=np.ones(n, np.uint8))
    if how == "hole":
        s["kind"][off] = O.BLACK_HOLE
    else:
        s["alive"][off] = 0
    return s, [rng.normal(size=n) for _ in range(3)]


def tree(s):
    return O.Tree(s["px"], s["py"], s["pz"], s["mass"], s["kind"], s["alive"], theta=THETA, leaf=LEAF)


@pytest.mark.parametrize("how", ["hole", "dead"])
@pytest.mark.parametrize("name", SCENES)
def test_corner_stars(name, how):
    s, acc = state(name, how)
    n = len(s["px"])
    t = tree(s)
    want, e = t.accelerations(EPS, acc=[a.copy() for a in acc]), t.export()
    with abi.Context(0) as ctx:
        got = [a.copy() for a in acc]
        ctx.call("gbh_accelerations", abi.make_params(THETA, EPS, LEAF, walk="fp64"), n, P(s["px"]), P(s["py"]),
                 P(s["pz"]), P(s["mass"]), P(s["kind"]), P(s["alive"]), *[P(a) for a in got])
        g = ctx.tree_export()
    assert np.array_equal(g["keys"], e["keys"]) and np.array_equal(g["order"], e["order"])
    assert np.array_equal(g["nodes"], e["nodes"])
    assert np.array_equal(np.stack(got, 1), want)
    if how == "dead":  # a dead body keeps its entry
        off = s["alive"] == 0
        assert np.array_equal(np.stack(got, 1)[off], np.stack(acc, 1)[off])


@pytest.mark.parametrize("how", ["hole", "dead"])
def test_corner_stars_of_a_forest(how):
    parts = [state(name, how)[0] for name in SCENES]
    s = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    off = np.concatenate([[0], np.cumsum([len(p["px"]) for p in parts])]).astype(np.int64)
    zero, n = np.zeros(off[-1]), int(off[-1])
    with abi.Context(0) as ctx:
        ctx.forest_upload(off, s["px"], s["py"], s["pz"], zero, zero, zero, s["mass"], s["kind"], s["alive"])
        ctx.call("gbh_state_accelerations", abi.make_params(THETA, EPS, LEAF, walk="fp64"))
        got = [np.zeros(n) for _ in range(3)]
        ctx.call("gbh_state_download", *[None] * 6, *[P(a) for a in got])
        g = ctx.tree_export()
        stars, _ = ctx.forest_layout(len(parts))
    for q, p in enumerate(parts):
        t = tree(p)
        e, (lo, hi) = t.export(), stars[q]
        assert np.array_equal(g["keys"][lo:hi], e["keys"])
        assert np.array_equal(g["order"][lo:hi] - off[q], e["order"])
        assert np.array_equal(np.stack(got, 1)[off[q]:off[q + 1]], t.accelerations(EPS))


@pytest.mark.parametrize("how", ["hole", "dead"])
@pytest.mark.parametrize("name", SCENES)
def test_corner_stars_without_allocation(name, how):
    torch = pytest.importorskip("torch")
    s, _ = state(name, how)
    n, e = len(s["px"]), tree(s).export()
    d = {k: torch.from_numpy(s[k]).to("cuda:0") for k in ("px", "py", "pz", "kind", "alive")}
    keys = torch.full((n,), -1, dtype=torch.int64, device="cuda:0")
    order = torch.full((n,), -1, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    nstars, err = np.zeros(1, np.int64), ctypes.create_string_buffer(256)
    rc = abi.load().gbh_morton_order_noalloc(0, None, n, *[P(d[k].data_ptr()) for k in ("px", "py", "pz", "kind", "alive")],
                                             P(keys.data_ptr()), P(order.data_ptr()), P(nstars), err, 256)
    assert rc == abi.OK, err.value.decode()
    assert int(nstars[0]) == len(e["keys"])
    assert np.array_equal(keys.cpu().numpy()[:len(e["keys"])].view(np.uint64), e["keys"])
    assert np.array_equal(order.cpu().numpy()[:len(e["keys"])], e["order"])
