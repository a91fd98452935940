"""The tile sort and its merges against the oracle's keys and order, at the edges of tiles, runs and
merge levels: coincident stars, dead bodies and holes inside the tiles, whole tiles without a star."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu
P = abi.ptr
TILE = 1024


@pytest.fixture(scope="module")
def ctx():
    c = abi.Context(0)
    yield c
    c.close()


def state(n, seed, gaps):
    s = ics.plummer(n, seed=seed)
    rng = np.random.default_rng(seed)
    if n > 3:  # coincident stars near and far in state order
        for k in ("px", "py", "pz"):
            s[k][rng.integers(0, n, n // 5)] = s[k][n // 2]
    if gaps:
        s["alive"][rng.random(n) < 0.3] = 0
        s["kind"][rng.random(n) < 0.1] = O.BLACK_HOLE
        s["alive"][TILE:3 * TILE] = 0  # two tiles without a star
        s["alive"][0] = 1
        s["kind"][0] = O.STAR
    return s


@pytest.mark.parametrize("gaps", [False, True])
@pytest.mark.parametrize("n", [1, 2, 255, TILE - 1, TILE, TILE + 1, 5 * TILE, 16 * TILE, 16 * TILE + 1, 50 * TILE + 77,
                               144 * TILE, 144 * TILE + 1, 768 * TILE, 768 * TILE + 1])
def test_keys_and_order(ctx, n, gaps):
    s = state(n, n, gaps)
    acc = [np.zeros(n) for _ in range(3)]
    ctx.call("gbh_accelerations", abi.make_params(0.9, 0.01, 16, walk="plain"), n, P(s["px"]), P(s["py"]), P(s["pz"]),
             P(s["mass"]), P(s["kind"]), P(s["alive"]), *[P(a) for a in acc])
    got = ctx.tree_export()
    want = O.Tree(s["px"], s["py"], s["pz"], s["mass"], s["kind"], s["alive"], theta=0.9, leaf=16).export()
    assert np.array_equal(got["keys"], want["keys"])
    assert np.array_equal(got["order"], want["order"])


@pytest.mark.parametrize("sizes", [(1, 1, 1), (0, TILE, 0, TILE + 1, 5, 0), (17 * TILE, 3, 2 * TILE), (146 * TILE + 9, 1, 700)])
def test_forest_keys_and_order(ctx, sizes):
    parts = [state(k, 7 + q, gaps=q % 2 == 0 and k > 10) if k else None for q, k in enumerate(sizes)]
    real = [p for p in parts if p is not None]
    s = {k: np.concatenate([p[k] for p in real]) for k in real[0]}
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    ctx.forest_upload(off, *[s[k] for k in ("px", "py", "pz", "vx", "vy", "vz")], s["mass"], s["kind"], s["alive"])
    ctx.call("gbh_state_accelerations", abi.make_params(0.9, 0.01, 16, walk="plain"))
    got = ctx.tree_export()
    stars, _ = ctx.forest_layout(len(sizes))
    at = 0
    for q, p in enumerate(parts):
        assert stars[q][0] == at
        at = stars[q][1]
        if p is None:
            continue
        want = O.Tree(p["px"], p["py"], p["pz"], p["mass"], p["kind"], p["alive"], theta=0.9, leaf=16).export()
        lo, hi = stars[q]
        assert np.array_equal(got["keys"][lo:hi], want["keys"])
        assert np.array_equal(got["order"][lo:hi] - off[q], want["order"])
    assert at == len(got["keys"])
