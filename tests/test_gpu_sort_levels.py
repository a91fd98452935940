"""A forest whose largest system takes four merges (more than 1,728 sort tiles), beside small systems."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu
P = abi.ptr


def test_four_merges():
    sizes = (100, 1728 * 1024 + 7, 3000)
    parts = [ics.plummer(n, seed=n % 97) for n in sizes]
    parts[1]["alive"][::50] = 0
    s = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    with abi.Context(0) as ctx:
        ctx.forest_upload(off, *[s[k] for k in ("px", "py", "pz", "vx", "vy", "vz")], s["mass"], s["kind"], s["alive"])
        ctx.call("gbh_state_accelerations", abi.make_params(0.9, 0.01, 32, walk="plain"))
        got, (stars, _) = ctx.tree_export(), ctx.forest_layout(len(sizes))
    for q, p in enumerate(parts):
        want = O.Tree(p["px"], p["py"], p["pz"], p["mass"], p["kind"], p["alive"], theta=0.9, leaf=32).export()
        lo, hi = stars[q]
        assert np.array_equal(got["keys"][lo:hi], want["keys"])
        assert np.array_equal(got["order"][lo:hi] - off[q], want["order"])
