"""Builds in buffers that have just been allocated, on device memory that other contexts have used: the
first build after every growth gives the oracle's tree, and a block step the same bits in every context."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu
P = abi.ptr
F9 = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")


def block_steps(ctx, s):
    n = len(s["px"])
    ctx.call("gbh_state_upload", n, *[P(s[k]) for k in F9[:6]], None, None, None, P(s["mass"]), None, None)
    ctx.step_block(abi.make_params(0.7, 0.02, 16), 0.016, 0.025, 5, 1)
    out = [np.zeros(n) for _ in F9]
    ctx.call("gbh_state_download", *[P(o) for o in out])
    return out


def test_first_build_after_growth():
    want, sizes = {}, (300, 5_000, 60_000, 300_000)
    for n in sizes:
        s = ics.plummer(n, seed=n)
        want[n] = s, O.Tree(s["px"], s["py"], s["pz"], s["mass"], theta=0.7, leaf=16).export()
    for _ in range(4):
        with abi.Context(0) as ctx:  # grows at every size; closing it leaves its memory behind
            for n in sizes:
                s, e = want[n]
                acc = [np.zeros(n) for _ in range(3)]
                ctx.call("gbh_accelerations", abi.make_params(0.7, 0.02, 16, walk="plain"), n, P(s["px"]), P(s["py"]),
                         P(s["pz"]), P(s["mass"]), None, None, *[P(a) for a in acc])
                g = ctx.tree_export()
                assert np.array_equal(g["keys"], e["keys"]) and np.array_equal(g["order"], e["order"]), n


def test_first_block_step_in_fresh_contexts():
    s = ics.galaxy(30_000, seed=4)
    first = None
    for _ in range(4):
        with abi.Context(0) as ctx:
            got = block_steps(ctx, s)
        first = first or got
        for a, b in zip(got, first):
            assert np.array_equal(a, b)


def test_forest_layouts_one_after_another():
    """Every upload's layout reaches the build that follows it at once."""
    sizes = ((900, 1500, 40), (40, 2300, 100), (1200, 1200, 40), (2439, 0, 1))
    with abi.Context(0) as ctx:
        for k in range(12):
            parts = [ics.plummer(n, seed=10 * k + n) for n in sizes[k % 4] if n]
            s = {f: np.concatenate([p[f] for p in parts]) for f in parts[0]}
            off = np.concatenate([[0], np.cumsum(sizes[k % 4])]).astype(np.int64)
            ctx.forest_upload(off, *[s[f] for f in F9[:6]], s["mass"])
            ctx.call("gbh_state_accelerations", abi.make_params(0.7, 0.02, 16, walk="plain"))
            g, at = ctx.tree_export(), 0
            for p in parts:
                e = O.Tree(p["px"], p["py"], p["pz"], p["mass"], theta=0.7, leaf=16).export()
                assert np.array_equal(g["keys"][at:at + len(e["keys"])], e["keys"])
                at += len(e["keys"])
