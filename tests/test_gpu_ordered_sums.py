"""FP64 pair sums whose terms are formed in parallel and added in order: bit identical to the
oracle's serial loops at the edges of their tiles."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu
P = abi.ptr


@pytest.fixture(scope="module")
def ctx():
    c = abi.Context(0)
    yield c
    c.close()


def disk(n, seed=3):
    """n bodies: the test disk with its two holes, some dark matter, two bodies at one place."""
    s = ics.test_disk(max(n, 3) - 2, seed=seed)
    s["kind"][1:n - 1:7] = O.DARK_MATTER
    s["px"][n // 2], s["py"][n // 2], s["pz"][n // 2] = s["px"][1], s["py"][1], s["pz"][1]
    return {k: np.ascontiguousarray(v[:n]) for k, v in s.items()}


@pytest.mark.parametrize("n,ntargets", [(1, 1), (2, 2), (63, 5), (64, 64), (65, 1), (255, 9), (257, 33), (3001, 304),
                                        (3001, 2433), (5000, 5000)])
def test_direct_sum_bit_identical(ctx, n, ntargets):
    s = disk(n)
    tg = np.sort(np.random.default_rng(n).choice(n, ntargets, replace=False)).astype(np.int64)
    for dm_off in (False, True):
        got = np.full((3, ntargets), 7.0)
        ctx.call("gbh_direct_accelerations", abi.make_params(0, 0.03, 0, False, dm_off, "fp64"), n, P(s["px"]),
                 P(s["py"]), P(s["pz"]), P(s["mass"]), P(s["kind"]), P(tg), ntargets, *[P(g) for g in got])
        want = O.direct(s["px"], s["py"], s["pz"], s["mass"], s["kind"], eps=0.03, dm_off=dm_off, targets=tg)
        assert np.array_equal(got.T, want)


def upload(ctx, s):
    ctx.call("gbh_state_upload", len(s["px"]), *[P(s[k]) for k in ("px", "py", "pz", "vx", "vy", "vz")], None, None, None,
             P(s["mass"]), P(s["kind"]), P(s["alive"]))


@pytest.mark.parametrize("n", [1, 2, 31, 63, 64, 65, 607, 2047, 2049, 4097])
def test_exact_potential_bit_identical(ctx, n):
    s = disk(n)
    upload(ctx, s)
    for dm_off, c in ((False, 0.0), (True, 0.0), (True, 4.0), (False, 4.0), (False, -1.0)):
        d = ctx.diagnostics(abi.make_params(0.5, 0.03, 8, False, dm_off, "mixed"), c)
        assert d["quality"] == 2
        assert d["potential"] == O.potential_exact(s["px"], s["py"], s["pz"], s["mass"], s["kind"], 0.03, c, dm_off)


@pytest.mark.parametrize("n,nholes,scale", [(3, 1, 1.0), (255, 2, 1.0), (256, 1, 0.1), (257, 8, 0.3), (512, 2, 0.1), (513, 2, 0.1), (600, 15, 0.3), (1200, 3, 0.1)])
def test_hole_steps_bit_identical(ctx, n, nholes, scale):
    """Hole counts at the edges of the batches, few to all stars near a hole (scale shrinks the disk),
    a dead hole with an acceleration of its own."""
    s = ics.test_disk(n, seed=5, holes=False)
    for k in ("px", "py", "pz"):
        s[k] *= scale
    at = np.linspace(0, n - 1, nholes).astype(int)
    s["kind"][at] = O.BLACK_HOLE
    s["mass"][at] = 2.0 / nholes
    dead = int(at[-1]) if nholes > 2 else -1
    if dead >= 0:
        s["alive"][dead] = 0
        s["ax"][dead] = 0.25
    f9 = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")
    got = {k: s[k].copy() for k in (*f9, "mass", "kind", "alive")}
    ref = {k: v.copy() for k, v in got.items()}
    ctx.call("gbh_step_kdk", abi.make_params(0.5, 0.06, 8, False, False, "fp64"), 4e-3, 3, 1, n, *[P(got[k]) for k in f9],
             P(s["mass"]), P(s["kind"]), P(s["alive"]))
    O.split_kdk(ref, 4e-3, 0.06, 0.5, 8, 3, acc_valid=True)
    for k in f9:
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("n", [1, 5, 2432, 2433, 4863, 4865, 9728, 9729, 12001])
def test_fp64_walk_bit_identical(ctx, n):
    """4, 8, 16 and 32 stars a warp, the last warp full or not."""
    s = disk(n)
    got = [np.zeros(n) for _ in range(3)]
    ctx.call("gbh_accelerations", abi.make_params(0.7, 0.03, 8, walk="fp64"), n, P(s["px"]), P(s["py"]), P(s["pz"]),
             P(s["mass"]), P(s["kind"]), P(s["alive"]), *[P(g) for g in got])
    tree = O.Tree(s["px"], s["py"], s["pz"], s["mass"], s["kind"], s["alive"], theta=0.7, leaf=8)
    assert np.array_equal(np.stack(got, 1), tree.accelerations(0.03))
