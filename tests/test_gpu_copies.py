"""The copies of a call's arrays: by one kernel on the caller's memory (small, aligned arrays), or array
by array (misaligned, or more than 2^18 elements). Both give the same results, bit for bit."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics

pytestmark = pytest.mark.gpu
P = abi.ptr
LIMIT = 1 << 18


def shifted(a, by):
    """A copy of a at an address `by` bytes off its alignment."""
    raw = np.zeros(a.nbytes + 64, np.uint8)
    view = raw[by:by + a.nbytes]
    view[:] = np.ascontiguousarray(a).view(np.uint8)
    return raw, raw.ctypes.data + by


@pytest.mark.parametrize("n", [1, 255, 1000, 16385])
def test_misaligned_arrays(n):
    s = ics.plummer(n, seed=n)
    par = abi.make_params(0.7, 0.02, 16)
    f9 = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")
    with abi.Context(0) as ctx:
        want = {k: s[k].copy() for k in f9}
        ctx.call("gbh_step_kdk", par, 1e-3, 2, 0, n, *[P(want[k]) for k in f9], P(s["mass"]), P(s["kind"]), P(s["alive"]))
        for by in (1, 4):
            got = {k: shifted(s[k], by) for k in (*f9, "mass", "kind", "alive")}
            ctx.call("gbh_step_kdk", par, 1e-3, 2, 0, n, *[P(got[k][1]) for k in (*f9, "mass", "kind", "alive")])
            for k in f9:
                assert np.array_equal(got[k][0][by:by + 8 * n].view(np.uint8), want[k].view(np.uint8)), k


@pytest.mark.parametrize("n", [LIMIT, LIMIT + 1])
def test_arrays_at_the_limit(n):
    """Small systems of a forest in one upload and download: every element comes back as it went."""
    rng = np.random.default_rng(n)
    cols = [rng.normal(size=n) for _ in range(9)]
    mass, kind, alive = rng.uniform(0.5, 1.0, n), np.zeros(n, np.uint8), np.ones(n, np.uint8)
    out = [np.empty(n) for _ in range(9)]  # pages that nothing has touched
    with abi.Context(0) as ctx:
        ctx.call("gbh_state_upload", n, *[P(c) for c in cols], P(mass), P(kind), P(alive))
        ctx.call("gbh_state_download", *[P(o) for o in out])
        for a, b in zip(out, cols):
            assert np.array_equal(a, b)
        ctx.call("gbh_state_download", None, P(out[1]), None, None, None, None, None, None, P(out[0]))
        assert np.array_equal(out[1], cols[1]) and np.array_equal(out[0], cols[8])
