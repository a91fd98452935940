"""Arrays in memory that nothing has written yet, and calls that mix aligned arrays with misaligned ones,
give what arrays in use give, and no byte beside an array changes."""
import mmap

import numpy as np
import pytest

from gravitas_gb300 import abi, ics

pytestmark = pytest.mark.gpu
P = abi.ptr
F9 = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")


def untouched(n):
    """n doubles (zeros) in the middle of a mapping that nothing has written."""
    m = mmap.mmap(-1, 8 * n + (1 << 18), flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    return np.frombuffer(m, np.float64)[1000:1000 + n], m


# few pages: the kernel's way, in use or not; 100,001 and 262,144 by copies when new; beyond: always
@pytest.mark.parametrize("n", [1000, 30_000, 100_001, 262_144, 262_145])
def test_new_pages(n):
    s = ics.plummer(n, seed=n)
    par = abi.make_params(0.9, 0.02, 24)
    with abi.Context(0) as ctx:
        def accelerations(a):
            ctx.call("gbh_accelerations", par, n, P(s["px"]), P(s["py"]), P(s["pz"]), P(s["mass"]), None, None,
                     *[P(x) for x in a])

        def kdk(a, acc_valid):
            for k, x in zip(F9[:6], a):
                x[:] = s[k]
            ctx.call("gbh_step_kdk", par, 1e-3, 1, acc_valid, n, *[P(x) for x in a], P(s["mass"]), None, None)

        for call, count in ((accelerations, 3), (lambda a: kdk(a, 0), 9), (lambda a: kdk(a, 1), 9)):
            want, new = [np.zeros(n) for _ in range(count)], [untouched(n) for _ in range(count)]
            for w in want:
                w[:] = 0.0
            for _ in range(2):  # new, then in use
                call(want)
                call([x for x, _ in new])
                for w, (x, m) in zip(want, new):
                    assert np.array_equal(w, x)
                    around = np.frombuffer(m, np.uint8)
                    assert not around[:8000].any() and not around[8000 + 8 * n:].any()
        out = [untouched(n) for _ in range(9)]  # written without being read
        ctx.call("gbh_state_download", *[P(x) for x, _ in out])
        for w, (x, _) in zip(want, out):
            assert np.array_equal(w, x)


@pytest.mark.parametrize("n", [257, 40_000])
@pytest.mark.parametrize("odd", ["px", "vz", "ay"])
def test_one_misaligned_array(n, odd):
    s = ics.plummer(n, seed=n)
    par = abi.make_params(0.9, 0.02, 24)
    with abi.Context(0) as ctx:
        want, got = {k: s[k].copy() for k in F9}, {k: s[k].copy() for k in F9}
        raw = np.zeros(8 * n + 16, np.uint8)
        raw[4:4 + 8 * n] = s[odd].view(np.uint8)
        ctx.call("gbh_step_kdk", par, 1e-3, 2, 0, n, *[P(want[k]) for k in F9], P(s["mass"]), None, None)
        at = {k: P(raw.ctypes.data + 4) if k == odd else P(got[k]) for k in F9}
        ctx.call("gbh_step_kdk", par, 1e-3, 2, 0, n, *[at[k] for k in F9], P(s["mass"]), None, None)
        got[odd] = raw[4:4 + 8 * n].copy().view(np.float64)
        for k in F9:
            assert np.array_equal(got[k], want[k]), k
        assert not raw[:4].any() and not raw[4 + 8 * n:].any()
