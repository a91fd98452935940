"""The FP64 walk of target lists (block steps) and of few stars in a large context: the stars a warp holds
follow the body count, so dead bodies behind the same stars change them, and no bit of the stars."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics

pytestmark = pytest.mark.gpu
P = abi.ptr
F9 = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az")


def padded(s, n):
    k = n - len(s["px"])
    t = {f: np.concatenate([s[f], np.zeros(k, s[f].dtype)]) for f in s}
    t["alive"][n - k:] = 0
    return t


def upload(ctx, s):
    ctx.call("gbh_state_upload", len(s["px"]), *[P(s[k]) for k in F9[:6]], None, None, None, P(s["mass"]), P(s["kind"]),
             P(s["alive"]))


def state(ctx, n):
    out = [np.zeros(n) for _ in F9]
    ctx.call("gbh_state_download", *[P(o) for o in out])
    return np.stack(out)


# 4, 8, 16 and 32 stars a warp on 152 SMs
def test_block_steps_with_any_stars_a_warp():
    s = ics.galaxy(2000, seed=8)
    par, want = abi.make_params(0.6, 0.02, 8, walk="fp64"), None
    for n in (2000, 2433, 4000, 4865, 9000, 9729, 14_000):
        with abi.Context(0) as ctx:
            upload(ctx, padded(s, n))
            st = ctx.step_block(par, 0.016, 0.025, 6, 2)
            got = state(ctx, n)[:, :2000]
        assert st["substeps"] > 4  # lists of some of the stars
        want = got if want is None else want
        assert np.array_equal(got, want), n


@pytest.mark.parametrize("n", [1, 33, 1000, 5000])
def test_few_stars_in_a_large_context(n):
    s, par = ics.plummer(n, seed=n), abi.make_params(0.6, 0.02, 8, walk="fp64")
    got = []
    for size in (0, 300_000):
        with abi.Context(0) as ctx:
            if size:
                upload(ctx, ics.plummer(size, seed=1))
                ctx.call("gbh_state_accelerations", abi.make_params(0.9, 0.02, 24))
            upload(ctx, s)
            ctx.call("gbh_state_accelerations", par)
            got.append(state(ctx, n))
    assert np.array_equal(got[0], got[1])
