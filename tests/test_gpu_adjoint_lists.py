"""Tree adjoint at the edges of its source lists, which take four stars at a time (every remainder of
four and of a warp, split walks whose parts hold a few stars): with a tiny opening angle it is the
direct-sum adjoint, here in FP64. The lists are summed in FP32: each term within a few rounding errors
of 2^-24, a sum of at most 130 of them well within 2e-5 of the gradient's norm."""
import numpy as np
import pytest

from gravitas_gb300 import abi, ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 31, 32, 33, 34, 63, 65, 66, 67, 130])
def test_few_stars_tree_adjoint_is_the_direct_adjoint(n):
    s, targets = ics.adjoint_problem(n, seed=n)
    x0, v0 = (np.stack([s[a + b] for b in "xyz"], 1) for a in "pv")
    with abi.Context(0) as ctx:
        got = {}
        for key, args in (("tree", (abi.ADJ_FP32, abi.ADJ_TREE, 1e-4, 8)), ("direct", (abi.ADJ_FP64, abi.ADJ_DIRECT))):
            x, _ = ctx.fwd_save(x0, v0, s["mass"], 1e-3, 0.05, 5, 2, *args)
            got[key] = ctx.bwd(2.0 * (x - targets) / n, None)
    for a, b in zip(got["tree"], got["direct"]):
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b)
