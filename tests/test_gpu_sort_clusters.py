"""Clusters of stars far tighter than the sort word's resolution: runs of equal words of every length around
the line between counting and a second pass of the network, up to a whole tile, with stars of different
keys and of equal ones in them, in state order and shuffled, with dead bodies between."""
import numpy as np
import pytest

from gravitas_gb300 import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu
P = abi.ptr


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("n,cluster", [(40, 2), (600, 7), (600, 8), (600, 9), (600, 10), (1024, 33), (1024, 1022),
                                       (2500, 500), (2500, 1024), (5000, 2000), (40_000, 9), (40_000, 30_000)])
def test_clusters(n, cluster, shuffle):
    rng = np.random.default_rng(n + cluster)
    p = rng.uniform(-1.0, 1.0, (n, 3))
    p[0], p[1] = -1.0, 1.0
    cell = 2.0 / 2**21
    k = 2  # clusters, each in a few cells of the finest level: some stars share all of them, some none
    while k + cluster <= n:
        p[k:k + cluster] = rng.uniform(-0.9, 0.9, 3) + rng.integers(0, 4, (cluster, 3)) * cell
        k += cluster
    if shuffle:
        p = p[rng.permutation(n)]
    alive = np.ones(n, np.uint8)
    alive[rng.random(n) < 0.05] = 0
    x, y, z = (p[:, c].copy() for c in range(3))
    mass, acc = np.full(n, 1.0 / n), [np.zeros(n) for _ in range(3)]
    with abi.Context(0) as ctx:
        ctx.call("gbh_accelerations", abi.make_params(0.9, 0.05, 16, walk="plain"), n, P(x), P(y), P(z), P(mass), None,
                 P(alive), *[P(a) for a in acc])
        got = ctx.tree_export()
    want = O.Tree(x, y, z, mass, None, alive, theta=0.9, leaf=16).export()
    assert np.array_equal(got["keys"], want["keys"])
    assert np.array_equal(got["order"], want["order"])
