"""Resident LE-list batches (k_le_batches) and the split push levels of BFS (k_bfs_heavy,
csrc/lelist.cu): lists and distances against the sequential oracle (exact) where pairs become
heavy, where the list is extended between launches, and where a batch outgrows the
table and the host takes it over."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _stars(sizes, loose=7):
    """Stars of the given sizes whose hubs form a ring, and loose vertices."""
    k, src, dst, n = len(sizes), [], [], len(sizes)
    for hub, leaves in enumerate(sizes):
        src += [hub] * leaves + [hub]
        dst += list(range(n, n + leaves)) + [(hub + 1) % k]
        n += leaves
    return psc.HostGraph.from_edges(n + loose, src, dst).symmetrize()


GRAPHS = {
    "path": lambda: psc.HostGraph.from_edges(1500, np.arange(1499), np.arange(1, 1500)).symmetrize(),
    "stars_around_the_split": lambda: _stars([125, 126, 127, 128, 253, 254, 255, 256, 400]),
    "big_stars": lambda: _stars([9000, 300, 8192, 5]),
    "rmat": lambda: psc.HostGraph.rmat(12, 1 << 15, seed=4).symmetrize(),
    "knn": lambda: psc.HostGraph.knn(4003, 5, seed=5).symmetrize(),
    "two_vertices": lambda: psc.HostGraph.from_edges(2, [0], [1]).symmetrize(),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("beta", [1.5, 1.05, 400.0])
def test_lists_equal_oracle(name, beta):
    g = GRAPHS[name]()
    perm = psc.random_permutation(g.n, 11)
    want = np.asarray(O.lelist_seq(g.n, g.off, g.E, perm)).reshape(-1, 3)
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):
            assert np.array_equal(dg.lelist(perm, beta=beta), want)
        for src in (0, g.n - 1):
            assert np.array_equal(dg.bfs(src), O.bfs_seq(g.n, g.off, g.E, src))
