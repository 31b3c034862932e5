"""Tables of the resident LE-list batches (csrc/lelist.cu) hold the batches of spatial graphs, also
where vertex counts lie at a power of two and batches grow by 3: none is done twice, so the whole call
is a few dozen launches.  Both widths of the kernel equal each other's lists."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


def test_batches_of_knn_fit(cuda_device):
    g = psc.HostGraph.knn(1 << 21, 5, seed=1).symmetrize()
    perm = psc.random_permutation(g.n, 11)
    with psc.DeviceGraph(g) as dg:
        lists = []
        for beta in (1.5, 3.0):  # (the lists do not depend on it)
            lists.append(dg.lelist(perm, beta=beta))
            # (a level launched from the host is one launch at least, a batch hundreds of levels)
            assert dg.stats().kernel_launches < 200
        assert np.array_equal(*lists)


def test_wide_graphs(cuda_device):
    """More than 2^21 vertices (the wide kernel) against the same graph among loose vertices."""
    r = np.random.default_rng(5)
    n, m = 5000, 20000
    src, dst = r.integers(0, n, m), r.integers(0, n, m)
    lists = []
    for extra in (0, (1 << 21) + 1):
        g = psc.HostGraph.from_edges(n + extra, src, dst).symmetrize()
        perm = np.concatenate([psc.random_permutation(n, 3),
                               np.arange(n, n + extra, dtype=np.uint32)]).astype(np.uint32)
        with psc.DeviceGraph(g) as dg:
            got = dg.lelist(perm)
        lists.append(got[got[:, 0] < n])
        loose = got[got[:, 0] >= n]
        assert len(loose) == extra and np.array_equal(loose[:, 0], loose[:, 1]) and not loose[:, 2].any()
    assert np.array_equal(*lists)
    assert np.array_equal(lists[0], np.asarray(O.lelist_seq(
        n, *(lambda g: (g.off, g.E))(psc.HostGraph.from_edges(n, src, dst).symmetrize()),
        psc.random_permutation(n, 3))).reshape(-1, 3))
