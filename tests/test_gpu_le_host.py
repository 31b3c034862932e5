"""LE-lists launched level by level from the host (graphs above 2^23 vertices, csrc/lelist.cu): the
lists of a graph among loose vertices equal the graph's own, with pairs on both sides of the split
between light and heavy ones."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


def test_large_graph_of_mostly_loose_vertices(cuda_device):
    r = np.random.default_rng(8)
    hubs = [255, 256, 257, 128, 129, 3000]
    n = 6000
    src = np.concatenate([np.repeat(np.arange(len(hubs)), hubs), r.integers(0, n, 9000)])
    dst = np.concatenate([r.integers(len(hubs), n, sum(hubs)), r.integers(0, n, 9000)])
    small = psc.HostGraph.from_edges(n, src, dst).symmetrize()
    order = psc.random_permutation(n, 3)
    want = np.asarray(O.lelist_seq(n, small.off, small.E, order)).reshape(-1, 3)
    extra = (1 << 23) + 5
    g = psc.HostGraph.from_edges(n + extra, src, dst).symmetrize()
    perm = np.concatenate([order, np.arange(n, n + extra, dtype=np.uint32)]).astype(np.uint32)
    with psc.DeviceGraph(g) as dg:
        got = dg.lelist(perm)
    assert np.array_equal(got[got[:, 0] < n], want)
    loose = got[got[:, 0] >= n]
    assert len(loose) == extra and np.array_equal(loose[:, 0], loose[:, 1]) and not loose[:, 2].any()
