"""Resident search rounds (k_reach_rounds, csrc/reach.cu): reach sets and round counts in both
directions (exact) on graphs that push, pull, meet heavy vertices (257 and more out-edges) and
go on after the launch's last round; with and without local searches."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _depth(n, off, E, src):
    seen = np.zeros(n, bool)
    seen[src] = True
    front, rounds = np.array([src]), 0
    while len(front):
        rounds += 1
        nxt = np.concatenate([E[int(off[u]):int(off[u + 1])] for u in front])
        front = np.unique(nxt[~seen[nxt]])
        seen[front] = True
    return rounds


def _fans(sizes):
    """A path of hubs with the given out-degrees; every leaf leads to the next hub."""
    src, dst, n = [], [], len(sizes) + 1
    for hub, d in enumerate(sizes):
        leaves = n + np.arange(d - 1)
        src += [np.full(d, hub), leaves]
        dst += [np.append(leaves, hub + 1), np.full(d - 1, hub + 1)]
        n += d - 1
    return psc.HostGraph.from_edges(n + 1, np.concatenate(src), np.concatenate(dst))


GRAPHS = {
    "rmat": (lambda: psc.HostGraph.rmat(13, 1 << 16, seed=1), 3),
    "fans": (lambda: _fans([255, 256, 257, 258, 511, 513, 4000, 70]), 0),
    "fans_deep": (lambda: _fans([70] * 60), 0),
    "dense": (lambda: psc.HostGraph.from_edges(97, np.repeat(np.arange(97), 97),
                                               np.tile(np.arange(97), 97)), 5),
    "single": (lambda: psc.HostGraph.from_edges(1, [], []), 0),
    "words": (lambda: psc.HostGraph.rmat(6, 3000, seed=2), 0),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("local", [True, False])
def test_sets_and_rounds(name, local):
    make, src = GRAPHS[name]
    g = make()
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):
            for back, off, E in ((False, g.off, g.E), (True, g.in_off, g.in_E)):
                got = dg.reach(src, backward=back, local=local)
                assert np.array_equal(got, O.reach_seq(g.n, off, E, src))
                if not local:
                    assert dg.last_rounds == _depth(g.n, off, E, src)
        got = dg.scc(psc.default_params(seed=4, local_reach=int(local)))
        assert np.array_equal(got, O.scc(g.n, g.off, g.E, g.in_off, g.in_E, seed=4))
