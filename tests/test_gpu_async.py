"""Searches without rounds (k_reach_async, k_reach_async_low in csrc/reach.cu): reach sets
in both directions and SCC labels against the oracle (exact), at the degrees where records and
continuations begin and end, and where a launch stops for the rounds to go on."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _edges(n, *pairs):
    return psc.HostGraph.from_edges(n, np.concatenate([a for a, _ in pairs]),
                                    np.concatenate([b for _, b in pairs]))


def _regular(d, n=4001):
    """A ring whose vertices also lead to the d - 1 next ones but one: out- and in-degree d."""
    v = np.arange(n)
    return _edges(n, *[(v, (v + 1 + k * 3) % n) for k in range(d)])


def _strip(first, rows, cols, seed):
    g = psc.HostGraph.grid(rows, cols, 0.9, seed=seed)
    s, t = g.edge_list()
    return s.astype(np.int64) + first, t.astype(np.int64) + first


def _hub_behind_strip():
    """A long narrow strip, then a vertex with 9,000 out-edges, then another strip."""
    hub = 12000
    leaves = hub + 1 + np.arange(9000)
    second = hub + 9001
    return _edges(second + 12000, _strip(0, 3, 4000, 1),
                  (np.arange(0, 12000, 500), np.full(24, hub)),
                  (np.full(9000, hub), leaves), (leaves[::100], second + np.arange(90)),
                  _strip(second, 3, 4000, 2), (np.array([second + 11999]), np.array([0])))


def _tree(depth):
    n = (1 << (depth + 1)) - 1
    child = np.arange(1, n)
    return _edges(n, ((child - 1) // 2, child))


def _ladder(n=20000):
    v = np.arange(n - 1)
    return _edges(n, (v, v + 1), (v[::7] + 1, v[::7]))


def _band(top, n=60011):
    """Vertex u leads to up to top of the 40 after it (every 5th to the next one too); one vertex
    of 70 out-edges keeps the graph off the records."""
    r = np.random.default_rng(top)
    d = r.integers(0, top + 1, n)
    s = np.repeat(np.arange(n), d)
    v = np.arange(0, n, 5)
    return _edges(n, (s, (s + r.integers(1, 41, len(s))) % n), (v, (v + 1) % n),
                  (np.full(70, 11), 12 + np.arange(70)))


GRAPHS = {
    "ladder": (_ladder, 0),
    "grid": (lambda: psc.HostGraph.grid(301, 217, 0.5, seed=3), 4000),
    "knn": (lambda: psc.HostGraph.knn(30011, 5, seed=4), 17),
    "hub_behind_strip": (_hub_behind_strip, 0),
    # eight lanes per entry up to degree 8, the balanced expansion above it
    "band_7": (lambda: _band(7), 3),
    "band_8": (lambda: _band(8), 3),
    "band_11": (lambda: _band(11), 3),
    "tree": (lambda: _tree(17), 0),
    **{f"degree_{d}": (lambda d=d: _regular(d), 7) for d in (1, 5, 6, 7, 12, 13, 63, 64, 65)},
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_reach_and_scc_equal_oracle(name):
    make, src = GRAPHS[name]
    g = make()
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):  # the second pass meets what the first one left on the handle
            assert np.array_equal(dg.reach(src), O.reach_seq(g.n, g.off, g.E, src))
            assert np.array_equal(dg.reach(src, backward=True),
                                  O.reach_seq(g.n, g.in_off, g.in_E, src))
        if name != "tree":
            got = dg.scc(psc.default_params(seed=5))
            assert np.array_equal(got, O.scc(g.n, g.off, g.E, g.in_off, g.in_E, seed=5))
