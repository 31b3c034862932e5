"""Resident LDD rounds (k_ldd_rounds, csrc/cc.cu) and the label mode on the device: cluster
properties, the centre schedule and component partitions (exact) where launches pause, turn
wide, meet big vertices, and at the degrees where records and continuations begin and end."""
import math

import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _ring(half, n=3001):
    """A ring whose vertices reach the next `half` ones at stride 5: degree 2 half."""
    v = np.arange(n)
    src = np.concatenate([v] * half)
    dst = np.concatenate([(v + 1 + 5 * k) % n for k in range(half)])
    return psc.HostGraph.from_edges(n, src, dst).symmetrize()


def _stars():
    """Stars of 511 to 9,000 leaves on a path, and loose pairs."""
    src, dst, n = [], [], 6
    for hub, leaves in enumerate([511, 512, 513, 9000, 300]):
        src += [hub] * leaves + [hub]
        dst += list(range(n, n + leaves)) + [hub + 1]
        n += leaves
    for _ in range(200):
        src.append(n)
        dst.append(n + 1)
        n += 2
    return psc.HostGraph.from_edges(n + 3, src, dst).symmetrize()


GRAPHS = {
    "knn": lambda: psc.HostGraph.knn(40013, 5, seed=1).symmetrize(),
    "grid": lambda: psc.HostGraph.grid(150, 401, 0.3, seed=2).symmetrize(),
    "rmat": lambda: psc.HostGraph.rmat(15, 1 << 18, seed=3).symmetrize(),
    "stars": _stars,
    "edges_none": lambda: psc.HostGraph.from_edges(77, [], []).symmetrize(),
    **{f"degree_{2 * h}": (lambda h=h: _ring(h)) for h in (3, 4, 6, 7, 32, 33)},
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("beta", [0.2, 0.004, 2.5])
def test_clusters_schedule_and_components(name, beta):
    g = GRAPHS[name]()
    n = g.n
    comp = O.canon(O.cc(n, g.off, g.E))
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):
            assert np.array_equal(O.canon(dg.cc(beta)), comp)
        lab, par = dg.ldd(beta)
        rows = dg.ldd_rounds()
    at = 0
    for r, (first, work, fresh) in enumerate(rows.tolist(), start=1):
        assert (first, work) == (at, min(math.floor(math.exp(r * beta)), 1024 - at))
        assert fresh <= work
        at += work
    assert at == 1024
    cand = np.unique(np.array([O.lib().orc_hash32_at(1024 + i) % n for i in range(1024)]))
    assert rows[:, 2].sum() == (lab[cand] == cand).sum()
    centres = lab == np.arange(n)
    assert (lab[lab] == lab).all() and (comp[lab] == comp).all()
    assert (par[centres] == np.nonzero(centres)[0]).all()
    v = np.nonzero(~centres)[0]
    assert (lab[par[v]] == lab[v]).all() and np.isin(lab[v], cand).all()
    for x in v[:: max(1, len(v) // 500)].tolist():
        assert par[x] in g.E[g.off[x]:g.off[x + 1]]
