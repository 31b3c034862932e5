"""Device transpose of graphs whose edges leave long runs of vertices without edges (k_edge_sources,
csrc/transpose.cu): exact on both sides of the limit where a tile is searched and not walked, and a
gap inside one tile costs no more than edges spread over the vertices."""
import time

import numpy as np
import pytest

import psc

pytestmark = pytest.mark.gpu

WIDE, TILE = 16 * 3072, 3072


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _csr(n, src, dst):
    order = np.lexsort((dst, src))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(src, minlength=n))
    return off, np.ascontiguousarray(dst[order], dtype=np.uint32)


def _ends(n, m, span):
    """Half of the edges from the first `span` vertices, half from the last."""
    k = np.arange(m)
    return np.where(k < m // 2, k % span, n - 1 - k % span)


SOURCES = {
    **{f"one_gap_{w}": (w + 1, lambda w=w: np.repeat([0, w], [5, 6]))
       for w in (WIDE - 1, WIDE, WIDE + 1)},
    "two_vertices_far": (300_000, lambda: np.repeat([0, 299_999], [TILE - 1, TILE + 1])),
    "last_edge_far": (300_000, lambda: np.repeat([7, 299_999], [2 * TILE - 1, 1])),
    "scattered": (3_000_001, lambda: np.random.default_rng(3).integers(0, 3_000_001, 20_003)),
    "ends": (5_000_000, lambda: _ends(5_000_000, 50_001, 1000)),
}


@pytest.mark.parametrize("name", sorted(SOURCES))
def test_wide_tiles(name):
    n, make = SOURCES[name]
    src = make()
    dst = np.random.default_rng(len(name)).integers(0, n, len(src))
    off, E = _csr(n, src, dst)
    in_off, in_E = _csr(n, dst, src)
    with psc.DeviceGraph.directed(off, E) as dg:
        got_off, got_E = dg.transpose()
        assert np.array_equal(got_off, in_off) and np.array_equal(got_E, in_E)


def test_a_gap_costs_no_walk():
    n, m = 1 << 25, 100_000
    dst = np.random.default_rng(1).integers(0, n, m)
    ms = {}
    for name, src in (("even", np.random.default_rng(2).integers(0, n, m)), ("ends", _ends(n, m, 1000))):
        off, E = _csr(n, src, dst)
        best = []
        for _ in range(6):
            t = time.perf_counter()
            dg = psc.DeviceGraph.directed(off, E)
            best.append(1e3 * (time.perf_counter() - t))
            dg.free()
        ms[name] = min(best)
    # (walked by one block: 25 ms at half this size)
    assert ms["ends"] < 4 * ms["even"] + 2, ms
