"""Hubs among narrow levels (csrc/levels.cuh): BFS distances and allocation-free reachability where
vertices around the cluster's degree bound follow each other, exact, and a search from a hub costs no
multiple of one from any other vertex."""
import ctypes as C
import time

import numpy as np
import pytest

import psc
import pyoracle as O
from psc import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _chain(degrees, gap):
    """A path on which every gap-th vertex has that many leaves as well, and a far vertex with
    edges enough to keep the searches pushing."""
    n = gap * len(degrees)
    src, dst = [np.arange(n - 1)], [np.arange(1, n)]
    for k, d in enumerate(degrees):
        src.append(np.full(d, k * gap))
        dst.append(n + np.arange(d))
        n += d
    extra = np.arange(400_000)
    src.append(n + extra % 1000)
    dst.append(n + extra // 1000 % 1000)
    return psc.HostGraph.from_edges(n + 1000, np.concatenate(src), np.concatenate(dst))


def _noalloc(g, src):
    lib = psc.cuda()
    ptr = []
    for a in (g.off, g.E, g.in_off, g.in_E):
        p = C.c_void_p()
        _lib.check(lib.psc_device_alloc(a.nbytes, C.byref(p)), "alloc")
        _lib.check(lib.psc_copy(p, a.ctypes.data, a.nbytes), "copy")
        ptr.append(p)
    d, out, r = C.c_void_p(), np.empty(g.n, np.uint8), C.c_uint32()
    _lib.check(lib.psc_device_alloc(g.n, C.byref(d)), "alloc")
    t = []
    try:
        for _ in range(15):
            t0 = time.perf_counter()
            _lib.check(lib.psc_reach_noalloc(*ptr, g.n, g.m, src, 0, d, None, C.byref(r)), "reach")
            t.append(time.perf_counter() - t0)
        _lib.check(lib.psc_copy(out.ctypes.data, d, g.n), "copy")
    finally:
        for p in ptr + [d]:
            lib.psc_device_free(p)
    return out, 1e3 * float(np.median(t))


@pytest.mark.parametrize("gap", [1, 2, 3, 11])
@pytest.mark.parametrize("top", [1023, 1024, 1025, 9000])
def test_hubs_on_a_path(gap, top):
    g = _chain([top, 3, top, top, 0, 1024, 1025, 9000] * 2, gap)
    with psc.DeviceGraph(g) as dg:
        for src in (0, gap, 2 * gap - 1):
            assert np.array_equal(dg.bfs(src), O.bfs_seq(g.n, g.off, g.E, src))
            assert np.array_equal(_noalloc(g, src)[0] != 0, O.reach_seq(g.n, g.off, g.E, src) != 0)


def test_sources_without_edges_and_hubs_alone():
    g = psc.HostGraph.from_edges(20_002, np.zeros(20_000, np.int64), np.arange(1, 20_001))
    with psc.DeviceGraph(g) as dg:
        for src in (0, 5, 20_001):
            assert np.array_equal(dg.bfs(src), O.bfs_seq(g.n, g.off, g.E, src))


def test_hub_source_costs_no_more():
    g = psc.HostGraph.rmat(18, 16 << 18, seed=1).symmetrize()
    hub = int(np.argmax(np.diff(g.off.astype(np.int64))))
    with psc.DeviceGraph(g) as dg:
        ms = {}
        for src in (hub, 5):
            t = []
            for _ in range(25):
                t0 = time.perf_counter()
                dg.bfs(src)
                t.append(time.perf_counter() - t0)
            ms[src] = 1e3 * float(np.median(t))
    # (one warp on the hub: 0.92 and 0.30 ms)
    assert ms[hub] < 1.6 * ms[5], ms
    g = psc.HostGraph.rmat(20, 16 << 20, seed=1)
    hub = int(np.argmax(np.diff(g.off.astype(np.int64))))
    a, b = _noalloc(g, hub)[1], _noalloc(g, 5)[1]
    # (1.79 and 0.48 ms)
    assert a < 1.6 * b, (a, b)
