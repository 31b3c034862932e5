"""Narrow search levels on one thread-block cluster (csrc/levels.cuh): BFS
distances and push reachability at the sizes where it hands back to the wide
rounds, against distances by definition (exact)."""
import ctypes as C

import numpy as np
import pytest

import psc
from psc import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _bfs(g, src):
    dist = np.full(g.n, 0xFFFFFFFF, np.uint32)
    dist[src] = 0
    front, level = np.array([src]), 0
    while len(front):
        level += 1
        nxt = np.concatenate([g.E[int(g.off[u]):int(g.off[u + 1])] for u in front])
        front = np.unique(nxt[dist[nxt] == 0xFFFFFFFF])
        dist[front] = level
    return dist, level


def _tree(fan, extra=1_700_000):
    """Levels of sizes 1, fan[0], fan[0]*fan[1], ... below vertex 0 (the last vertices of each
    level lead on in a path), and enough unrelated edges to keep the search pushing."""
    src, dst, first, n = [], [], 0, 1
    width = 1
    for f in fan:
        u = np.repeat(np.arange(first, first + width), f)
        v = n + np.arange(width * f)
        src.append(u)
        dst.append(v)
        first, width, n = n, width * f, n + width * f
    path = np.arange(n - 1, n + 40)
    src.append(path[:-1])
    dst.append(path[1:])
    n += 40
    side = 1500
    e = np.arange(extra)
    src.append(n + e % side)
    dst.append(n + (e // side) % side)
    n += side
    return psc.HostGraph.from_edges(n, np.concatenate(src), np.concatenate(dst))


def _band(top, n=20_011):
    """Vertex u has 0 to top edges into the 60 vertices after it (and u -> u + 1 every 7th)."""
    rng = np.random.default_rng(top)
    deg = rng.integers(0, top + 1, n)
    src = np.repeat(np.arange(n), deg)
    dst = np.minimum(src + rng.integers(1, 61, len(src)), n - 1)
    chain = np.arange(0, n - 1, 7)
    return psc.HostGraph.from_edges(n, np.concatenate([src, chain]),
                                    np.concatenate([dst, chain + 1]))


GRAPHS = {
    "path": lambda: psc.HostGraph.from_edges(3001, np.arange(3000), np.arange(1, 3001)),
    "grid_narrow": lambda: psc.HostGraph.grid(3, 4001, 0.9, seed=5),
    "grid": lambda: psc.HostGraph.grid(173, 211, 0.6, seed=6),
    "front_8191": lambda: _tree([8191, 3]),
    "front_8192_edges_65536": lambda: _tree([8192, 8]),
    "front_8193": lambda: _tree([8193, 2]),
    "edges_65535": lambda: _tree([257, 255]),
    "edges_65537": lambda: _tree([65537, 1]),
    "hub_then_fan": lambda: _tree([33, 9, 70, 3]),
    # eight lanes per entry up to degree 24, the balanced expansion above it
    "fan_8": lambda: _tree([8] * 5),
    "fan_9": lambda: _tree([9] * 4),
    "degrees_0_to_8": lambda: _band(8),
    "degrees_0_to_12": lambda: _band(12),
    "degrees_0_to_24": lambda: _band(24),
    "degrees_0_to_27": lambda: _band(27),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_levels_match_definition(name):
    g = GRAPHS[name]()
    want, levels = _bfs(g, 0)
    lib = psc.cuda()
    with psc.DeviceGraph(g) as dg:
        assert np.array_equal(dg.bfs(0), want)
        assert dg.last_rounds == levels
    ptrs = []
    try:
        for a in (g.off, g.E, g.in_off, g.in_E, np.zeros(g.n, np.uint8)):
            p = C.c_void_p()
            _lib.check(lib.psc_device_alloc(max(a.nbytes, 1), C.byref(p)), "psc_device_alloc")
            ptrs.append(p.value)
            _lib.check(lib.psc_copy(p, a.ctypes.data, a.nbytes), "psc_copy")
        r = C.c_uint32()
        _lib.check(lib.psc_reach_noalloc(*ptrs[:4], g.n, g.m, 0, 0, ptrs[4], None, C.byref(r)),
                   "psc_reach_noalloc")
        out = np.empty(g.n, np.uint8)
        _lib.check(lib.psc_copy(out.ctypes.data, ptrs[4], g.n), "psc_copy")
        assert np.array_equal(out.astype(bool), want != 0xFFFFFFFF)
        assert r.value == levels
    finally:
        for p in ptrs:
            lib.psc_device_free(p)
