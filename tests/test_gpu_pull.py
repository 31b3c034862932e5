"""Pull rounds of the searches (k_reach_pull, csrc/reach.cu): reach sets (exact) at the edges of
bitmap words and warp steps, with dead vertices, in-lists around the lone scan's 64 edges and far
above it, and heavy vertices at the limit of a sparse round's direct expansion."""
import ctypes as C

import numpy as np
import pytest

import psc
import pyoracle as O
from psc import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _graph(n, hub_deg, seed):
    """A path of 24 (deeper than the resident rounds), a hub, and a body of n vertices: a
    quarter without in-edges, the rest random, some with 63 to 700 in-edges that come from
    vertices without in-edges but for the last one."""
    r = np.random.default_rng(seed)
    first = 25
    perm = first + r.permutation(n)
    dead, body = perm[: n // 4], perm[n // 4:]
    src = [np.arange(24), np.full(hub_deg, 24)]
    dst = [np.arange(1, 25), body[r.integers(0, len(body), hub_deg)]]
    k = 6 * n
    src.append(perm[r.integers(0, n, k)])
    dst.append(body[(len(body) * r.random(k) ** 2).astype(np.int64)])
    for i, d in enumerate((63, 64, 65, 128, 129, 320, 700)):
        t = body[-1 - i]
        d = min(d, len(dead))
        src += [dead[:d], [body[i]]]
        dst += [np.full(d, t), [t]]
    return psc.HostGraph.from_edges(first + n, np.concatenate(src), np.concatenate(dst))


@pytest.mark.parametrize("n,hub", [(2015, 900), (4071, 1023), (4072, 1024), (4103, 1025),
                                   (30_011, 8192), (30_020, 8193), (262_119, 20_000),
                                   (1_500_007, 9000)])
def test_pull_matches_definition(n, hub):
    g = _graph(n, hub, n)
    want = O.reach_seq(g.n, g.off, g.E, 0)
    back = O.reach_seq(g.n, g.in_off, g.in_E, g.n - 1)
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):
            assert np.array_equal(dg.reach(0), want)
            assert np.array_equal(dg.reach(g.n - 1, backward=True), back)
    lib, ptrs = psc.cuda(), []
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
        assert np.array_equal(out != 0, want != 0)
    finally:
        for p in ptrs:
            lib.psc_device_free(p)


def test_sparse_round_hands_large_vertices_to_the_grid():
    """Past the resident rounds and a stopped resident search (a vertex of 8,193 out-edges), a
    round of three vertices around the direct limit of 2,048 out-edges, without pulls."""
    hub, fans, side = 8193, (2048, 2049, 5000), 1500
    src, dst = [np.arange(24), np.full(hub, 24)], [np.arange(1, 25), 25 + np.arange(hub)]
    n = 25 + hub
    top = n + np.arange(3)
    src.append(np.full(3, 25))
    dst.append(top)
    n += 3
    for t, d in zip(top, fans):
        src += [np.full(d, t), [n + d - 1]]
        dst += [n + np.arange(d), [n + d]]
        n += d + 1
    e = np.arange(1_500_000)
    src.append(n + e % side)
    dst.append(n + e // side)
    g = psc.HostGraph.from_edges(n + side, np.concatenate(src), np.concatenate(dst))
    with psc.DeviceGraph(g) as dg:
        for back, off, E, s in ((False, g.off, g.E, 0), (True, g.in_off, g.in_E, n - 1)):
            assert np.array_equal(dg.reach(s, backward=back), O.reach_seq(g.n, off, E, s))
