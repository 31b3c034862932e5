"""Searches of a few vertices (psc_reach with local searches, csrc/reach.cu) on graphs of low
degree: exact sets, and no slower than a call whose rounds run in one resident launch."""
import time

import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


def test_few_vertices(cuda_device):
    k, length = 40_000, 5
    v = np.arange(k * length)
    g = psc.HostGraph.from_edges(k * length, v, v // length * length + (v % length + 1) % length)
    ms = {}
    with psc.DeviceGraph(g) as dg:
        for src in (0, 7, g.n - 1):
            for local in (True, False):
                assert np.array_equal(dg.reach(src, local=local), O.reach_seq(g.n, g.off, g.E, src))
        for local in (True, False):
            t = []
            for _ in range(60):
                t0 = time.perf_counter()
                dg.reach(11, local=local)
                t.append(1e3 * (time.perf_counter() - t0))
            ms[local] = float(np.median(t))
    # (idle warps that saw the end at their 16th poll, and seven launches and copies: 0.97 times)
    assert ms[True] < 0.9 * ms[False], ms


def test_path_and_sinks(cuda_device):
    """One warp at work while all others wait for its end, and searches that end at once."""
    n = 30_001
    g = psc.HostGraph.from_edges(n, np.arange(n - 1), np.arange(1, n))
    with psc.DeviceGraph(g) as dg:
        for src in (0, n - 1, n - 2, n // 2):
            for backward in (False, True):
                off, E = (g.in_off, g.in_E) if backward else (g.off, g.E)
                assert np.array_equal(dg.reach(src, backward=backward), O.reach_seq(n, off, E, src))
        for seed in (1, 2):
            assert np.array_equal(dg.scc(psc.default_params(seed=seed)),
                                  O.scc(n, g.off, g.E, g.in_off, g.in_E, seed=seed))
