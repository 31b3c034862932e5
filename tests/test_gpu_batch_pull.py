"""Pull rounds over a batch whose members' pivots miss their large components (csrc/reach.cu): the
hubs of such a member are scanned whole, spread over the grid; exact labels, and no slower than the
same members solved alone."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


def test_members_with_missed_components(cuda_device):
    count = 48
    u, vb = psc.batch_workload(count, 1000, 14, 18)
    seeds = 1000 + np.arange(count, dtype=np.uint64)
    with psc.DeviceGraph(u) as dg:
        dg.set_batch(vb)
        for _ in range(2):
            lab = dg.scc_batch(psc.default_params(), seeds)
        batch_ms = dg.stats().total_ms
    alone = 0.0
    for k in range(count):
        g = u.member(vb, k)
        with psc.DeviceGraph(g) as one:
            p = psc.default_params(seed=int(seeds[k]))
            one.scc(p)
            got = one.scc(p)
            alone += one.stats().total_ms
        assert np.array_equal(got, lab[int(vb[k]):int(vb[k + 1])])
        if k < 12:
            assert np.array_equal(O.canon(got), O.canon(O.tarjan(g.n, g.off, g.E)[0]))
    assert batch_ms < alone, (batch_ms, alone)
