"""Multi-search whose tables run full on hubs (csrc/multisearch.cu): a batch of four large graphs
in which the largest one's first pivot lies outside its giant component, so that a prefix-doubling
batch of a few pivots meets it.  Exact labels, and the refills cost no multiple of the solve."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


def test_hubs_meet_small_tables(cuda_device):
    u, vb = psc.batch_workload(4, 1000, 16, 20)
    ms = {}
    with psc.DeviceGraph(u) as dg:
        dg.set_batch(vb)
        for seed in (4, 3):  # 3 is the unlucky one
            p = psc.default_params(seed=seed)
            dg.scc_batch(p)
            lab = dg.scc_batch(p)
            ms[seed] = dg.stats().total_ms
        assert dg.stats().table_grows > 0
    for k in range(4):
        g = u.member(vb, k)
        got = lab[int(vb[k]):int(vb[k + 1])]
        assert np.array_equal(O.canon(got), O.canon(O.tarjan(g.n, g.off, g.E)[0]))
        with psc.DeviceGraph(g) as one:
            assert np.array_equal(one.scc(psc.default_params(seed=3)), got)
    # (every insert into a full table spends the whole probe limit: 40 times the lucky solve when
    # a sub-round goes on with the rest of its work, 3 times now)
    assert ms[3] < 12 * ms[4], ms
