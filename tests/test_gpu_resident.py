"""Prefix-doubling batches in one resident launch (k_ms_batches, csrc/multisearch.cu):
raw SCC labels against the oracle (exact) where its windows are selected by one block or
by the grid, where its tables run full and the host takes a batch over, with heavy
pairs, without local searches, and for windows of many graphs."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _hubs(n=30000, hubs=3, seed=9):
    """Cycles through hubs with more than 8192 out-edges, one-way tails behind them."""
    r = np.random.default_rng(seed)
    src = [np.repeat(np.arange(hubs), 12000)]
    dst = [r.integers(hubs, n, hubs * 12000)]
    back = r.integers(hubs, n, 6000)
    src.append(back)
    dst.append(r.integers(hubs, n, 6000))
    src.append(back[:200])
    dst.append(np.arange(200) % hubs)
    return psc.HostGraph.from_edges(n, np.concatenate(src), np.concatenate(dst))


CASES = {
    "one_vertex_windows": (lambda: psc.HostGraph.grid(17, 19, 0.3, seed=3), {"beta": 1.01}),
    "path_tables_full": (lambda: psc.HostGraph.from_edges(6001, np.arange(6000), np.arange(1, 6001)),
                         {"beta": 100.0}),
    "wide_windows": (lambda: psc.HostGraph.rmat(14, 1 << 16, seed=4), {"beta": 9.0}),
    "window_383_to_385": (lambda: psc.HostGraph.knn(3000, 3, seed=5), {"beta": 384.0}),
    "no_local_search": (lambda: psc.HostGraph.knn(9001, 4, seed=6), {"local_scc": 0}),
    "small_tau": (lambda: psc.HostGraph.grid(120, 131, 0.3, seed=7), {"tau": 3}),
    "hubs": (_hubs, {}),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("seed", [1, 12])
def test_resident_batches_equal_oracle(name, seed):
    make, kw = CASES[name]
    g = make()
    with psc.DeviceGraph(g) as dg:
        got = dg.scc(psc.default_params(seed=seed, **kw))
    want = O.scc(g.n, g.off, g.E, g.in_off, g.in_E, seed=seed,
                 **{k: v for k, v in kw.items() if k in ("beta", "tau")})
    assert np.array_equal(got, want)


@pytest.mark.parametrize("beta", [1.5, 40.0])
def test_resident_windows_of_many_graphs(beta):
    members = [psc.HostGraph.grid(3 + k, 40, 0.3, seed=k) for k in range(60)]
    members += [psc.HostGraph.from_edges(1, [], []), psc.HostGraph.rmat(9, 1 << 12, seed=2),
                psc.HostGraph.from_edges(901, np.arange(900), np.arange(1, 901))]
    u, vb = psc.HostGraph.pack(members)
    seeds = np.arange(len(members), dtype=np.uint64) + 3
    with psc.DeviceGraph(u) as dg:
        dg.set_batch(vb)
        got = dg.scc_batch(psc.default_params(beta=beta), seeds)
    for k, g in enumerate(members):
        want = O.scc(g.n, g.off, g.E, g.in_off, g.in_E, seed=int(seeds[k]), beta=beta)
        assert np.array_equal(got[int(vb[k]):int(vb[k + 1])], want)
