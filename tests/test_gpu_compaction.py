"""Order-preserving compactions (csrc/scan.cuh) at the edges of words, tiles (2,048 items) and
tile counts: SCC labels, which hold the places of trimmed vertices, against the oracle (exact)."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


@pytest.mark.parametrize("n", [1, 31, 32, 33, 2047, 2048, 2049, 2080, 4095, 4096, 4097, 6175,
                               2048 * 65 - 1, 2048 * 65, 2048 * 1024 + 1])
@pytest.mark.parametrize("degree", [0.4, 2.5])
def test_labels_equal_oracle(n, degree):
    r = np.random.default_rng(n)
    m = int(degree * n)
    g = psc.HostGraph.from_edges(n, r.integers(0, n, m), r.integers(0, n, m))
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):
            got = dg.scc(psc.default_params(seed=9))
            assert np.array_equal(got, O.scc(g.n, g.off, g.E, g.in_off, g.in_E, seed=9))
