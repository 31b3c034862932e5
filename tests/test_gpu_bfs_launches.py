"""Push levels of BFS (csrc/lelist.cu): graphs without vertices for k_bfs_heavy stop launching it
after a few levels, graphs with some late in the search keep it; distances exact."""
import numpy as np
import pytest

import psc
import pyoracle as O

pytestmark = pytest.mark.gpu


def _layers(count, width, deg, hub_at=None):
    r = np.random.default_rng(count)
    v = np.arange(count * width)
    src = np.repeat(v, deg)
    dst = np.minimum((src // width + 1) * width + r.integers(0, width, len(src)), count * width - 1)
    if hub_at is not None:
        u = hub_at * width + 5
        src = np.concatenate([src, np.full(700, u), [(hub_at - 1) * width]])
        dst = np.concatenate([dst, (hub_at + 1) * width + np.arange(700) % width, [u]])
    return psc.HostGraph.from_edges(count * width, src, dst)


@pytest.mark.parametrize("hub_at", [None, 3, 30])
def test_wide_layers(cuda_device, hub_at):
    g = _layers(40, 3000, 60, hub_at)
    with psc.DeviceGraph(g) as dg:
        for _ in range(2):
            for src in (0, 7, 3000):
                assert np.array_equal(dg.bfs(src), O.bfs_seq(g.n, g.off, g.E, src))
