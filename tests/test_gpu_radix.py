"""Device transpose and symmetrisation (csrc/transpose.cu): exact against the host graph
library at the edges of tiles (4,608 pairs) and digits (2^8, 2^16 ids), with hubs, long runs of
vertices without edges, and more tiles than run at once."""
import numpy as np
import pytest

import psc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _dev(cuda_device):
    return cuda_device


def _csr(n, src, dst):
    """CSR that keeps duplicates and self-loops."""
    order = np.lexsort((dst, src))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(src, minlength=n))
    return off, np.ascontiguousarray(dst[order], dtype=np.uint32)


def _random(n, m, seed, skew=1.0):
    r = np.random.default_rng(seed)
    src = (n * r.random(m) ** skew).astype(np.int64)
    dst = (n * r.random(m) ** skew).astype(np.int64)
    return n, src, dst


CASES = {
    **{f"m_{m}": (lambda m=m: _random(300, m, m)) for m in (1, 31, 383, 385, 3073, 4607, 4608, 4609, 9217)},
    **{f"n_{n}": (lambda n=n: _random(n, 20011, n)) for n in (1, 2, 255, 256, 257, 65535, 65536, 65537)},
    "skewed": lambda: _random(1 << 20, 700_017, 5, skew=6.0),
    "many_tiles": lambda: _random((1 << 21) + 3, 4_000_001, 6),
    "all_to_last": lambda: (200_001, np.arange(50_000) * 4, np.full(50_000, 200_000)),
    "first_only": lambda: (100_000, np.zeros(5000, np.int64), np.zeros(5000, np.int64)),
    "gaps_of_64_65": lambda: (10_000, np.arange(0, 9000, 65), np.arange(0, 9000, 65) // 65 * 64),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_transpose_and_symmetrise(name):
    n, src, dst = CASES[name]()
    off, E = _csr(n, src, dst)
    in_off, in_E = _csr(n, dst, src)
    for _ in range(2):
        with psc.DeviceGraph.directed(off, E) as dg:
            got_off, got_E = dg.transpose()
            assert np.array_equal(got_off, in_off) and np.array_equal(got_E, in_E)
    keep = src != dst
    a, b = np.concatenate([src[keep], dst[keep]]), np.concatenate([dst[keep], src[keep]])
    pairs = np.unique(a.astype(np.uint64) << np.uint64(32) | b.astype(np.uint64))
    s_off, s_E = _csr(n, (pairs >> np.uint64(32)).astype(np.int64), (pairs & np.uint64(0xFFFFFFFF)).astype(np.int64))
    with psc.DeviceGraph.symmetrized(off, E) as dg:
        got_off, got_E = dg.download()
    assert np.array_equal(got_off, s_off) and np.array_equal(got_E, s_E)
