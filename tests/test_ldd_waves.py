"""Rounds of the decomposition on adjacency records (ldd_low_round, csrc/cc.cu) come to an end: a
round expands the entries of its first wave whole, whatever comes in behind them (replayed on the CPU
with the constants of csrc/rec_rules.h), and components of graphs with vertices of every degree up to
the records' largest are exact (GPU)."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import psc
import pyoracle as O

CSRC = Path(__file__).resolve().parent.parent / "parallel-strong-connectivity_gb300" / "csrc"
# One warp's queue: an entry is its index among the chunk's vertices (or -1, claimed in this
# round) and the edges that it has left.
PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <utility>
#include "rec_rules.h"
using namespace psc;
int main() {
  long bad = 0;
  for (int trial = 0; trial < 50000; trial++) {
    srand(trial);
    const int chunk = 1 + rand() % 32, kind = rand() % 3;
    const int top = 1 + rand() % (int)kRecMaxDeg;  // the graph's largest degree
    const uint32_t waves = ldd_waves(top);
    std::deque<std::pair<int, int>> q;
    for (int i = 0; i < chunk; i++)
      q.push_back({i, kind == 0 ? top : kind == 1 ? rand() % (top + 1) : rand() % top % 8});
    for (uint32_t wave = 0; !q.empty() && wave < waves; wave++) {
      const int n = (int)q.size() < kLrWave ? (int)q.size() : kLrWave;
      std::deque<std::pair<int, int>> back;
      for (int i = 0; i < n; i++) {
        const auto e = q.front();
        q.pop_front();
        if (e.second > kRecEdges) back.push_back({e.first, e.second - kRecEdges});
      }
      for (int i = rand() % (n * kRecEdges + 1); i > 0 && q.size() < 100; i--)
        q.push_back({-1, rand() % (top + 1)});
      q.insert(q.begin(), back.begin(), back.end());
    }
    for (auto& e : q) bad += e.first >= 0 && e.first < kLrWave;
  }
  printf("%ld\n", bad);
}
'''


def test_first_entries_are_expanded_whole(tmp_path):
    (tmp_path / "w.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(tmp_path / "w.cpp"), "-o",
                    str(tmp_path / "w")], check=True)
    assert subprocess.run([str(tmp_path / "w")], check=True, capture_output=True).stdout == b"0\n"


def _deep(degree, hubs=20, rows=400, cols=700):
    """A grid, so that frontiers stay narrow, on which a few vertices have `degree` neighbours."""
    g = psc.HostGraph.grid(rows, cols, 0.3, seed=degree).symmetrize()
    src, dst = (x.astype(np.int64) for x in g.edge_list())
    near = np.unique(np.linspace(2000, g.n - 2000, hubs).astype(np.int64))
    a, b = [], []
    for h in near:
        have = set(g.E[int(g.off[h]):int(g.off[h + 1])].tolist())
        add = [x for x in range(h - 2 * degree, h + 2 * degree) if x != h and x not in have]
        add = np.random.default_rng(h).permutation(add)[: degree - len(have)]
        a.append(np.full(len(add), h))
        b.append(add)
    out = psc.HostGraph.from_edges(g.n, np.concatenate([src] + a), np.concatenate([dst] + b)).symmetrize()
    assert np.diff(out.off.astype(np.int64)).max() == degree
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("degree", [12, 13, 54, 59, 60, 61, 62, 63, 64, 65])
def test_degrees_up_to_the_records_largest(cuda_device, degree):
    g = _deep(degree)
    comp = O.canon(O.cc(g.n, g.off, g.E))
    with psc.DeviceGraph(g) as dg:
        for beta in (0.2, 0.01):
            assert np.array_equal(O.canon(dg.cc(beta)), comp)
            lab, _ = dg.ldd(beta)
            assert (lab[lab] == lab).all() and (comp[lab] == comp).all()
        assert np.array_equal(dg.reach(5), O.reach_seq(g.n, g.off, g.E, 5))
