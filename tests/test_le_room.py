"""Room of the LE-list entry buffers (csrc/le_room.h): the bound that k_le_batches gets is
never above what the shortest of its three arrays holds (CPU), and lists that fill the buffers on a
fresh handle equal the oracle and leave their neighbours alone (GPU)."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import psc
import pyoracle as O

CSRC = Path(__file__).resolve().parent.parent / "parallel-strong-connectivity_gb300" / "csrc"
PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include "le_room.h"
using namespace psc;
// bytes of the three buffers -> the highest entry that a launch may write must lie in each
int main(int argc, char** argv) {
  for (int i = 1; i + 4 < argc; i += 5) {
    const uint64_t kb = strtoull(argv[i], 0, 10), db = strtoull(argv[i + 1], 0, 10);
    const uint64_t len = strtoull(argv[i + 2], 0, 10), cap = strtoull(argv[i + 3], 0, 10);
    uint64_t sb = strtoull(argv[i + 4], 0, 10);
    if (sb == 0) sb = 4 * le_room(kb, db, SIZE_MAX) + 16;  // as lelist.cu asks for it
    const uint64_t room = le_room(kb, db, sb);
    printf("%llu %llu\n", (unsigned long long)room,
           (unsigned long long)le_entries_wanted(len, cap));
  }
}
'''


def _run(tmp_path, rows):
    src, exe = tmp_path / "room.cpp", tmp_path / "room"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)] + [str(x) for r in rows for x in r], check=True,
                         capture_output=True, text=True).stdout.split()
    return [(int(out[2 * i]), int(out[2 * i + 1])) for i in range(len(rows))]


def test_room_is_what_every_buffer_holds(tmp_path):
    rows = []
    for n in (2, 1500, 4003, 30000, 1 << 20, 1 << 23):
        cap = min(1 << 24, max(8192, 1 << (4 * n - 1).bit_length()))
        for length in (1, n, 9 * n):
            want = max(4 * n, 1024, length + 2 * cap)
            # keys and distances as le_list_reserve sizes them, slots for them or too short
            for sb in (0, want // 2 * 4, 4):
                rows.append((8 * want + 16, 4 * want + 16, length, cap, sb))
    for (kb, db, length, cap, sb), (room, wanted) in zip(rows, _run(tmp_path, rows)):
        assert 8 * room <= kb and 4 * room <= db
        assert wanted == length + 2 * cap
        if sb:
            assert 4 * room <= sb
        else:  # sized for them: no entry less than keys and distances have
            assert room >= wanted


GRAPHS = {
    "grid": lambda: psc.HostGraph.grid(150, 200, 0.3, seed=2).symmetrize(),
    "knn": lambda: psc.HostGraph.knn(30000, 5, seed=2).symmetrize(),
    "path": lambda: psc.HostGraph.from_edges(1500, np.arange(1499), np.arange(1, 1500)).symmetrize(),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_fresh_handle_list_and_neighbours(cuda_device, name):
    g = GRAPHS[name]()
    perm = psc.random_permutation(g.n, 11)
    want = np.asarray(O.lelist_seq(g.n, g.off, g.E, perm)).reshape(-1, 3)
    with psc.DeviceGraph(g) as other, psc.DeviceGraph(g) as dg:
        assert np.array_equal(dg.lelist(perm), want)  # the first call of the handle
        for d in (other, dg):
            off, E = d.download()
            assert np.array_equal(off, g.off) and np.array_equal(E, g.E)
            assert np.array_equal(d.bfs(g.n // 2), O.bfs_seq(g.n, g.off, g.E, g.n // 2))
