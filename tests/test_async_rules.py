"""Hand-over rules of the searches without rounds (csrc/async_rules.h), replayed on the CPU: no
vertex that a warp took from the slots is given away again while a launch runs, whatever comes back
or is new in a wave and however many warps are idle."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "parallel-strong-connectivity_gb300" / "csrc"
# One warp's ring as a list of marks: 't' taken and not expanded, 'b' came back with targets
# left, 'n' new.  Every wave expands the front; the tail is given to endlessly hungry warps.
PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <deque>
#include "async_rules.h"
using namespace psc;
int main(int argc, char** argv) {
  const bool low = atoi(argv[1]);
  srand(atoi(argv[2]));
  long bad = 0, given = 0;
  for (int trial = 0; trial < 20000; trial++) {
    const uint32_t warps = 1 + rand() % 2000;
    const uint32_t take = async_take(rand() % (1 << 20), warps, low ? kAsyncTakeLow : kAsyncTake);
    if (take < 1 || take > 32) bad++;
    std::deque<char> ring(take, 't');
    for (int wave = 0; wave < 12 && !ring.empty(); wave++) {
      const uint32_t w = low ? kLowWave : (rand() & 1 ? kAsyncFewWave : 32);
      uint32_t n = ring.size() < w ? ring.size() : w, back = 0;
      for (uint32_t i = 0; i < n; i++) {
        ring.pop_front();
        back += low && rand() % 3;
      }
      ring.insert(ring.begin(), back, 'b');
      ring.insert(ring.end(), rand() % (6 * n + 1), 'n');
      const int32_t hungry = rand() % 8 ? 1 << 20 : rand() % 64 - 8;
      for (uint32_t g = async_give(hungry, ring.size()); g > 0; g--, given++) {
        bad += ring.back() != 'n';
        ring.pop_back();
      }
    }
  }
  printf("%ld %ld\n", bad, given);
}
'''


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    d = tmp_path_factory.mktemp("async")
    (d / "replay.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "replay.cpp"), "-o",
                    str(d / "replay")], check=True)
    return d / "replay"


@pytest.mark.parametrize("low", [0, 1])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_taken_vertices_are_not_given_away(replay, low, seed):
    bad, given = map(int, subprocess.run([str(replay), str(low), str(seed)], check=True,
                                         capture_output=True, text=True).stdout.split())
    assert given > 10000 and bad == 0


def test_slots(tmp_path):
    """Room for every frontier that a launch takes, never more than the vertices, and enough
    after a few launches that ran out."""
    (tmp_path / "s.cpp").write_text(r'''
#include <cstdio>
#include "async_rules.h"
using namespace psc;
int main() {
  long bad = 0;
  const uint64_t sizes[] = {1, 7, 262144, 262145, 10000000, 1ull << 24, 3000000000ull, 4294967294ull};
  const uint64_t fronts[] = {0, 1, 9728, 1ull << 20, kAsyncSlots / 4};
  for (uint64_t n : sizes)
    for (uint64_t f : fronts)
      for (uint32_t full = 0; full < 40; full++) {
        if (f > n) continue;
        const uint64_t s = async_slots(n, f, full);
        bad += s < f || s > n || s > kAsyncSlots;
        bad += full > 2 && s != (n < kAsyncSlots ? n : kAsyncSlots);
        bad += full && s < async_slots(n, f, full - 1);
      }
  printf("%ld\n", bad);
}
''')
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(tmp_path / "s.cpp"), "-o",
                    str(tmp_path / "s")], check=True)
    assert subprocess.run([str(tmp_path / "s")], check=True, capture_output=True).stdout == b"0\n"
