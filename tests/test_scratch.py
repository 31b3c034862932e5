"""Growth of scratch buffers (csrc/scratch.h) against a counting allocator, on the CPU: an allocation
that fails gives back what the handle can do without, once, and is tried again; contents are kept or
dropped as asked, and nothing is freed twice or lost, also when it fails for good."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "parallel-strong-connectivity_gb300" / "csrc"
PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include "scratch.h"
using namespace psc;
struct Fake {
  size_t room;
  DevBuf* extra = nullptr;  // what can be given back
  std::map<void*, size_t> live;
  int spared = 0, bad = 0;
  int alloc(void** p, size_t n) {
    if (n > room) return 2;
    room -= n;
    *p = malloc(n);
    live[*p] = n;
    return 0;
  }
  int free(void* p) {
    if (!live.count(p)) { bad++; return 1; }
    room += live[p];
    live.erase(p);
    ::free(p);
    return 0;
  }
  int copy(void* to, const void* from, size_t n) {
    if (live[to] < n || live[const_cast<void*>(from)] < n) { bad++; return 1; }
    memcpy(to, from, n);
    return 0;
  }
  bool spare(int e) {
    spared++;
    if (e != 2 || !extra || !extra->p) return false;
    free(extra->p);
    *extra = DevBuf{};
    return true;
  }
};
#define CHECK(c) do { if (!(c)) { printf("line %d\n", __LINE__); return 1; } } while (0)
int main() {
  Fake f{1000};
  DevBuf a, rec;
  CHECK(scratch_grow(f, rec, 600, 0) == 0 && f.room == 400);
  f.extra = &rec;
  CHECK(scratch_grow(f, a, 300, 0) == 0 && rec.p && f.spared == 0);
  memset(a.p, 7, 300);
  void* old = a.p;
  CHECK(scratch_grow(f, a, 200, 0) == 0 && a.p == old);          // large enough already
  CHECK(scratch_grow(f, a, 500, 300) == 0);                       // needs the extra's room
  CHECK(!rec.p && !rec.bytes && f.spared == 1 && a.bytes == 500 && f.room == 500);
  for (int i = 0; i < 300; i++) CHECK(((char*)a.p)[i] == 7);
  CHECK(scratch_grow(f, a, 600, 500) == 2 && a.bytes == 500 && a.p);  // nothing left to give back
  CHECK(f.spared == 2 && ((char*)a.p)[299] == 7);
  CHECK(scratch_grow(f, a, 900, 0) == 0 && a.bytes == 900 && f.room == 100);  // the old one goes first
  CHECK(scratch_grow(f, a, 1100, 0) == 2 && !a.p && !a.bytes && f.room == 1000);
  CHECK(scratch_grow(f, a, 50, 0) == 0 && f.live.size() == 1 && f.bad == 0);
  CHECK(scratch_grow(f, rec, 940, 0) == 0);
  Fake* g = &f;
  g->extra = nullptr;                                             // (growing the extra itself)
  CHECK(scratch_grow(f, rec, 960, 0) == 2 && !rec.p && f.room == 950 && f.bad == 0);
  puts("ok");
}
'''


def test_growth(tmp_path):
    (tmp_path / "s.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(tmp_path / "s.cpp"),
                    "-o", str(tmp_path / "s")], check=True)
    r = subprocess.run([str(tmp_path / "s")], capture_output=True, text=True)
    assert r.stdout == "ok\n", r.stdout
