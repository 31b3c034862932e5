// Growth of a handle's scratch buffers.  Some of what a handle keeps is only there to be
// faster (adjacency records: 64 bytes per vertex of a directed graph), so an allocation that
// fails gives that back and tries once more before the call fails.
#pragma once
#include <stddef.h>

namespace psc {

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

// Makes d hold at least `bytes`; keep: its first bytes stay (and the old buffer until they are
// copied), 0: the contents go, and the old buffer before the new one comes.  Ops: alloc(void**, size),
// free(void*), copy(to, from, size) return 0 or an error, spare(error) releases what the handle
// can do without and says whether that was worth another try.  After an error d holds what
// it held (keep) or nothing.
template <class Ops>
int scratch_grow(Ops& ops, DevBuf& d, size_t bytes, size_t keep) {
  if (d.bytes >= bytes) return 0;
  int e = 0;
  if (!keep && d.p) {
    e = ops.free(d.p);
    d = DevBuf{};
    if (e) return e;
  }
  void* np = nullptr;
  e = ops.alloc(&np, bytes);
  if (e && ops.spare(e)) e = ops.alloc(&np, bytes);
  if (e) return e;
  if (d.p) {
    e = ops.copy(np, d.p, keep < d.bytes ? keep : d.bytes);
    if (!e) e = ops.free(d.p);
  }
  d.p = np;
  d.bytes = bytes;
  return e;
}

}  // namespace psc
