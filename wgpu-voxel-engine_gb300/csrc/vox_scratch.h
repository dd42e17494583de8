// vox_scratch.h — growth of the per-chunk scratch of a context's batches (host).
//
// A batch of n chunks takes n slots: the face lists' (list_slot bytes), or where these do not
// fit in memory the persistent launch's (spill_slot bytes, smaller at 64^3 only). The buffer grows
// and never shrinks, to at least `floor` bytes, so that small batches do not grow it in steps.
// A buffer that works is given back only for one that is there, or when nothing smaller would do;
// a size that had no room is not asked for again (every batch would pay for the attempt).
// Plain C++ over an allocator, so that host tests check it against one that runs out of memory.
#pragma once

#include <algorithm>
#include <cstddef>

namespace vox {

struct ScratchBuffer {
  void* data = nullptr;
  size_t bytes = 0;
  size_t no_room = ~(size_t)0;  // list slots of this many bytes did not fit
};

// Makes `b` hold n slots; clears `lists` where only the persistent launch's fit. alloc(bytes, &p) and
// release(p) are the allocator; alloc returns 0, `out_of_memory` or another error, which ends the
// call with nothing given back. Returns 0 or alloc's last error.
template <typename Alloc, typename Release>
int grow_scratch(ScratchBuffer& b, size_t n, size_t list_slot, size_t spill_slot, size_t floor, bool& lists,
                 int out_of_memory, Alloc alloc, Release release) {
  const bool smaller = spill_slot < list_slot;  // there is a choice
  if (lists && smaller && n * list_slot > b.bytes && n * list_slot >= b.no_room) lists = false;
  size_t need = n * (lists ? list_slot : spill_slot);
  if (need <= b.bytes) return 0;
  auto take = [&](size_t bytes) {
    void* p = nullptr;
    const int e = alloc(bytes, &p);
    if (e == 0) {
      if (b.data) release(b.data);
      b.data = p;
      b.bytes = bytes;
    }
    return e;
  };
  int e = take(std::max(need, floor));
  if (e != out_of_memory) return e;
  if (lists && smaller && n * spill_slot <= b.bytes) {  // the buffer at hand serves the other launch
    b.no_room = need;
    lists = false;
    return 0;
  }
  if (b.data) release(b.data);
  b.data = nullptr;
  b.bytes = 0;
  e = take(need);
  if (e == out_of_memory && lists && smaller) {
    b.no_room = need;
    lists = false;
    e = take(n * spill_slot);
  }
  return e;
}

}  // namespace vox
