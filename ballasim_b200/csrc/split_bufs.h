// The split engine's device buffers: its scratch (the pixel and quick records, the blob boxes), the posted-pixel list (a
// record for every slot of the tiles) and the list's counts per window. Host code over any buffer type with a pointer p, a
// capacity cap, ensure(n) (which frees the old allocation before it makes the new one, and throws where that fails) and
// release(), so that the CPU tests run it over buffers that fail.
#pragma once

#include <cstddef>

namespace bs {

template <class Scratch, class Rest, class Counts>
struct SplitBufs {
  Scratch scratch;
  Rest rest;
  Counts counts;
  unsigned int capacity = 0;  // the records `rest` has room for: 0 wherever it is not allocated

  // moving(): called before a buffer is replaced, to drop what holds its address (a captured step).
  template <class Moving>
  void ensure(size_t scratch_n, unsigned int slots, size_t record_bytes, size_t windows, Moving moving) {
    const auto grow = [&](auto& buf, size_t n) {
      if (n <= buf.cap && buf.p) return;
      moving();
      buf.ensure(n);
    };
    if (capacity < slots || !rest.p) {
      capacity = 0;
      grow(rest, static_cast<size_t>(slots) * record_bytes);
      capacity = slots;
    }
    grow(scratch, scratch_n);
    grow(counts, windows);
  }
  bool empty() const { return !rest.p && !scratch.p && !counts.p; }
  void release() {
    capacity = 0;
    rest.release();
    scratch.release();
    counts.release();
  }
};

// need(), which allocates; where memory is short (it throws Short) and give_way() could free some, once more.
template <class Short, class Need, class GiveWay>
void with_room(Need need, GiveWay give_way) {
  try {
    need();
    return;
  } catch (const Short&) {
    if (!give_way()) throw;
  }
  need();
}

}  // namespace bs
