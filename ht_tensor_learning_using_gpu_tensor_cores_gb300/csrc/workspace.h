// The block of device memory a call works in: kept between calls, grown when a
// call needs more.  Some calls want more than they need (`want` bytes with the
// BF16 planes of their operands or the records of a sort, `least` without).  The
// rule for those, apart from the CUDA calls it makes so that it can be tested
// without a device:
//   * what the block holds is used as it is;
//   * a larger block is asked for while the old one is still held, or, where only
//     both together make the room, after giving the old one back;
//   * where the device has no room for `want`, a block of at least `least` bytes is
//     left alone: the call neither waits for the device nor frees and allocates,
//     on this call and on the next ones alike;
//   * an allocation that failed although there seemed to be room is not tried
//     again until the room has grown or the block has been released.
#pragma once
#include <cstddef>

namespace htgb {

struct WorkspaceBlock {
  void *ptr = nullptr;
  size_t bytes = 0;
  size_t refused = 0, refused_room = 0;   // an allocation that failed, and the room there was
};

enum class Granted { want, least, none };

// Memory: bool room(size_t *free_bytes); bool allocate(void **, size_t); bool
// release(void *), which waits for the device first.  optional: false where only
// `least` may be allocated (a stream capture).
template <class Memory>
Granted grant_workspace(WorkspaceBlock &w, size_t want, size_t least, bool optional, Memory &mem) {
  if (w.bytes >= want) return Granted::want;
  auto give_back = [&]() {
    if (!w.ptr) return true;
    if (!mem.release(w.ptr)) return false;
    w.ptr = nullptr;
    w.bytes = 0;
    return true;
  };
  auto fresh = [&](size_t bytes) {   // with no block held
    if (!mem.allocate(&w.ptr, bytes)) {
      w.ptr = nullptr;
      return false;
    }
    w.bytes = bytes;
    return true;
  };
  size_t free_bytes = 0;
  if (want > least && optional && mem.room(&free_bytes)) {
    const size_t room = free_bytes + w.bytes;
    if (room >= want && !(w.refused && want >= w.refused && room <= w.refused_room)) {
      if (free_bytes >= want) {
        void *p = nullptr;
        if (mem.allocate(&p, want)) {
          if (!give_back()) {
            mem.release(p);
            return Granted::none;
          }
          w.ptr = p;
          w.bytes = want;
          return Granted::want;
        }
      } else {
        if (!give_back()) return Granted::none;
        if (fresh(want)) return Granted::want;
      }
      w.refused = want;
      w.refused_room = room;
    }
  }
  if (w.bytes >= least) return want > least ? Granted::least : Granted::want;
  if (!give_back() || !fresh(least)) return Granted::none;
  return want > least ? Granted::least : Granted::want;
}

}  // namespace htgb
