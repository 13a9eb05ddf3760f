// When the room of a delta arena is read back from the device (graph.cu): host
// arithmetic only.
#pragma once

#include <cstdint>

namespace vxh {

// A bound of arena_top for which room has been made when nothing else is
// inserted: the rows' next blocks (see reserve_arena).
inline uint64_t arena_bound_from(uint64_t top, uint64_t live) { return top + 4 * live; }

// Whether a batch that brings the bound to `need` asks for a readback: once the
// bound has used up five eighths of the room that the last readback (`read`, 0
// before the first) left, so that a readback gives back at least half of that
// room.  With half of the arena as a fixed mark, a graph whose rows hold more
// than that asked with every batch, a copy and an event each.
inline bool arena_ask_due(uint64_t need, uint64_t read, uint64_t cap) {
  return need > read + (cap > read ? (cap - read) / 8 * 5 : 0);
}

}  // namespace vxh
