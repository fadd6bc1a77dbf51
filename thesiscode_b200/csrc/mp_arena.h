// A context's scratch: one block that grows on demand.  The memory functions are a
// parameter, so that the rules can be checked without a device: Mem has alloc(bytes) (null
// if there is no room), free(p) and room() (bytes that alloc may find).
#pragma once

#include <stddef.h>

namespace mpgpu {

struct Arena {
    void* p = nullptr;
    size_t bytes = 0;
    size_t refused = 0;       // smallest optional size that the device refused (0: none) ...
    size_t refused_room = 0;  // ... and the room it had then
};

// At least `bytes`; what was there is given back first.
template <class Mem>
bool arena_reserve(Arena& a, size_t bytes, Mem& mem) {
    if (bytes <= a.bytes) return true;
    if (a.p) mem.free(a.p);
    a.p = mem.alloc(bytes);
    a.bytes = a.p ? bytes : 0;
    return a.p != nullptr;
}

// At least `bytes`, which the caller can do without, `need` of them not.  A block that
// holds the need is not given back before there is a larger one.  A size that was refused
// is asked for again only once the device has that much room, and more than it had then:
// an allocation that fails waits for the device, and so would one in every call.
template <class Mem>
bool arena_try(Arena& a, size_t need, size_t bytes, Mem& mem) {
    if (bytes <= a.bytes) return true;
    if (a.refused && bytes >= a.refused) {
        const size_t room = mem.room();
        if (room < bytes || room <= a.refused_room) return false;
    }
    const bool beside = a.p && a.bytes >= need;
    if (a.p && !beside) {
        mem.free(a.p);
        a.p = nullptr;
        a.bytes = 0;
    }
    void* p = mem.alloc(bytes);
    if (!p) {
        a.refused = bytes;
        a.refused_room = mem.room();
        return false;
    }
    if (a.p) mem.free(a.p);
    a.p = p;
    a.bytes = bytes;
    a.refused = 0;
    return true;
}

}  // namespace mpgpu
