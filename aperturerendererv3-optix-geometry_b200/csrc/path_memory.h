// path_memory.h -- the blocks of device memory that hold path state, kept
// between calls and shared by the scenes of a device.  Memory is the allocator:
// static void* alloc(size_t), NULL when there is none, and static void free(void*),
// both for the current device.
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace ar {

// One block per device, lent to a call for its duration, so scenes that render in
// turn share it.  A call that finds it lent out allocates a block of its own; of
// the blocks that come back one is kept, the larger, and it is freed with the
// device's last scene.  (A stream-ordered memory pool did the same but took 25 ms
// longer to grow to 3.6 GB than cudaMalloc.)
template <class Memory>
class PathMemory {
public:
    static void add_scene(int device)
    {
        std::lock_guard<std::mutex> g(lock());
        ++entries()[device].scenes;
    }
    static void remove_scene(int device)
    {
        std::lock_guard<std::mutex> g(lock());
        Entry& e = entries()[device];
        if (--e.scenes > 0) return;
        if (e.mem) Memory::free(e.mem);
        e.mem = nullptr;
        e.bytes = 0;
    }
    // at least `bytes` (set to the block's size) on the current device, or NULL
    static char* take(int device, size_t& bytes)
    {
        {
            std::lock_guard<std::mutex> g(lock());
            Entry& e = entries()[device];
            if (e.mem && e.bytes >= bytes) {
                char* p = e.mem;
                bytes = e.bytes;
                e.mem = nullptr;
                return p;
            }
            if (e.mem) Memory::free(e.mem);   // too small: its successor comes back instead
            e.mem = nullptr;
        }
        return static_cast<char*>(Memory::alloc(bytes));
    }
    static void give(int device, char* p, size_t bytes)   // idle: its last kernel has finished
    {
        std::lock_guard<std::mutex> g(lock());
        Entry& e = entries()[device];
        if (e.scenes > 0 && (!e.mem || e.bytes < bytes)) {
            std::swap(p, e.mem);
            e.bytes = bytes;
        }
        if (p) Memory::free(p);
    }
private:
    struct Entry { char* mem = nullptr; size_t bytes = 0; int scenes = 0; };
    // never destroyed: scenes owned by objects with static storage are released
    // during process exit, after the destructors of what was first used later
    static std::mutex& lock() { static std::mutex* m = new std::mutex; return *m; }
    static std::map<int, Entry>& entries() { static auto* e = new std::map<int, Entry>; return *e; }
};

}  // namespace ar
