// path_memory.h -- the blocks of device memory that hold path state, kept
// between calls and shared by the scenes of a device.  Memory is the allocator:
// static void* alloc(size_t), NULL when there is none, static void free(void*),
// both for the current device, and kKeep, the size of the largest block kept.
#pragma once

#include <cstddef>
#include <iterator>
#include <map>
#include <mutex>

namespace ar {

// A block is lent to a call for its duration, so scenes that render in turn share
// one.  A call that finds none idle that is large enough allocates; the largest
// idle block then gives way, as the new one will come back in its place.  So a
// device holds as many blocks as calls have run on it at once, and no more than
// it has scenes: with one block for all, two threads that rendered at the same
// time allocated and freed 3.6 GB on every call.  Blocks above Memory::kKeep bytes
// are not kept, an allocation that finds no room has the idle ones freed and tries
// again (trim), and the last scene of the device frees them all.  (A
// stream-ordered memory pool did the same but took 25 ms longer to grow to 3.6 GB
// than cudaMalloc.)
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
        std::multimap<size_t, void*> gone;
        {
            std::lock_guard<std::mutex> g(lock());
            Entry& e = entries()[device];
            if (--e.scenes > 0) return;
            gone.swap(e.idle);
        }
        for (auto& b : gone) Memory::free(b.second);
    }
    // at least `bytes` (set to the block's size) on the current device, or NULL
    static char* take(int device, size_t& bytes)
    {
        void* gone = nullptr;
        {
            std::lock_guard<std::mutex> g(lock());
            auto& idle = entries()[device].idle;
            auto fit = idle.lower_bound(bytes);
            if (fit != idle.end()) {
                char* p = static_cast<char*>(fit->second);
                bytes = fit->first;
                idle.erase(fit);
                return p;
            }
            if (!idle.empty()) {
                auto last = std::prev(idle.end());
                gone = last->second;
                idle.erase(last);
            }
        }
        if (gone) Memory::free(gone);
        void* p = Memory::alloc(bytes);
        if (!p && trim(device)) p = Memory::alloc(bytes);
        return static_cast<char*>(p);
    }
    // Frees the idle blocks, for an allocation that found no room; false if there were none.
    static bool trim(int device)
    {
        std::multimap<size_t, void*> gone;
        {
            std::lock_guard<std::mutex> g(lock());
            gone.swap(entries()[device].idle);
        }
        for (auto& b : gone) Memory::free(b.second);
        return !gone.empty();
    }
    static void give(int device, char* p, size_t bytes)   // idle: its last kernel has finished
    {
        {
            std::lock_guard<std::mutex> g(lock());
            Entry& e = entries()[device];
            if (bytes <= Memory::kKeep && static_cast<int>(e.idle.size()) < e.scenes) {
                e.idle.emplace(bytes, p);
                return;
            }
        }
        Memory::free(p);
    }
private:
    struct Entry { std::multimap<size_t, void*> idle; int scenes = 0; };   // blocks by size
    // never destroyed: scenes owned by objects with static storage are released
    // during process exit, after the destructors of what was first used later
    static std::mutex& lock() { static std::mutex* m = new std::mutex; return *m; }
    static std::map<int, Entry>& entries() { static auto* e = new std::map<int, Entry>; return *e; }
};

}  // namespace ar
