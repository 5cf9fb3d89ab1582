// Host checks of the kept blocks of path state (csrc/path_memory.h) with a fake
// allocator, run by tests/test_cpu_path_memory.py under AddressSanitizer: one
// check per name, "OK" and exit code 0 when it holds.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "../../aperturerendererv3-optix-geometry_b200/csrc/path_memory.h"

struct Fake {
    static std::map<void*, size_t>& live() { static auto* m = new std::map<void*, size_t>; return *m; }
    static size_t room;   // bytes that may be live at once
    static int allocs;
    static size_t used()
    {
        size_t n = 0;
        for (auto& b : live()) n += b.second;
        return n;
    }
    static void* alloc(size_t bytes)
    {
        if (used() + bytes > room) return nullptr;
        ++allocs;
        void* p = std::malloc(1);   // its address is all that is used
        live()[p] = bytes;
        return p;
    }
    static void free(void* p)
    {
        if (live().erase(p) != 1) { std::printf("freed twice\n"); std::_Exit(1); }
        std::free(p);
    }
};
size_t Fake::room = 1000;
int Fake::allocs = 0;
using Blocks = ar::PathMemory<Fake>;

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

// A scene owned by an object with static storage: made in main, released by a
// destructor that runs after those of everything first used since.
struct Owner {
    bool scene = false;
    ~Owner()
    {
        if (!scene) return;
        Blocks::remove_scene(0);
        if (!Fake::live().empty()) { std::printf("block left behind\n"); std::_Exit(1); }
        std::printf("OK\n");
    }
} owner;

int at_exit()
{
    Blocks::add_scene(0);
    owner.scene = true;
    size_t n = 100;
    char* p = Blocks::take(0, n);
    CHECK(p && n == 100);
    Blocks::give(0, p, n);
    return 0;   // "OK" comes from the owner's destructor
}

int main(int argc, char** argv)
{
    const char* what = argc > 1 ? argv[1] : "";
    if (!std::strcmp(what, "exit")) return at_exit();
    return 2;
}
