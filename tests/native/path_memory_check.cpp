// Host checks of the kept blocks of path state (csrc/path_memory.h) with a fake
// allocator, run by tests/test_cpu_path_memory.py under AddressSanitizer: one
// check per name, "OK" and exit code 0 when it holds.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "../../aperturerendererv3-optix-geometry_b200/csrc/path_memory.h"

struct Fake {
    static constexpr size_t kKeep = 500;
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

// Calls in turn share one block; it grows with the largest.
int in_turn()
{
    Blocks::add_scene(0);
    Blocks::add_scene(0);
    for (size_t need : {100, 60, 100, 200, 30, 200}) {
        size_t n = need;
        char* p = Blocks::take(0, n);
        CHECK(p && n >= need);
        CHECK(Fake::live().size() == 1);
        Blocks::give(0, p, n);
    }
    CHECK(Fake::allocs == 2 && Fake::used() == 200);
    Blocks::remove_scene(0);
    CHECK(Fake::live().size() == 1);
    Blocks::remove_scene(0);
    CHECK(Fake::live().empty());
    return std::printf("OK\n"), 0;
}

// Calls at once keep a block each, of their own size, and allocate no more.
int at_once()
{
    for (int k = 0; k < 2; ++k) Blocks::add_scene(3);
    for (int round = 0; round < 4; ++round) {
        size_t a = 100, b = 40;
        char *p = Blocks::take(3, a), *q = Blocks::take(3, b);
        CHECK(p && q && p != q && a == 100 && b == 40);
        Blocks::give(3, q, b);
        Blocks::give(3, p, a);
        CHECK(Fake::allocs == 2 && Fake::live().size() == 2);
    }
    // a third at once: only as many blocks as scenes are kept
    size_t n[3] = {100, 40, 30};
    char* r[3];
    for (int k = 0; k < 3; ++k) r[k] = Blocks::take(3, n[k]);
    for (int k = 0; k < 3; ++k) Blocks::give(3, r[k], n[k]);
    CHECK(Fake::live().size() == 2);
    size_t big = 501;   // above kKeep
    char* p = Blocks::take(3, big);
    CHECK(p);
    Blocks::give(3, p, big);
    CHECK(Fake::used() <= 500);
    for (int k = 0; k < 2; ++k) Blocks::remove_scene(3);
    CHECK(Fake::live().empty());
    return std::printf("OK\n"), 0;
}

// Where memory is short the idle blocks give way.
int pressure()
{
    for (int k = 0; k < 3; ++k) Blocks::add_scene(0);
    size_t n[3] = {100, 120, 130};
    char* p[3];
    for (int k = 0; k < 3; ++k) p[k] = Blocks::take(0, n[k]);
    for (int k = 0; k < 3; ++k) Blocks::give(0, p[k], n[k]);
    CHECK(Fake::used() == 350);
    Fake::room = 400;
    size_t big = 390;   // fits only without all three
    char* q = Blocks::take(0, big);
    CHECK(q && Fake::used() == 390);
    size_t more = 20;   // no room, nothing idle
    CHECK(!Blocks::take(0, more));
    Blocks::give(0, q, big);
    CHECK(!Blocks::trim(1) && Fake::used() == 390);
    CHECK(Blocks::trim(0) && Fake::live().empty() && !Blocks::trim(0));
    for (int k = 0; k < 3; ++k) Blocks::remove_scene(0);
    return std::printf("OK\n"), 0;
}

int main(int argc, char** argv)
{
    const char* what = argc > 1 ? argv[1] : "";
    if (!std::strcmp(what, "exit")) return at_exit();
    if (!std::strcmp(what, "in_turn")) return in_turn();
    if (!std::strcmp(what, "at_once")) return at_once();
    if (!std::strcmp(what, "pressure")) return pressure();
    return 2;
}
