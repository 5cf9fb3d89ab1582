// Host check of the jumps of the per-pixel generator initialisation
// (csrc/xorwow_jump.h), run by tests/test_cpu_rng_init.py.  For images of every
// accepted shape family (1 to 4096 pixels wide or high, up to kMaxImagePixels)
// the group index must fit in the tables' bits, and for the last pixel of the
// largest ones the walk along those tables must give the state that plain jumps
// along the bits of the reference pixel index give.  Prints "OK" and exits 0, or
// the first failure and exits 1.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../../aperturerendererv3-optix-geometry_b200/csrc/xorwow_jump.h"

using ar::Bits160;

static Bits160 jump(const std::vector<uint32_t>& tables, int t, const Bits160& v)
{
    const std::vector<uint32_t> one(tables.begin() + static_cast<int64_t>(t) * ar::kJumpWords,
                                    tables.begin() + static_cast<int64_t>(t + 1) * ar::kJumpWords);
    return ar::xorwow_jump_apply(one, v);
}

static int64_t blocks(int64_t w, int64_t h) { return ((w + 7) / 8) * ((h + 3) / 4); }

int main()
{
    const int64_t most = int64_t(1) << 28;   // pixels of the largest image a camera may ask for
    for (int64_t side = 1; side <= 4096; ++side)
        for (int turn = 0; turn < 2; ++turn) {
            const int64_t w = turn ? most / side : side, h = turn ? side : most / side;
            const int64_t last = (blocks(w, h) + 7) / 8 - 1;
            if (last >> ar::kInitGroupBits) {
                std::printf("%lld x %lld: group %lld needs more than %d bits\n", static_cast<long long>(w),
                            static_cast<long long>(h), static_cast<long long>(last), ar::kInitGroupBits);
                return 1;
            }
        }
    const std::vector<uint32_t> tables = ar::xorwow_init_tables();
    if (tables.size() != static_cast<size_t>(ar::kInitTables) * ar::kJumpWords) { std::printf("table count\n"); return 1; }
    std::vector<int> e;
    for (int k = 0; k < 32; ++k) e.push_back(67 + k);
    const std::vector<uint32_t> plain = ar::xorwow_jump_tables(e);
    const Bits160 seed = {{0x12345678u, 0x9abcdef0u, 0x0badf00du, 0xdeadbeefu, 0x13579bdfu}};
    const int64_t shapes[][2] = {{1, most}, {1, (most >> 1) + 4}, {1, 1}, {7, most / 7}, {9, most / 9}, {most, 1}, {16384, 16384}};
    for (const auto& s : shapes) {
        const int64_t w = s[0], h = s[1], grid_x = (w + 7) / 8, i = w - 1, j = h - 1;
        const int64_t b = (i >> 3) + (j >> 2) * grid_x;   // 8x4 block, then its group of 8
        const uint64_t index = static_cast<uint64_t>(32 * b + (j & 3) * 8 + (i & 7));
        Bits160 want = seed;
        for (int k = 0; k < 32; ++k)
            if ((index >> k) & 1) want = jump(plain, k, want);
        Bits160 got = seed;
        for (int k = 0; k < ar::kInitGroupBits; ++k)
            if (((b >> 3) >> k) & 1) got = jump(tables, ar::kInitFrameBits + ar::kInitLaneTables + k, got);
        const int lane = static_cast<int>((j & 3) + 4 * (b & 7));
        for (int k = 0; k < 5; ++k)
            if ((lane >> k) & 1) got = jump(tables, ar::kInitFrameBits + 1 + k, got);
        for (int x = 0; x < (i & 7); ++x) got = jump(tables, ar::kInitFrameBits, got);
        for (int k = 0; k < 5; ++k)
            if (got.w[k] != want.w[k]) {
                std::printf("%lld x %lld: state of the last pixel\n", static_cast<long long>(w), static_cast<long long>(h));
                return 1;
            }
    }
    std::printf("OK\n");
    return 0;
}
