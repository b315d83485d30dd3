// Host check of csrc/net_buffers.h with a counting allocator in the device's
// place: a network that goes from one grid to another holds, in every buffer
// of its sparse plan, at least what the plan's kernels write for the new grid
// (counted here from the kernels' own indices, voxel by voxel), also where
// the grids have equal volume; a set of buffers is whole or empty after a
// failed allocation, and a network's layers are then no grid's, so that the
// next call takes them again instead of using what is missing; OnError runs
// on an exception alone.  Built and run by tests/test_cpu_net_buffers.py.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <new>

#include "net_buffers.h"

using namespace lhi;

static int failures = 0;
static void check(bool ok, const char* what, int a, int b, int c) {
    if (!ok && failures++ < 20) std::printf("FAIL %s (%d, %d, %d)\n", what, a, b, c);
}

struct Mem {
    static std::map<void*, size_t> live;
    static int takes, fail_at;  // fail_at: the take that fails (-1: none)
    static void* take(size_t n) {
        if (takes++ == fail_at) throw std::bad_alloc();
        void* p = std::malloc(1);
        live[p] = n;
        return p;
    }
    static void give(void* p) {
        live.erase(p);
        std::free(p);
    }
};
std::map<void*, size_t> Mem::live;
int Mem::takes = 0, Mem::fail_at = -1;

// one past the largest tile index that a level's voxels set
static size_t tiles_written(const int* d) {
    size_t n = 0;
    for (int x = 0; x < d[0]; ++x)
        for (int y = 0; y < d[1]; ++y)
            for (int z = 0; z < d[2]; ++z)
                n = std::max(n, (size_t(x) * size_t((d[1] + 15) / 16) + size_t(y >> 4)) * size_t((d[2] + 7) / 8) +
                                    size_t(z >> 3) + 1);
    return n;
}

static void check_plan(const BufferSet<Mem>& s, const int* dims) {
    const int lvl_mask[7] = {0, 0, 1, 1, 2, 2, 0}, lvl_list[11] = {0, 1, 2, 1, 0, 0, 0, 1, 2, 1, 0};
    size_t vox[3], tiles[3];
    for (int l = 0; l < 3; ++l) {
        const int d[3] = {dims[0] >> l, dims[1] >> l, dims[2] >> l};
        vox[l] = size_t(d[0]) * size_t(d[1]) * size_t(d[2]);
        tiles[l] = tiles_written(d);
    }
    check(s.size() == 7 + 3 + 11 + 1, "buffers of a plan", dims[0], dims[1], dims[2]);
    auto held = [&](size_t i) { return Mem::live.at(s.at<void>(i)); };
    for (size_t i = 0; i < 7; ++i) check(held(i) >= vox[lvl_mask[i]], "mask", dims[0], dims[1], dims[2]);
    for (size_t i = 0; i < 3; ++i) check(held(7 + i) >= tiles[i], "tile flags", dims[0], dims[1], dims[2]);
    for (size_t i = 0; i < 11; ++i) check(held(10 + i) >= 4 * tiles[lvl_list[i]], "tile list", dims[0], dims[1], dims[2]);
    check(held(21) >= 4 * 11, "list counts", dims[0], dims[1], dims[2]);
}

int main() {
    // one network over grids of equal volume in every order, and others between
    const int grids[][3] = {{17, 16, 16}, {16, 17, 16}, {16, 16, 17}, {64, 64, 64}, {256, 16, 64}, {4096, 8, 8},
                            {8, 4096, 8},  {8, 8, 4096}, {129, 128, 4}, {128, 129, 4}, {4, 128, 129}, {12, 10, 9},
                            {9, 10, 12},   {5, 4, 4},    {4, 5, 4},     {4, 4, 5}};
    const int n = int(sizeof(grids) / sizeof(grids[0]));
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) {
            BufferSet<Mem> s;
            s.fit(plan_bytes(net_levels(grids[i])));
            check_plan(s, grids[i]);
            s.fit(plan_bytes(net_levels(grids[j])));
            check_plan(s, grids[j]);
            const int before = Mem::takes;
            s.fit(plan_bytes(net_levels(grids[j])));
            check(Mem::takes == before, "taken again for the same grid", grids[j][0], grids[j][1], grids[j][2]);
        }
    check(Mem::live.empty(), "given back with the set", 0, 0, 0);
    // the k-th allocation fails: nothing is held, and the next call takes the whole set
    for (int k = 0; k < 22; ++k) {
        BufferSet<Mem> s;
        const int small[3] = {4, 4, 4}, large[3] = {16, 17, 16};
        s.fit(plan_bytes(net_levels(small)));
        Mem::fail_at = Mem::takes + k;
        bool threw = false;
        try {
            s.fit(plan_bytes(net_levels(large)));
        } catch (const std::bad_alloc&) {
            threw = true;
        }
        Mem::fail_at = -1;
        check(threw && s.size() == 0 && Mem::live.empty(), "held after a failed allocation", k, 0, 0);
        s.fit(plan_bytes(net_levels(large)));
        check_plan(s, large);
    }
    // the same of a network's layers: 19 buffers
    for (int k = 0; k < 19; ++k) {
        GridBuffers<Mem> g;
        const int small[3] = {4, 4, 4}, large[3] = {16, 17, 16};
        auto fit = [&](const int* d) { g.fit(d, layer_bytes(net_levels(d))); };
        check(!g.fits(small), "layers of no grid", k, 0, 0);
        fit(small);
        check(g.fits(small) && !g.fits(large), "layers of the grid", k, 0, 0);
        for (int again = 0; again < 2; ++again) {  // refused each time, not taken for laid out
            Mem::fail_at = Mem::takes + k;
            bool threw = false;
            try {
                fit(large);
            } catch (const std::bad_alloc&) {
                threw = true;
            }
            Mem::fail_at = -1;
            check(threw && Mem::live.empty() && !g.fits(small) && !g.fits(large), "layers held after a failed allocation", k,
                  again, 0);
        }
        fit(large);
        check(g.fits(large) && g.set().size() == 19, "layers taken after a failed allocation", k, 0, 0);
        fit(small);
        check(g.set().capacity(0) == 4 * 4 * 4 * 32, "a smaller grid gives the memory back", k, 0, 0);
    }
    int ran = 0;
    {
        OnError quiet([&] { ++ran; });
    }
    check(ran == 0, "OnError without an error", ran, 0, 0);
    try {
        OnError loud([&] { ++ran; });
        throw std::bad_alloc();
    } catch (const std::bad_alloc&) {
        OnError handled([&] { ran += 10; });
    }
    check(ran == 1, "OnError with one", ran, 0, 0);
    std::printf("%s: %d failures\n", failures ? "failed" : "ok", failures);
    return failures ? 1 : 0;
}
