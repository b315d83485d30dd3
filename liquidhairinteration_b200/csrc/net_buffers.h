// net_buffers.h -- device buffers that are taken and given back together, and
// the sizes of those a network's sparse plan needs.  Host arithmetic only:
// tests/cpp/net_buffers_check.cpp runs it without a GPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace lhi {

// Buffers from Mem (void* take(size_t), which throws; void give(void*)), each
// with a capacity of its own.  fit() keeps the set while every buffer holds
// what is asked of it; otherwise it takes a new one, or none where one buffer
// cannot be had.
template <class Mem> class BufferSet {
public:
    BufferSet() = default;
    BufferSet(const BufferSet&) = delete;
    BufferSet& operator=(const BufferSet&) = delete;
    ~BufferSet() { release(); }
    bool holds(const std::vector<size_t>& bytes) const {
        if (bytes.size() != cap_.size()) return false;
        for (size_t i = 0; i < bytes.size(); ++i)
            if (bytes[i] > cap_[i]) return false;
        return true;
    }
    void fit(const std::vector<size_t>& bytes) {
        if (holds(bytes)) return;
        release();
        try {
            for (size_t n : bytes) {
                buf_.push_back(nullptr);
                cap_.push_back(std::max(n, size_t(1)));
                buf_.back() = Mem::take(cap_.back());
            }
        } catch (...) {
            release();
            throw;
        }
    }
    void release() {
        for (void* p : buf_)
            if (p) Mem::give(p);
        buf_.clear();
        cap_.clear();
    }
    template <class T> T* at(size_t i) const { return static_cast<T*>(buf_[i]); }
    size_t capacity(size_t i) const { return cap_[i]; }
    size_t size() const { return buf_.size(); }

private:
    std::vector<void*> buf_;
    std::vector<size_t> cap_;
};

// A grid's three levels of the network: every axis halved, rounded down.
struct NetLevels {
    int d[3][3];
    long long vox(int l) const { return (long long)d[l][0] * d[l][1] * d[l][2]; }
};
inline NetLevels net_levels(const int dims[3]) {
    NetLevels n;
    for (int a = 0; a < 3; ++a) {
        n.d[0][a] = dims[a];
        n.d[1][a] = dims[a] / 2;
        n.d[2][a] = n.d[1][a] / 2;
    }
    return n;
}

// Brick tiles of a level: one x plane, 16 y, 8 z.  Grids of equal volume can
// differ in their tiles and in their coarse levels' voxels.
inline long long brick_tiles(const int d[3]) { return (long long)d[0] * ((d[1] + 15) / 16) * ((d[2] + 7) / 8); }

// The sparse plan's buffers: voxel masks (two per level and the dilations'
// intermediate, level 0's size), tile flags per level, tile lists, list counts.
constexpr int kPlanMasks = 7, kPlanFlags = 3, kPlanLists = 11;
// level of each mask; of each list: the six convolutions' outputs, then the
// input channels (0), pool to 1, pool to 2, upsample to 1, upsample to 0
constexpr int kPlanMaskLevel[kPlanMasks] = {0, 0, 1, 1, 2, 2, 0};
constexpr int kPlanListLevel[kPlanLists] = {0, 1, 2, 1, 0, 0, 0, 1, 2, 1, 0};
inline std::vector<size_t> plan_bytes(const NetLevels& n) {
    std::vector<size_t> b;
    for (int l : kPlanMaskLevel) b.push_back(size_t(n.vox(l)));
    for (int l = 0; l < kPlanFlags; ++l) b.push_back(size_t(brick_tiles(n.d[l])));
    for (int l : kPlanListLevel) b.push_back(size_t(brick_tiles(n.d[l])) * 4);
    b.push_back(size_t(kPlanLists) * 4);
    return b;
}

}  // namespace lhi
