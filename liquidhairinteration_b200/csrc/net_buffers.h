// net_buffers.h -- device buffers that are taken and given back together, and
// the sizes of those a network's layers and its sparse plan need.  Host
// arithmetic only: tests/cpp/net_buffers_check.cpp runs it without a GPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <exception>
#include <vector>

namespace lhi {

// Runs f when an exception leaves the scope.
template <class F> class OnError {
public:
    explicit OnError(F f) : f_(f), before_(std::uncaught_exceptions()) {}
    OnError(const OnError&) = delete;
    OnError& operator=(const OnError&) = delete;
    ~OnError() {
        if (std::uncaught_exceptions() > before_) f_();
    }

private:
    F f_;
    int before_;
};

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

// A set laid out for one grid: another grid gives it back and takes its own,
// and it is no grid's after a failed allocation.
template <class Mem> class GridBuffers {
public:
    bool fits(const int dims[3]) const { return dims[0] == dims_[0] && dims[1] == dims_[1] && dims[2] == dims_[2]; }
    void fit(const int dims[3], const std::vector<size_t>& bytes) {
        for (int& d : dims_) d = 0;
        set_.release();
        set_.fit(bytes);
        for (int a = 0; a < 3; ++a) dims_[a] = dims[a];
    }
    template <class T> T* at(size_t i) const { return set_.template at<T>(i); }
    const BufferSet<Mem>& set() const { return set_; }

private:
    BufferSet<Mem> set_;
    int dims_[3] = {0, 0, 0};
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

// The layers' buffers, in NetBuffers' order: BF16 activations a0 .. u0, FP32 y,
// BF16 gradients g[0 .. 5], FP32 dx and acc.
inline std::vector<size_t> layer_bytes(const NetLevels& n) {
    const size_t V0 = size_t(n.vox(0)), V1 = size_t(n.vox(1)), V2 = size_t(n.vox(2));
    return {V0 * 32,  V0 * 32, V1 * 32, V1 * 64, V2 * 64,  V2 * 128,  // a0 h0 p0 h1 p1 h2
            V1 * 128, V1 * 64, V0 * 64, V0 * 32, V0 * 4,              // q1 u1 q0 u0 y
            V0 * 32,  V1 * 64, V2 * 128, V1 * 64, V0 * 32, V0 * 32,   // g
            std::max(V0 * 128, V1 * 256), std::max(V1 * 128, V2 * 256)};
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
