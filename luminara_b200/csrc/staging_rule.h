// staging_rule.h -- which calls' transfers between pageable host memory and the device take the pinned
// staging buffers, whose chunks a team of host threads copies.
//
// A team's threads sleep 2 to 4 ms after their last copy, and waking them costs a call more than a short
// transfer gains.  On B200, ms a call: direct copy / through the buffers right after another call /
// with the threads asleep:
//   40k rays (1.9 MB each way) 0.43 / 0.28 / 0.51    640x360 frame (2.8 MB) 0.34 / 0.27 / 0.38
//   100k rays (4.8 MB)         0.85 / 0.56 / 1.04    960x540 frame (6.2 MB) 0.57 / 0.45 / 0.65
//   200k rays (9.6 MB)         1.60 / 0.95 / 1.42    720p frame (11 MB)     0.93 / 0.64 / 0.77
//   400x225 frame (1.0 MB)     0.22 / 0.18 / 0.24    800x450 AOVs (3.6 MB)  0.38 / 0.24 / 0.32
// So a call that follows others within 2 ms takes the buffers from kMin bytes on, any other call from
// kMinAlone (AOVs, three transfers to one waking, from kMinPlanes).
// Allocating the buffers takes 5-10 ms (a process's first 40k rays 1.1 ms direct, 13.6 with it): a
// frame of kMinAlone bytes does so at once, other calls once kAfter bytes would have used them.
// Plain C++ without locking: the caller holds a mutex.
#pragma once

#include <cstddef>
#include <cstdint>

namespace lum {

enum class StagingUse { Frame, Rays, Planes };

class StagingRule {
public:
    static constexpr size_t kMin = 1u << 20, kMinPlanes = 3u << 20, kMinAlone = 8u << 20, kAfter = 64u << 20;
    static constexpr int64_t kInARow = 2000000;   // ns
    static constexpr int kRow = 4;                // calls before it that make a row: pairs of calls gain nothing

    // A call that transfers `bytes` (its largest transfer; all planes) begins: whether it takes the
    // buffers.  ready: they are allocated, as large as it needs them.
    bool begin(StagingUse use, size_t bytes, bool ready, int64_t now) {
        if (bytes < kMin) return false;
        row_ = now - last_ < kInARow ? row_ + 1 : 0;
        const size_t least = use == StagingUse::Planes ? kMinPlanes : row_ >= kRow ? kMin : kMinAlone;
        if (bytes < least) return false;
        if (ready || (use == StagingUse::Frame && bytes >= kMinAlone)) return true;
        direct_ += bytes;
        return direct_ > kAfter;
    }
    void end(size_t bytes, int64_t now) {
        if (bytes >= kMin) last_ = now;
    }

private:
    int64_t last_ = INT64_MIN / 2;   // the last call's end
    int row_ = 0;
    size_t direct_ = 0;
};

}  // namespace lum
