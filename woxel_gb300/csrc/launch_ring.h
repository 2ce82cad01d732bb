// launch_ring.h — what else runs beside a small frame, and how many warps its tiles get.
//
// A frame too small to fill the chip ends sooner when several warps share each tile (kernels.cu: k_pixel), but costs more issue
// slots: where frames of other streams fill the chip, that is time. Whether they do is not known at a launch, so the last
// launches of the process stand for it: a stream that launched among the last kLaunches counts with the tiles of its last launch.
// Only speed depends on the answer.
#pragma once

#include <cstdint>

namespace wxk {

class LaunchRing {
public:
    static constexpr uint32_t kLaunches = 32;
    // Enters a launch; returns the tiles of the other streams of its device, or any number above `enough` once they exceed it.
    // thread: for cudaStreamPerThread, which is one handle for a stream in each host thread.
    uint64_t enter(int device, uintptr_t stream, uintptr_t thread, uint64_t tiles, uint64_t enough) {
        Entry &own = ring_[next_++ % kLaunches];
        own = Entry{device, stream, thread, tiles};
        uint64_t others = 0;
        for (uint32_t i = 2; i <= kLaunches && i <= next_ && others <= enough; i++) {  // newest first
            const Entry &e = at(i);
            if (e.device != device || e.same_stream(own)) continue;
            uint32_t j = 2;
            while (j < i && !(at(j).device == device && at(j).same_stream(e))) j++;
            if (j == i) others += e.tiles;
        }
        return others;
    }

private:
    struct Entry {
        int device;
        uintptr_t stream, thread;
        uint64_t tiles;
        bool same_stream(const Entry &o) const { return stream == o.stream && thread == o.thread; }
    };
    const Entry &at(uint32_t back) const { return ring_[(next_ - back) % kLaunches]; }
    Entry ring_[kLaunches] = {};
    uint64_t next_ = 0;
};

// 2^n warps a tile: as many, up to 8, as keep the warps of this frame and of the frames beside it within 28 an SM (of 64).
// Mode 3 over 500 spheres and over one, queued frames on one stream, us at 1, 2, 4 and 8 warps a tile: 192 tiles 94, 63, 56, 51 and
// 44, 30, 27, 25; 600 tiles 74, 65, 62, 62 and 34, 30, 27, 28; 2048 tiles 82, 74, 77, 101 and 33, 32, 37, 60; 3750 tiles 85, 84, 96, 152
// and 34, 36, 53, 99. On 16 streams at a time, us a frame at 1 warp a tile and as many as one frame alone would get: 192 tiles
// 8.2, 10.9 and 4.6, 6.7; 600 tiles 9.8, 17.7 and 5.4, 9.8; 2048 tiles 21.5, 33.6 and 10.0, 16.2.
constexpr uint32_t kSplitWarps = 28u;
inline uint32_t pixel_split(uint64_t tiles, uint64_t others, int num_sms) {
    uint32_t s = 0;
    while (s < 3u && ((tiles + others) << (s + 1u)) <= (uint64_t)num_sms * kSplitWarps) s++;
    return s;
}

}  // namespace wxk
