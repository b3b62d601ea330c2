// The tags of the face words of a context's solves held in shared memory (hns_rbgs_chip.cu). A launch of n
// half-sweeps uses n + 1 tags from its first one on. A word that carries a tag must be of the launch that
// waits for it, so no tag may still lie in the words from another launch.
#pragma once

#include <cstdint>

namespace hns {

class ChipTags {
public:
    struct Launch {
        uint32_t first;
        bool clear;  // the words are cleared before the launch
    };
    // Eager launches count on from each other and clear the words only when the count begins: the first
    // time, and again after 2^31 tags (half an hour of the smallest solves). A captured launch has
    // the same tags at every replay, whenever that is, so the words are cleared before it, in the graph,
    // and its tags are of a range that eager launches never use.
    Launch take(uint32_t half_sweeps, bool captured) {
        if (captured) return {kCaptured, true};
        const bool begin = next_ == 0 || half_sweeps >= kCaptured - next_;
        if (begin) next_ = 1;
        const uint32_t first = next_;
        next_ += half_sweeps + 1;
        return {first, begin};
    }

private:
    static constexpr uint32_t kCaptured = 1u << 31;
    uint32_t next_ = 0;  // 0: no eager launch yet
};

}  // namespace hns
