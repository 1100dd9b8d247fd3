// refusal.h -- remembers that an optional allocation was refused.
//
// A frame can do without some buffers (the binned stage 3's chains, oriented
// sub-boxes).  Asking for one costs a device synchronisation or a query, so a
// refused request is not made again in every frame: only for less memory, or after
// kEvery frames that did without it, when others may have given memory back.
#pragma once
#include <cstddef>
#include <cstdint>

namespace cr {

class Refusal {
public:
    static constexpr uint32_t kEvery = 64;

    // Whether a frame that wants `bytes` goes without them unasked.
    bool stands(size_t bytes) {
        if (bytes_ == 0 || bytes < bytes_) return false;
        if (++frames_ < kEvery) return true;
        bytes_ = 0;
        return false;
    }
    void refused(size_t bytes) {
        bytes_ = bytes;
        frames_ = 0;
    }

private:
    size_t bytes_ = 0;     // the least size refused last (0: none)
    uint32_t frames_ = 0;  // frames that went without it since
};

}  // namespace cr
