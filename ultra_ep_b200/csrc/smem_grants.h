// Which kernel may use how much dynamic shared memory on which device. The setting belongs to the pair: a kernel that was
// set up on one device starts with 48 KB on the next. Host code without CUDA types.
#pragma once

#include <cstddef>

namespace uep {

class SmemGrants {
    static constexpr int kMost = 512;  // pairs beyond are set up at every launch
    struct Pair {
        const void* fn;
        int device;
        size_t bytes;
    };
    Pair pairs_[kMost];
    int n_ = 0;

public:
    static constexpr size_t kDefault = 48 * 1024;

    // What the pair was granted, 0 if it was never set up.
    size_t granted(const void* fn, int device) const {
        for (int i = 0; i < n_; ++i) {
            if (pairs_[i].fn == fn && pairs_[i].device == device) return pairs_[i].bytes;
        }
        return 0;
    }
    void grant(const void* fn, int device, size_t bytes) {
        for (int i = 0; i < n_; ++i) {
            if (pairs_[i].fn == fn && pairs_[i].device == device) {
                pairs_[i].bytes = bytes;
                return;
            }
        }
        if (n_ < kMost) pairs_[n_++] = Pair{fn, device, bytes};
    }
};

}  // namespace uep
