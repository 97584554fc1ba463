// Host memory for copies from the device, free of CUDA so that it can be checked without a device.
#pragma once
#include <cstddef>
#include <cstdlib>

namespace stb {

// One block of host memory, page-locked where that is to be had (Pinned: alloc(void **, size_t) -> bool,
// free(void *)), ordinary memory where not: copies into it are slower then, but a run does not
// depend on the system's page-locked memory.
template <typename Pinned>
class HostBlock {
    void *p_ = nullptr;
    bool pinned_ = false;

  public:
    HostBlock() = default;
    HostBlock(const HostBlock &) = delete;
    HostBlock &operator=(const HostBlock &) = delete;
    ~HostBlock() {
        if (p_ && pinned_) Pinned::free(p_);
        if (p_ && !pinned_) free(p_);
    }
    // the block, taken at the first call; null when there is no memory of either kind
    void *take(size_t bytes) {
        if (p_) return p_;
        pinned_ = Pinned::alloc(&p_, bytes);
        if (!pinned_) p_ = malloc(bytes);
        return p_;
    }
    bool pinned() const { return pinned_; }
};

}  // namespace stb
