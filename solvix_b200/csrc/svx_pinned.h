// svx_pinned.h - a growable page-locked host buffer (host code; its allocator
// is a template parameter, so that the growth is tested without a device).
#ifndef SVX_PINNED_H
#define SVX_PINNED_H

#include <cstddef>

namespace svx {

// Contents are valid until the next try_get(); callers synchronise their
// stream first.  Sizes up to POW2_MAX double, so that a growing series
// allocates rarely; larger ones take what they ask for, and so does any size
// whose doubled one is refused.
template <class Host>
class PinnedBufferT {
public:
    static constexpr size_t POW2_MAX = size_t(256) << 20;
    size_t limit = ~size_t(0);  // sizes above are refused (tests, measurements)

    PinnedBufferT() = default;
    PinnedBufferT(const PinnedBufferT&) = delete;
    PinnedBufferT& operator=(const PinnedBufferT&) = delete;
    ~PinnedBufferT() {
        if (p_) Host::free(p_);
    }
    // At least `bytes`, or nullptr where the host refuses them.
    void* try_get(size_t bytes) {
        if (bytes > limit) return nullptr;
        if (bytes > cap_) {
            if (p_) Host::free(p_);
            p_ = nullptr;
            cap_ = 0;
            size_t want = bytes;
            if (bytes <= POW2_MAX)
                for (want = size_t(1) << 20; want < bytes;) want *= 2;
            if (want > limit) want = bytes;
            p_ = Host::alloc(want);
            if (!p_ && want > bytes) p_ = Host::alloc(want = bytes);
            if (p_) cap_ = want;
        }
        return p_;
    }

private:
    void* p_ = nullptr;
    size_t cap_ = 0;
};

}  // namespace svx

#endif  // SVX_PINNED_H
