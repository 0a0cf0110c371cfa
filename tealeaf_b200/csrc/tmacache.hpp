// tmacache.hpp -- the tensor maps of a suite's arrays, each encoded once per
// (array, kind). A launch looks up all the maps its kernel takes and then copies
// them, so a map stays valid for the next N - 1 lookups at least: a full cache
// gives up the entry that was looked up the longest ago (those of released
// buffers come first by themselves). Giving entries up in the order of their
// slots would hand a map found for a launch to the launch's next miss: a chunk's
// own arrays and the refinement's in both precisions come to 50 maps.
#pragma once

namespace tl __attribute__((visibility("hidden"))) {

template <typename Map, int N>
class TmaCache {
public:
    // The map of (ptr, kind), made by encode(Map*) when it is not here; null
    // (and nothing given up) when the encoding is refused.
    template <typename Encode>
    const Map* lookup(const void* ptr, int kind, Encode encode)
    {
        for (int i = 0; i < n_; ++i)
            if (e_[i].ptr == ptr && e_[i].kind == kind) {
                e_[i].used = ++clock_;
                return &e_[i].map;
            }
        Map m;
        if (!encode(&m)) return nullptr;
        int slot = n_;
        if (n_ == N) {
            slot = 0;
            for (int i = 1; i < N; ++i)
                if (e_[i].used < e_[slot].used) slot = i;
        } else {
            ++n_;
        }
        e_[slot].map = m;
        e_[slot].ptr = ptr;
        e_[slot].kind = kind;
        e_[slot].used = ++clock_;
        return &e_[slot].map;
    }

private:
    struct Entry {
        const void* ptr;
        int kind;
        unsigned long long used;   // number of the lookup that last returned it
        Map map;
    };
    Entry e_[N];
    int n_ = 0;
    unsigned long long clock_ = 0;
};

}  // namespace tl
