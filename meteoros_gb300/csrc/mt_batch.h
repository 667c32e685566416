// Host rules of a batch that need no CUDA headers.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace mt {

// The bytes of an image that a batch's reprojections read or write.
struct ImageBytes {
    uintptr_t begin, end;
    bool written;
};

inline ImageBytes image_bytes(const void* p, size_t bytes, bool written) {
    return ImageBytes{(uintptr_t)p, (uintptr_t)p + bytes, written};
}

// Whether a written image overlaps any other image: one sweep by address, each
// image against the furthest end of all before it, or of the written ones.
inline bool written_overlap(std::vector<ImageBytes> images) {
    std::sort(images.begin(), images.end(), [](const ImageBytes& a, const ImageBytes& b) { return a.begin < b.begin; });
    uintptr_t end = 0, written_end = 0;
    for (const ImageBytes& i : images) {
        if (i.begin < (i.written ? end : written_end)) return true;
        end = std::max(end, i.end);
        if (i.written) written_end = std::max(written_end, i.end);
    }
    return false;
}

}  // namespace mt
