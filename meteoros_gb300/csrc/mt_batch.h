// Launch rules of the host that need no CUDA headers.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace mt {

// Lanes that march one ray together when the tuning leaves it open, by the rays
// of the launch.  More lanes shorten a ray's serial chain (32 rays alone take 159
// to 218 us by view at one lane, 18 to 20 at 32) and fill the 152 SMs' 155 648
// resident threads; they also compute steps past a ray's exit and scan.  Measured
// both sides of each line, us by view (frames are checkerboard, 1/16 of the pixels):
//   32 | 16  480x270 frame 46 / 36 | 42 / 41, 128x72 full 36 / 25 | 30 / 30
//   16 | 8   800x450 frame 65 / 53 | 69 / 65, 960x540 frame 82 / 65 | 77 / 70
//   8 | 4    1440x810 frame 136 / 114 | 141 / 163, 1600x900 frame 164 / 136 | 161 / 159
//   4 | 2    2240x1260 frame 270 / 220 | 251 / 263, 2560x1440 frame 346 / 282 | 307 / 267
//   2 | 1    3000x1688 frame 417 / 347 | 407 / 466, 860x484 full 311 / 200 | 294 / 219,
//            960x540 full 371 / 241 | 345 / 230
// The lines above are RGBA8's.  On 16-bit volumes a step costs more (wider texels to
// load and convert), and steps past the exit with it, so fewer lanes win from fewer
// rays on, in a light view (few of its steps in cloud) later than in a heavy one:
// the two upper lines lie where no view loses more than 5 %, below the mean's
// crossings (FP16, time of the first over the second, mean and range of 14 views;
// checkerboard frames and bfloat16 within 0.05 of it):
//   32 | 16  75x73 1.08, 0.95 to 1.43; 90x90 1.24, 1.05 to 1.56
//   16 | 8   150x140 1.14, 0.95 to 1.51; 165x160 1.27, 1.15 to 1.44
//   8 | 4    255x255 1.04, 0.84 to 1.23; 300x300 1.20, 1.06 to 1.39, but 1200x1200
//            frames 1.13, 0.90 to 1.30: RGBA8's line holds
//   2 | 1    600x600 367 / 304 / 238 | 331 / 321 / 297 us by view, 670x670
//            437 / 355 / 276 | 366 / 347 / 314: RGBA8's line holds
inline int auto_lanes(long long rays, bool texels16) {
    if (rays <= (texels16 ? 7500 : 8192)) return 32;
    if (rays <= (texels16 ? 22000 : 28000)) return 16;
    if (rays <= 90000) return 8;
    if (rays <= 210000) return 4;
    return rays <= 450000 ? 2 : 1;
}

struct BatchShape {
    int lanes, tile_w, tile_h;
};

// The lanes and tile of a batch: those asked for, or with 0 lanes what mt_render
// would take for its rays (`by_rays`), on tiles shrunk to one pass each (a CTA's
// 128 threads) where the rays are too few to fill the GPU at one lane: two
// sessions' frames (72 000 rays) 307 / 398 -> 168 / 192 us by view.
inline BatchShape batch_shape(int lanes, int tile_w, int tile_h, int by_rays) {
    if (lanes != 0) return BatchShape{lanes, tile_w, tile_h};
    lanes = by_rays;
    while (lanes > 1 && tile_w * tile_h > 128 / lanes) {
        if (tile_w >= tile_h)
            tile_w = (tile_w + 1) / 2;
        else
            tile_h = (tile_h + 1) / 2;
    }
    return BatchShape{lanes, tile_w, tile_h};
}

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
