// orient_tile.h -- which source bytes one tile of an orientation reads, on the
// device and, for checks of the arithmetic, on the host.
#pragma once
#include <stdint.h>

#include "../../include/jxr_b200.h"
#include "lifting.cuh"   // JXR_HD

namespace jxr {

JXR_HD bool swaps_axes(int o) { return o >= JXRB_ORIENT_TRANSPOSE; }

// source_coordinates (orientation.rs:193-211): the source pixel of
// destination pixel (dx, dy) of a w x h source.
JXR_HD void source_of(int o, uint32_t w, uint32_t h, uint32_t dx, uint32_t dy, uint32_t &sx, uint32_t &sy) {
    switch (o) {
    case JXRB_ORIENT_MIRROR_HORIZONTAL: sx = w - 1 - dx; sy = dy; break;
    case JXRB_ORIENT_ROTATE180: sx = w - 1 - dx; sy = h - 1 - dy; break;
    case JXRB_ORIENT_MIRROR_VERTICAL: sx = dx; sy = h - 1 - dy; break;
    case JXRB_ORIENT_TRANSPOSE: sx = dy; sy = dx; break;
    case JXRB_ORIENT_ROTATE90: sx = dy; sy = h - 1 - dx; break;
    case JXRB_ORIENT_TRANSVERSE: sx = w - 1 - dy; sy = h - 1 - dx; break;
    case JXRB_ORIENT_ROTATE270: sx = w - 1 - dy; sy = dx; break;
    default: sx = dx; sy = dy;
    }
}

// A tile of up to `side` x `side` pixels at destination pixel (dx0, dy0) and
// the source rectangle it comes from.
struct OrientTile {
    int dw, dh;          // destination pixels
    uint32_t sx0, sy0;   // source rectangle
    int sw, sh;
};
JXR_HD OrientTile orient_tile(int o, uint32_t w, uint32_t h, uint32_t side, uint32_t dx0, uint32_t dy0) {
    const bool swap = swaps_axes(o);
    const uint32_t ow = swap ? h : w, oh = swap ? w : h;
    OrientTile t;
    t.dw = (int)((dx0 + side < ow ? dx0 + side : ow) - dx0);
    t.dh = (int)((dy0 + side < oh ? dy0 + side : oh) - dy0);
    // the extremes of the tile's corners
    uint32_t ax, ay, bx, by;
    source_of(o, w, h, dx0, dy0, ax, ay);
    source_of(o, w, h, dx0 + t.dw - 1, dy0 + t.dh - 1, bx, by);
    t.sx0 = ax < bx ? ax : bx;
    t.sy0 = ay < by ? ay : by;
    t.sw = swap ? t.dh : t.dw;
    t.sh = swap ? t.dw : t.dh;
    return t;
}

// Whether the aligned words that hold a tile's source rows all lie inside the
// surface of `bytes` bytes at `src`; its first row starts `offset` bytes into
// it.  Rows ascend, so the word of the first row's first byte and the one of
// the last row's last byte decide: the tile may touch neither end of the
// surface and still have fewer bytes before or after it than a word has (a
// column of one or two 1-byte pixels beside it, a surface one or two pixels
// wide).
JXR_HD bool words_inside(uintptr_t src, uint64_t bytes, uint64_t offset, uint64_t pitch, int row_bytes, int rows) {
    const uint64_t left = bytes - (offset + (uint64_t)(rows - 1) * pitch + row_bytes);   // after the last row
    const uint32_t before = (uint32_t)(src + offset) & 3, after = (uint32_t)(left - (src + bytes)) & 3;
    return offset >= before && left >= after;
}

// Whether pixels of `n` bytes on surfaces at `address` (the two pointers' bits
// together) go to the kernel compiled for their size: the usual sizes, where
// both surfaces are aligned to its unit.  Other sizes, and surfaces off that
// alignment, keep the kernel that takes any of them.
//
// So do small surfaces of 1 to 3 bytes a pixel: until every SM has tiles
// enough, a tile's latency counts, and its three passes over 64 x 64 pixels take
// longer than the one word a thread moves at a time over 32 x 32 (us, any
// size's kernel / the pixel's: 301 x 217 of 1, 2, 3 bytes 2.8 / 5.3, 2.9 / 6.1,
// 6.0 / 7.6; 999 x 801 5.0 / 5.6, 5.0 / 6.4, 10.5 / 7.0; 1203 x 900 of 2 bytes 6.1
// / 6.4; 1600 x 1204 8.7 / 5.2, 8.8 / 5.9, 20 / 8.4; 601 x 499 of 3 bytes 7.1 /
// 7.9, 801 x 603 8.2 / 6.1 to 8.3).
//
// And narrow ones, whose tiles leave most of a warp's lanes and of a tile's
// groups without pixels (the pixel's kernel's time over any size's, surfaces of
// 2 M pixels 7, 8 and 12 wide or high: 1 byte 1.62, 1.27, 0.94; 2 bytes 1.81, 1.35,
// 1.01 (8 M pixels 1.09), and 1.00 at 16; 3 bytes 1.23, 0.85, 0.67; 4 bytes 1.13, 1.06, 0.87; 6 bytes 1.48, 1.15,
// 0.86; 8, 12 and 16 bytes 1.0 to 1.05, 0.94 to 0.99, 0.72 to 0.87).
inline bool takes_pixel_kernel(uint32_t n, uintptr_t address, uint32_t width, uint32_t height) {
    const uint32_t unit = n % 4 == 0 ? 4 : n % 2 == 0 ? 2 : 1, side = width < height ? width : height;
    if (!(n <= 4 || n == 6 || n == 8 || n == 12 || n == 16) || address % unit != 0) return false;
    const uint64_t pixels = (uint64_t)width * height;
    if (pixels < (n == 1 ? uint64_t(1) << 20 : n == 2 ? uint64_t(5) << 18 : n == 3 ? uint64_t(3) << 17 : 0)) return false;
    return side >= (n == 3 || n >= 8 ? 8u : n == 2 ? 16u : 12u);
}

}  // namespace jxr
