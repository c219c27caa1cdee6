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

}  // namespace jxr
