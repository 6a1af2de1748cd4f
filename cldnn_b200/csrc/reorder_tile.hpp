// Which reorders the tiled transposition takes (tail_ops.cu: reorder_tile_kernel) and what it then touches: host arithmetic only, so that it can be
// checked without a device.
#pragma once
#include <initializer_list>
#include <stdint.h>
#include "../../include/cldnn_b200.h"

namespace b200 {

constexpr int kTileF = 64, kTileP = 64;      // features and pixels of a tile

struct ReorderTilePlan {
    bool to_inner;                           // planar -> feature-innermost; else the other way
    int element;                             // bytes per element, 1 or 2
    int vector;                              // bytes of pixels moved at once on the planar side: 16, 4 or one element
    int features;                            // features read, exactly these
    int stored;                              // features written (to_inner: the rest of them zero)
    int pixels, images;
    int64_t plane_pf, plane_pb, inner_px, inner_pb;      // pitches in elements
    int64_t in_offset, out_offset;           // elements
    unsigned grid_x, grid_y, grid_z;
};

// Both tensors of one element type of 1 or 2 bytes, one of them planes of contiguous pixels, the other rows of contiguous pixels with features
// innermost, in whole and aligned vectors of 16 bytes on that side; false: the general kernel serves the call.  `in` / `out` are the buffers' addresses.
inline bool reorder_tile_plan(const cldnn_b200_reorder_params& p, uintptr_t in, uintptr_t out, ReorderTilePlan& t)
{
    const int es = (p.in.dtype == CLDNN_B200_I8 || p.in.dtype == CLDNN_B200_U8) ? 1 : (p.in.dtype == CLDNN_B200_F16 ? 2 : 0);
    if (p.has_mean || p.in.dtype != p.out.dtype || !es) return false;
    const bool to = p.in.px == 1 && p.out.pf == 1 && p.out.px > 1, from = p.in.pf == 1 && p.in.px > 1 && p.out.px == 1;
    if (!to && !from) return false;
    const cldnn_b200_tensor& plane = to ? p.in : p.out; const cldnn_b200_tensor& inner = to ? p.out : p.in;
    const int64_t pixels = (int64_t)plane.y * plane.x, vf = 16 / es;
    if (pixels < 8 || plane.py != plane.x || inner.py != inner.px * inner.x || pixels >= (1 << 30)) return false;
    if (inner.px % vf || inner.pb % vf || inner.offset % vf || inner.f > inner.px) return false;
    if (to ? p.out.f % vf != 0 : p.out.f != p.in.f) return false;
    // one feature out of a wide row: a tile reads an element per pixel and leaves most of its threads idle.  Below 2^18 pixels it still wins (its blocks are
    // smaller), above it loses: 64 images of 112x112, 10 -> 17 us in 2 bytes; of three features 21 -> 17
    if (!to && p.in.f == 1 && pixels * p.in.b >= (1 << 18)) return false;
    const uintptr_t ia = in + (uintptr_t)(p.in.offset * es), oa = out + (uintptr_t)(p.out.offset * es);
    if ((to ? oa : ia) & 15) return false;
    t.vector = es;
    for (const int v : {16, 4})
        if (pixels * es % v == 0 && plane.pf * es % v == 0 && plane.pb * es % v == 0 && (to ? ia : oa) % (uintptr_t)v == 0) { t.vector = v; break; }
    t.to_inner = to; t.element = es; t.features = p.in.f; t.stored = p.out.f; t.pixels = (int)pixels; t.images = p.in.b;
    t.plane_pf = plane.pf; t.plane_pb = plane.pb; t.inner_px = inner.px; t.inner_pb = inner.pb;
    t.in_offset = p.in.offset; t.out_offset = p.out.offset;
    t.grid_x = (unsigned)((t.stored + kTileF - 1) / kTileF); t.grid_y = (unsigned)((pixels + kTileP - 1) / kTileP); t.grid_z = (unsigned)p.in.b;
    return t.grid_x > 0 && t.grid_y <= 65535u && p.in.b > 0 && t.grid_z <= 65535u;
}

}  // namespace b200
