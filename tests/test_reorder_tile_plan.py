"""The rule that sends a reorder to the tiled transposition, checked on the CPU over the forms it accepts: every element it reads is one the general
kernel reads, every element it writes one that kernel writes, each vector is aligned, and the tiles cover the tensor."""
import ctypes as C
import itertools
import os
import subprocess

import numpy as np
import pytest

from cldnn_b200 import abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = """#include "%s/cldnn_b200/csrc/reorder_tile.hpp"
extern "C" int plan(const cldnn_b200_reorder_params* p, uint64_t in, uint64_t out, int64_t* r)
{
    b200::ReorderTilePlan t;
    if (!b200::reorder_tile_plan(*p, (uintptr_t)in, (uintptr_t)out, t)) return 0;
    const int64_t v[] = {t.to_inner, t.element, t.vector, t.features, t.stored, t.pixels, t.images, t.plane_pf, t.plane_pb, t.inner_px, t.inner_pb,
                         t.in_offset, t.out_offset, t.grid_x, t.grid_y, t.grid_z, b200::kTileF, b200::kTileP};
    for (int i = 0; i < 18; ++i) r[i] = v[i];
    return 1;
}
""" % ROOT
FIELDS = ("to_inner element vector features stored pixels images plane_pf plane_pb inner_px inner_pb in_offset out_offset grid_x grid_y grid_z "
          "tile_f tile_p").split()


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("reorder_plan")
    src, so = str(d / "plan.cpp"), str(d / "plan.so")
    open(src, "w").write(SHIM)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-shared", "-fPIC", "-O1", src, "-o", so])
    lib = C.CDLL(so)

    def call(p, src_at, dst_at):
        r = (C.c_int64 * len(FIELDS))()
        return dict(zip(FIELDS, r)) if lib.plan(C.byref(p), C.c_uint64(src_at), C.c_uint64(dst_at), r) else None
    return call


def positions(t, features):
    b, f, y, x = np.ogrid[:t.b, :features, :t.y, :t.x]
    return t.offset + b * t.pb + f * t.pf + y * t.py + x * t.px


def inner_slice(dt, b, f, y, x, px, at):
    t, _ = abi.tensor(dt, b, f, y, x, "byxf")
    t.px, t.py, t.pb, t.offset = px, px * x, px * x * y, at
    return t


def planar(dt, b, f, y, x, gap, at):
    t, _ = abi.tensor(dt, b, f, y, x, "bfyx")
    t.pf, t.pb, t.offset = t.pf + gap, (t.pf + gap) * f, at
    return t


def check(p, q, src_at, dst_at):
    es, vf = q["element"], 16 // q["element"]
    # what the kernel touches, from the plan alone: pixels are contiguous on the planar side, features on the other
    b, f, s = np.ogrid[:q["images"], :max(q["features"], q["stored"]), :q["pixels"]]
    plane = b * q["plane_pb"] + f * q["plane_pf"] + s
    inner = b * q["inner_pb"] + f + s * q["inner_px"]
    read = (plane if q["to_inner"] else inner)[:, :q["features"]] + q["in_offset"]
    written = (inner[:, :q["stored"]] if q["to_inner"] else plane[:, :q["features"]]) + q["out_offset"]
    assert np.array_equal(read.ravel(), positions(p.in_, p.in_.f).ravel())
    assert np.array_equal(written.ravel(), positions(p.out, p.out.f).ravel())
    # vectors: rows of the planes from pixel 0 on, groups of 16 bytes of features from feature 0 on
    p_at, i_at = (src_at, dst_at) if q["to_inner"] else (dst_at, src_at)
    p_off, i_off = (q["in_offset"], q["out_offset"]) if q["to_inner"] else (q["out_offset"], q["in_offset"])
    v = q["vector"]
    assert v in (16, 4, es) and q["pixels"] * es % v == 0
    assert not ((p_at + es * (p_off + plane[:, :, :1])) % v).any()
    assert not ((i_at + es * (i_off + inner[:, ::vf])) % 16).any()
    if q["to_inner"]:
        assert q["stored"] % vf == 0
    assert q["grid_x"] * q["tile_f"] >= q["stored"] and q["grid_y"] * q["tile_p"] >= q["pixels"] and q["grid_z"] == q["images"]


def test_touches_what_the_general_kernel_touches(plan):
    taken = refused = 0
    for dt, b, (y, x) in itertools.product((abi.U8, abi.I8, abi.F16), (1, 3), ((1, 8), (3, 3), (7, 4), (5, 13))):
        for f, px, at in itertools.product((1, 5, 8, 16, 24, 33), (8, 16, 32, 48, 64), (0, 8, 16, 24, 40)):
            if at + f > px:
                continue
            for gap, start, base in itertools.product((0, 1, 4), (0, 2, 8), (0, 4, 6)):
                for inwards in (False, True):
                    p = abi.ReorderParams()
                    p.in_, p.out = inner_slice(dt, b, f, y, x, px, at), planar(dt, b, f, y, x, gap, start)
                    src_at, dst_at = 1 << 20, (1 << 24) + base
                    if inwards:
                        p.in_, p.out = p.out, p.in_
                        src_at, dst_at = dst_at, src_at
                        if f % 8:
                            p.out.f = min(-(-f // 16) * 16, px - at)       # the rest of the features is written as zero
                    q = plan(p, src_at, dst_at)
                    taken, refused = taken + (q is not None), refused + (q is None)
                    if q:
                        check(p, q, src_at, dst_at)
    assert taken > 5000 and refused > 5000


def test_a_slice_at_the_end_of_the_last_pixel(plan):
    """8 halves at offset 24 of 32 stored features: nothing lies behind the last pixel's slice."""
    p = abi.ReorderParams()
    p.in_, p.out = inner_slice(abi.F16, 2, 8, 4, 4, 32, 24), planar(abi.F16, 2, 8, 4, 4, 0, 0)
    q = plan(p, 1 << 20, 1 << 24)
    assert q and q["features"] == 8
    check(p, q, 1 << 20, 1 << 24)


@pytest.mark.parametrize("change", [dict(px=30), dict(offset=4), dict(pb=1004), dict(src_at=8), dict(has_mean=1), dict(dtype=abi.F32), dict(f=40), dict(y=1, x=4)])
def test_refused(plan, change):
    """Unaligned rows, bases and slices, a mean, other element types, more features than stored and maps below a vector stay with the general kernel."""
    p, src_at = abi.ReorderParams(), 1 << 20
    p.in_, p.out = inner_slice(abi.F16, 2, 8, 4, 4, 32, 0), planar(abi.F16, 2, 8, 4, 4, 0, 0)
    assert plan(p, src_at, 1 << 24)
    for k, v in change.items():
        if k == "src_at":
            src_at += v
        elif k == "has_mean":
            p.has_mean = v
        elif k in ("y", "x", "f", "dtype"):
            setattr(p.in_, k, v)
            setattr(p.out, k, v)
            if k == "x":
                p.in_.py, p.out.py = p.in_.px * v, v
        else:
            setattr(p.in_, k, v)
    assert plan(p, src_at, 1 << 24) is None


@pytest.mark.parametrize("f,images,taken", [(1, 20, True), (1, 21, False), (2, 21, True)])
def test_one_feature_of_many_pixels(plan, f, images, taken):
    """A single feature out of a wide row stays with the general kernel from 2^18 pixels on."""
    p = abi.ReorderParams()
    p.in_, p.out = inner_slice(abi.U8, images, f, 112, 112, 32, 0), planar(abi.U8, images, f, 112, 112, 0, 0)
    assert (plan(p, 1 << 20, 1 << 30) is not None) == taken
