"""Reorders between planar and feature-innermost layouts (the tiled transposition), element for element, at the sizes where a tile
or a vector ends early: map sizes that leave 16-byte, 4-byte and single-element vectors, feature counts around the tile."""
import ctypes as C

import numpy as np
import pytest

from cldnn_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.float16])
@pytest.mark.parametrize("shape", [(1, 128, 28, 28), (2, 65, 13, 13), (3, 33, 7, 10), (1, 1, 3, 3), (5, 3, 4, 2), (2, 200, 1, 63), (1, 70, 16, 4)])
def test_planar_to_inner_and_back(eng, dtype, shape):
    from cldnn_b200 import engine
    b, f, y, x = shape
    rng = np.random.default_rng(9)
    a = rng.integers(0, 100, size=shape).astype(dtype)
    inner = abi.to_layout(a, "byxf", 32)
    p = abi.ReorderParams()
    p.in_, _ = abi.tensor(abi.dtype_of(a.dtype), b, f, y, x, "bfyx")
    p.out, n = abi.tensor(abi.dtype_of(a.dtype), b, f, y, x, "byxf", 32)
    p.out.f = -(-f // 32) * 32                                    # feature padding is written as zero
    src, dst = eng.upload(a), eng.upload(np.full(n, 77, dtype=a.dtype))
    eng.kernel("reorder_ref").launch(p, engine.make_args(input0=src, output=dst))
    assert np.array_equal(dst.read(a.dtype), inner)
    q = abi.ReorderParams()
    q.in_, _ = abi.tensor(abi.dtype_of(a.dtype), b, f, y, x, "byxf", 32)
    q.out, n = abi.tensor(abi.dtype_of(a.dtype), b, f, y, x, "bfyx")
    back = eng.upload(np.full(n, 77, dtype=a.dtype))
    eng.kernel("reorder_ref").launch(q, engine.make_args(input0=dst, output=back))
    assert np.array_equal(back.read(a.dtype), a.reshape(-1))


@pytest.mark.parametrize("dtype", [np.uint8, np.float16])
@pytest.mark.parametrize("f,at,stored", [(8, 24, 32), (16, 16, 32), (5, 8, 16), (33, 16, 64), (64, 0, 64), (1, 48, 64)])
def test_a_slice_of_the_features(eng, dtype, f, at, stored):
    """Some of a pixel's features to planes and back, up to the last element of the buffer; the other features stay as they are."""
    from cldnn_b200 import engine
    b, y, x = 2, 9, 12
    rng = np.random.default_rng(10)
    whole = rng.integers(0, 100, size=(b, y, x, stored)).astype(dtype)
    p = abi.ReorderParams()
    p.in_, _ = abi.tensor(abi.dtype_of(whole.dtype), b, f, y, x, "byxf")
    p.in_.px, p.in_.py, p.in_.pb, p.in_.offset = stored, stored * x, stored * x * y, at
    p.out, n = abi.tensor(abi.dtype_of(whole.dtype), b, f, y, x, "bfyx")
    src, dst = eng.upload(whole), eng.upload(np.full(n, 77, dtype=dtype))
    eng.kernel("reorder_ref").launch(p, engine.make_args(input0=src, output=dst))
    want = np.ascontiguousarray(whole[..., at:at + f].transpose(0, 3, 1, 2))
    assert np.array_equal(dst.read(dtype), want.reshape(-1))
    q = abi.ReorderParams()
    q.in_, q.out = p.out, p.in_
    other = rng.integers(100, 120, size=whole.shape).astype(dtype)
    back = eng.upload(other)
    eng.kernel("reorder_ref").launch(q, engine.make_args(input0=dst, output=back))
    other[..., at:at + f] = whole[..., at:at + f]
    assert np.array_equal(back.read(dtype).reshape(whole.shape), other)
