"""8-bit averages over windows inside the map, on either side of the line between a block per window and a thread per output: against the CPU oracle
at the sizes where a window, a vector of features or the 16-bit sums end, and the time on the far side of that line."""
import numpy as np
import pytest

import oracle_lib
from cldnn_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


def average(dtype, images, features, size, window, stride, mode=abi.POOL_AVG):
    p, out = abi.PoolParams(), (size - window) // stride + 1
    p.in_, n_in = abi.tensor(abi.dtype_of(dtype), images, features, size, size, "byxf")
    p.out, n_out = abi.tensor(abi.dtype_of(dtype), images, features, out, out, "byxf")
    p.mode, p.size_x, p.size_y, p.stride_x, p.stride_y = mode, window, window, stride, stride
    return p, n_in, n_out


@pytest.mark.parametrize("dtype", [np.uint8, np.int8])
@pytest.mark.parametrize("shape", [
    (1, 16, 4, 4, 1), (1, 1280, 7, 7, 1), (2, 272, 16, 16, 1),           # 16 taps; five blocks of features; 256 taps and 17 vectors
    (3, 4096, 9, 8, 1), (5, 48, 21, 5, 2), (1, 256, 40, 4, 4),           # several outputs per image
    (12, 256, 40, 4, 4), (13, 256, 40, 4, 4), (40, 32, 33, 6, 3),        # 1200, 1300 and 4000 blocks: before and behind the line (1258 and 1350)
    (2, 64, 17, 17, 1),                                                  # 289 taps: beyond the 16-bit sums
])
def test_against_the_oracle(eng, dtype, shape):
    from cldnn_b200 import engine
    p, n_in, n_out = average(dtype, *shape)
    info = np.iinfo(dtype)
    for extreme in (False, True):
        x = np.full(n_in, info.min if extreme else 0, dtype)
        if not extreme:
            x = np.random.default_rng(15).integers(info.min, info.max + 1, n_in).astype(dtype)
        elif dtype == np.uint8:
            x[:] = info.max
        src, out = eng.upload(x), eng.upload(np.full(n_out, 77, dtype))
        eng.kernel("pooling_i8_byxf").launch(p, engine.make_args(input0=src, output=out))
        assert np.array_equal(out.read(dtype), oracle_lib.pooling(p, x)[:n_out])


def test_many_short_windows_cost_no_block_each(eng):
    """4x4 averages over a large map, 64 features: a block per output took twenty times the general kernel's time.  The maximum over the same windows
    runs on that kernel and moves the same bytes."""
    from cldnn_b200 import engine
    took = {}
    for mode in (abi.POOL_AVG, abi.POOL_MAX):
        p, n_in, n_out = average(np.uint8, 64, 64, 112, 4, 2, mode)
        src, out = eng.alloc(n_in), eng.alloc(n_out)
        r = eng.kernel("pooling_i8_byxf").prepare(p, engine.make_args(input0=src, output=out))
        took[mode] = min(r.time_ns(3, 10) for _ in range(3))
    assert took[abi.POOL_AVG] < 4 * took[abi.POOL_MAX]
