"""LRN and the 3x3 stride-2 maximum behind it in one launch, against the two kernels apart (bit for bit: the normalised values are rounded
to half before the maximum in both), over maps whose strips, rows and feature vectors end early."""
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


@pytest.mark.parametrize("shape", [(1, 8, 3, 3), (2, 96, 55, 55), (5, 256, 27, 27), (3, 40, 8, 13), (300, 16, 9, 6)])
def test_equals_the_two_kernels(eng, shape):
    from cldnn_b200 import engine
    b, f, y, x = shape
    oy, ox = (y - 3) // 2 + 1, (x - 3) // 2 + 1
    data = (np.random.default_rng(31).standard_normal(b * f * y * x) * 20).astype(np.float16)
    data[::97] = np.float16(np.nan)
    data[::89] = np.float16(-np.inf)
    p, l, q = abi.LrnPoolParams(), abi.LrnParams(), abi.PoolParams()
    q.in_, n_in = abi.tensor(abi.F16, b, f, y, x, "byxf")
    q.out, n_out = abi.tensor(abi.F16, b, f, oy, ox, "byxf")
    l.in_ = l.out = q.in_
    q.mode, q.size_x, q.size_y, q.stride_x, q.stride_y = abi.POOL_MAX, 3, 3, 2, 2
    l.size, l.k, l.alpha, l.beta = 5, 1.0, 1e-2, 0.75
    p.pool, p.lrn_size, p.lrn_k, p.lrn_alpha, p.lrn_beta = q, l.size, l.k, l.alpha, l.beta
    src, mid, two, one = eng.upload(data), eng.alloc(n_in * 2), eng.alloc(n_out * 2), eng.alloc(n_out * 2)
    eng.kernel("lrn_f16_byxf").launch(l, engine.make_args(src, None, mid))
    eng.kernel("pooling_f16_byxf").launch(q, engine.make_args(mid, None, two))
    assert eng.kernel("lrn_pool_f16_byxf").supports(p)
    eng.kernel("lrn_pool_f16_byxf").launch(p, engine.make_args(src, None, one))
    eng.sync()
    assert np.array_equal(two.read(np.uint16, n_out), one.read(np.uint16, n_out))


def test_refuses_what_it_does_not_compute(eng):
    p = abi.LrnPoolParams()
    q = p.pool
    q.in_, _ = abi.tensor(abi.F16, 1, 96, 54, 55, "byxf")
    q.out, _ = abi.tensor(abi.F16, 1, 96, 27, 27, "byxf")     # the last row of windows reaches past the map
    q.mode, q.size_x, q.size_y, q.stride_x, q.stride_y, p.lrn_size = abi.POOL_MAX, 3, 3, 2, 2, 5
    assert not eng.kernel("lrn_pool_f16_byxf").supports(p)


@pytest.mark.parametrize("features", [16, 96])
def test_network_on_a_planar_map(features):
    """In a layout the joint kernel does not take (the input's own, planar) the two kernels run; either way the network's result is that of the
    unoptimised build, up to the rounding of the device's power function."""
    from cldnn_b200 import cldnn as cl
    eng, dt = cl.engine(0), cl.data_types
    lay = cl.layout(dt.f16, cl.format.bfyx, cl.tensor(3, features, 13, 11))
    x = (np.random.default_rng(32).standard_normal((3, features, 11, 13)) * 4).astype(np.float16)
    got = []
    for optimize in (False, True):
        net = cl.network(eng, cl.topology(cl.input_layout("input", lay), cl.lrn("norm", "input"), cl.pooling("pool", "norm", cl.pooling_mode.max, size=(3, 3), stride=(2, 2))),
                         cl.build_options(optimize_data=optimize, outputs=["pool"]))
        net.set_input_data("input", cl.memory.from_numpy(eng, x))
        net.execute()
        got.append(net.get_output("pool").to_numpy().astype(np.float32))
        net.execute()
        assert np.array_equal(net.get_output("pool").to_numpy().astype(np.float32), got[-1])
    assert got[0].shape == got[1].shape and np.abs(got[0] - got[1]).max() <= 2e-3 * np.abs(got[0]).max()
