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
        assert _kernels(net) == {"input": "", "norm": "lrn_ref", "pool": "pooling_ref"}
        net.execute()
        assert np.array_equal(net.get_output("pool").to_numpy().astype(np.float32), got[-1])
    assert got[0].shape == got[1].shape and np.abs(got[0] - got[1]).max() <= 2e-3 * np.abs(got[0]).max()


def _build(eng, images, size, outputs, **options):
    """convolution -> LRN -> 3x3 stride-2 maximum -> convolution -> convolution, with intermediate buffers that are reused."""
    from cldnn_b200 import cldnn as cl
    rng, dt = np.random.default_rng(33), cl.data_types
    weights = {"w1": (32, 16, 3, 3), "w2": (64, 32, 3, 3), "w3": (256, 64, 3, 3)}
    mems = {n: cl.memory.from_numpy(eng, (rng.standard_normal(s) / np.sqrt(np.prod(s[1:]))).astype(np.float16)) for n, s in weights.items()}
    lay = cl.layout(dt.f16, cl.format.bfyx, cl.tensor(images, 16, size, size))
    x = (rng.standard_normal((images, 16, size, size)) * 4).astype(np.float16)
    prims = [cl.input_layout("input", lay)] + [cl.data(n, m) for n, m in mems.items()] + [
        cl.convolution("conv1", "input", "w1", input_offset=(-1, -1), with_activation=True), cl.lrn("norm1", "conv1", alpha=1e-2),
        cl.pooling("pool1", "norm1", cl.pooling_mode.max, size=(3, 3), stride=(2, 2)), cl.convolution("conv2", "pool1", "w2", input_offset=(-1, -1)),
        cl.convolution("conv3", "conv2", "w3", input_offset=(-1, -1))]
    net = cl.network(eng, cl.topology(*prims), cl.build_options(optimize_data=True, outputs=outputs, **options))
    inp = cl.memory.from_numpy(eng, x)
    net.set_input_data("input", inp)
    return net, inp, x


def _kernels(net):
    return {i["id"]: i["kernel"] for i in net.primitives_info()}


def test_forced_kernels_keep_the_two_launches(tmp_path):
    from cldnn_b200 import cldnn as cl
    eng = cl.engine(0)
    got = {}
    for forced in (None, "pool1=lrn_pool_f16_byxf", "pool1=pooling_f16_byxf", "pool1=pooling_ref", "norm1=lrn_f16_byxf", "norm1=lrn_ref"):
        net, inp, _ = _build(eng, 3, 21, ["conv3", "pool1"], force_kernel=forced)
        net.execute()
        got[forced], k = net.get_output("pool1").to_numpy(), _kernels(net)
        apart = forced is not None and forced != "pool1=lrn_pool_f16_byxf"
        assert ("norm1" in k) == apart and (k["pool1"] == "lrn_pool_f16_byxf") != apart
        if apart:
            assert k[forced.split("=")[0]] == forced.split("=")[1]
    for forced in list(got)[:5]:
        assert np.array_equal(got[forced], got[None]), forced
    scale = np.abs(got[None].astype(np.float32)).max()
    assert np.abs(got["norm1=lrn_ref"].astype(np.float32) - got[None].astype(np.float32)).max() <= 2e-3 * scale
    net, inp, _ = _build(eng, 3, 21, ["conv3"], tuning=cl.tuning_mode.tuning_tune_and_cache, tuning_cache_path=str(tmp_path / "cache.json"))
    net.execute()
    assert _kernels(net)["pool1"] == "lrn_pool_f16_byxf"


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("before", [False, True])
def test_the_normalised_map_can_be_asked_for(graph, before):
    """get_output of the LRN that runs inside the pooling's launch: its values of that pass, and again after the next one with other input."""
    from cldnn_b200 import cldnn as cl
    eng = cl.engine(0)
    apart, inp_a, x = _build(eng, 2, 19, ["conv3", "norm1"], use_graph=graph)
    net, inp, _ = _build(eng, 2, 19, ["conv3"], use_graph=graph)
    norm = net.get_output("norm1") if before else None
    for scale in (1, 2, -1):
        for n, m in ((apart, inp_a), (net, inp)):
            m.set_values((x * scale).astype(np.float16))
            n.execute()
        assert before or scale != 1 or "norm1" not in _kernels(net)
        norm = norm or net.get_output("norm1")
        net.wait()
        assert np.array_equal(norm.to_numpy(), apart.get_output("norm1").to_numpy())
        assert np.array_equal(net.get_output("conv3").to_numpy(), apart.get_output("conv3").to_numpy())
    assert _kernels(net)["norm1"] == "lrn_f16_byxf" and _kernels(net)["pool1"] == "pooling_f16_byxf"
