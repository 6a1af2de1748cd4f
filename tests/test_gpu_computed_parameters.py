"""Parameters that are not constants: weights, bias and factors written by the kernel in front of a convolution.  That kernel lets the convolution start
before it has ended, so the convolution reads its parameters only after it has waited.  And a bias that a network computes for itself."""
import ctypes as C

import numpy as np
import pytest

import cases
from cldnn_b200 import abi
from cldnn_b200 import cldnn as cl

pytestmark = pytest.mark.gpu
F16_TOL = 2.0 ** -10                                   # one rounding to half of fp32 sums in another order


@pytest.fixture(scope="module")
def eng():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


def slow_copy(eng, src, dst, nbytes, taps):
    """A prepared launch that writes `nbytes` (a multiple of 16) from src to dst as the maximum over a window of taps x taps equal pixels: one thread per 16
    bytes, so it runs long and leaves most of the device free.  Every pixel of the window is the same memory (pitches of zero)."""
    from cldnn_b200 import engine
    p = abi.PoolParams()
    p.in_, _ = abi.tensor(abi.U8, 1, nbytes, taps, taps, "byxf")
    p.out, _ = abi.tensor(abi.U8, 1, nbytes, 1, 1, "byxf")
    p.in_.px = p.in_.py = 0
    p.mode, p.size_x, p.size_y, p.stride_x, p.stride_y = abi.POOL_MAX, taps, taps, 1, 1
    return eng.kernel("pooling_i8_byxf").prepare(p, engine.make_args(input0=src, output=dst))


I8 = dict(N=1, C=64, K=64, H=20, W=20, out_dtype=np.uint8)
DEEP = dict(N=1, C=256, K=192, H=7, W=7, out_dtype=np.uint8)
HALF = dict(in_dtype=np.float16, out_dtype=np.float16, quant=False, bias="f32")
FORMS = {
    # kernel, tuning index, case
    "i8_patch": ("conv_i8_tc", 26, dict(I8, K=128)),
    "i8_tiled": ("conv_i8_tc", 10, I8),
    "i8_resident": ("conv_i8_tc", 2, dict(I8, N=40, H=33, W=31, kh=1, kw=1, pad=0)),
    "i8_pair": ("conv_i8_tc", 49, dict(I8, K=128, N=2)),
    "i8_rows_split": ("conv_i8_tc", 51 + 4 * 2 + 3, DEEP),
    "i8_rows": ("conv_i8_tc", 51 + 4 * 1, DEEP),
    "f16_patch": ("conv_f16_tc", 10, dict(N=1, C=64, K=64, H=20, W=20, **HALF)),
    "f16_rows_split": ("conv_f16_tc", 13 + 4 * 2 + 2, dict(DEEP, **HALF)),
    "untuned_i8": ("conv_i8_tc", 0, DEEP),
    "untuned_f16": ("conv_f16_tc", 0, dict(DEEP, **HALF)),
}


@pytest.mark.parametrize("form", sorted(FORMS))
def test_written_by_the_kernel_in_front(eng, form):
    from cldnn_b200 import engine
    kernel, tune, geom = FORMS[form]
    case = cases.make_conv_case(81, **geom)
    want, n, es = cases.run_oracle(case), case.out_elems, np.dtype(geom["out_dtype"]).itemsize
    arrays = {k: v for k, v in dict(weights=case.w, bias=case.bias, quant=case.quant).items() if v is not None}
    src, out = eng.upload(case.inp), eng.alloc(n * es)
    p = cases.copy_params(case.p)
    p.tune = tune
    assert p.constant_params == 0 and eng.kernel(kernel).supports(p)
    for late in arrays:
        bufs = {k: eng.upload(v) for k, v in arrays.items()}
        final, stale = eng.upload(arrays[late]), np.ones_like(arrays[late])
        copy = slow_copy(eng, final, bufs[late], arrays[late].nbytes, 64)
        conv = eng.kernel(kernel).prepare(p, engine.make_args(input0=src, output=out, **bufs))
        for _ in range(3):
            bufs[late].write(stale)
            copy.run()
            conv.run()
            eng.sync()
            assert eng.device_status() == 0
            got = out.read(np.dtype(geom["out_dtype"]), n)
            if es == 1:
                assert np.array_equal(got, want[:n]), late
            else:
                w32 = want[:n].astype(np.float32)
                assert np.abs(got.astype(np.float32) - w32).max() <= F16_TOL * np.abs(w32).max(), late


@pytest.mark.parametrize("form", ["i8_patch", "i8_tiled", "i8_pair", "i8_rows_split", "f16_patch", "f16_rows_split", "untuned_f16"])
def test_behind_a_kernel_that_runs_longer_than_the_waits(eng, form):
    """A launch set up ahead of a previous kernel that takes 2.6 s more: the limit of 2 s on waits inside a kernel is for that kernel's own time."""
    from cldnn_b200 import engine
    kernel, tune, geom = FORMS[form]
    case = cases.make_conv_case(82, **geom)
    want, n, dt = cases.run_oracle(case), case.out_elems, np.dtype(geom["out_dtype"])
    arrays = {k: v for k, v in dict(weights=case.w, bias=case.bias, quant=case.quant).items() if v is not None}
    src, out, bufs = eng.upload(case.inp), eng.alloc(n * dt.itemsize), {k: eng.upload(v) for k, v in arrays.items()}
    p = cases.copy_params(case.p)
    p.tune = tune
    conv = eng.kernel(kernel).prepare(p, engine.make_args(input0=src, output=out, **bufs))
    scrap = eng.alloc(256)
    probe = slow_copy(eng, scrap, scrap, 16, 512).time_ns(1, 3)
    slow = slow_copy(eng, scrap, scrap, 16, min(int(512 * (2.6e9 / probe) ** 0.5), 46000))   # at most 2^31 taps
    slow.run()
    conv.run()
    eng.sync()
    assert eng.device_status() == 0
    got = out.read(dt, n)
    if dt.itemsize == 1:
        assert np.array_equal(got, want[:n])
    else:
        w32 = want[:n].astype(np.float32)
        assert np.abs(got.astype(np.float32) - w32).max() <= F16_TOL * np.abs(w32).max()


def _weights(rng, k, c, f):
    return (rng.standard_normal((k, c, f, f)) / np.sqrt(c * f * f)).astype(np.float16)


def _run(eng, prims, x, lay, outputs, **options):
    net = cl.network(eng, cl.topology(cl.input_layout("input", lay), *prims), cl.build_options(outputs=outputs, **options))
    net.set_input_data("input", cl.memory.from_numpy(eng, x))
    net.execute()
    got = []
    for _ in range(20):
        net.execute()
        got = [net.get_output(o).to_numpy().astype(np.float32) for o in outputs]
    return got


@pytest.mark.parametrize("optimize", [False, True])
@pytest.mark.parametrize("graph", [False, True])
def test_bias_from_an_inner_product(optimize, graph):
    """The bias is computed early, other small results follow it, and the convolution that reads it comes last: its buffer is nobody else's until then."""
    eng, rng, dt = cl.engine(0), np.random.default_rng(51), cl.data_types
    c, k = 64, 128
    lay = cl.layout(dt.f16, cl.format.bfyx, cl.tensor(1, c, 7, 7))
    x = rng.standard_normal((1, c, 7, 7)).astype(np.float16)
    consts = {"w0": _weights(rng, c, c, 3), "wf": _weights(rng, k, c, 1), "wg": _weights(rng, k, c, 1), "w1": _weights(rng, k, c, 3)}
    mems = {n: cl.memory.from_numpy(eng, a) for n, a in consts.items()}
    datas = [cl.data(n, m) for n, m in mems.items()]
    head = [cl.convolution("conv0", "input", "w0", input_offset=(-1, -1)), cl.pooling("mean", "conv0", cl.pooling_mode.average, global_pooling=True),
            cl.fully_connected("bias", "mean", "wf"), cl.fully_connected("other", "mean", "wg"), cl.activation("square", "other", cl.activation_func.square)]
    last = [cl.convolution("conv1", "input", "w1", "bias", input_offset=(-1, -1))]
    got = _run(eng, datas + head + last, x, lay, ["conv1", "square"], optimize_data=optimize, use_graph=graph)
    # the same with the bias read back and given as data
    bias, = _run(eng, datas[:2] + head[:3], x, lay, ["bias"], optimize_data=optimize, use_graph=graph)
    given = cl.memory.from_numpy(eng, bias.reshape(1, k, 1, 1).astype(np.float16))
    want, = _run(eng, [datas[3], cl.data("bias", given)] + last, x, lay, ["conv1"], optimize_data=optimize, use_graph=graph)
    assert np.abs(bias).max() > 0 and np.array_equal(got[0], want)
