"""The feature-row form of the tensor-core convolutions (features as the rows of the tile, the reduction split over a cluster)
against the CPU oracle: every (columns, split) variant at the sizes where a tile, a column block or a CTA's share of the reduction
ends early, and the inner products that take it untuned."""
import numpy as np
import pytest

import cases
from cldnn_b200 import abi

pytestmark = pytest.mark.gpu
I8_BASE, F16_BASE, VARIANTS = 51, 13, 20


@pytest.fixture(scope="module")
def eng():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


GEOMS = {
    # one image, fewer features than a tile; ragged features; features over several tiles; pixel counts around the column widths
    "fc_1": dict(N=1, C=64, K=10, H=1, W=1, kh=1, kw=1, pad=0),
    "fc_17_ragged": dict(N=17, C=1056, K=131, H=1, W=1, kh=1, kw=1, pad=0),
    "fc_129": dict(N=129, C=512, K=256, H=1, W=1, kh=1, kw=1, pad=0),
    "deep_3x3": dict(N=1, C=512, K=136, H=7, W=7),
    "im2col_3x3": dict(N=5, C=160, K=130, H=14, W=13),
    "strided_1x1": dict(N=3, C=96, K=64, H=9, W=7, kh=1, kw=1, pad=0, stride=2),
}
# how many of the 20 variants run: a CTA needs a reduction step (of 128 bytes) for itself
RUNS_8BIT = {"fc_1": 5, "fc_129": 15, "strided_1x1": 10}
RUNS_F16 = {"fc_1": 5, "strided_1x1": 10}
F16 = dict(in_dtype=np.float16, out_dtype=np.float16, quant=False, bias="f32")
# fp32 sums of products of fp16 values, rounded once: the sum's own error is K * 2^-24 of the sum of magnitudes, one half ulp of
# fp16 (2^-11 of the value) is the rest; sqrt(K) cancellation stays below a factor of 16 here, so 2^-10 of the output scale holds both
F16_TOL = 2.0 ** -10


def _variants(k, p, base):
    for v in range(VARIANTS):
        q = cases.copy_params(p)
        q.tune = base + v
        if k.supports(q):
            yield base + v


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_every_8bit_variant_is_bit_exact(eng, name):
    for fused in (False, True):
        case = cases.make_conv_case(71, out_dtype=np.uint8, fused=fused, **GEOMS[name])
        want, ran = cases.run_oracle(case), 0
        for tune in _variants(eng.kernel("conv_i8_tc"), case.p, I8_BASE):
            got = cases.run_gpu(eng, case, "conv_i8_tc", tune)
            assert np.array_equal(want[:case.out_elems], got[:case.out_elems]), "tune %d fused %d" % (tune, fused)
            ran += 1
        assert ran == RUNS_8BIT.get(name, VARIANTS)


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_every_fp16_variant(eng, name):
    for fused in (False, True):
        case = cases.make_conv_case(72, fused=fused, **GEOMS[name], **F16)
        want, ran = cases.run_oracle(case).astype(np.float32), 0
        for tune in _variants(eng.kernel("conv_f16_tc"), case.p, F16_BASE):
            got = cases.run_gpu(eng, case, "conv_f16_tc", tune).astype(np.float32)
            n = case.out_elems
            assert np.abs(got[:n] - want[:n]).max() <= F16_TOL * np.abs(want[:n]).max(), "tune %d fused %d" % (tune, fused)
            ran += 1
        assert ran == RUNS_F16.get(name, VARIANTS)


@pytest.mark.parametrize("images", [1, 15, 33, 128, 300])
def test_untuned_inner_products(eng, images):
    geom = dict(N=images, C=2048, K=1000, H=1, W=1, kh=1, kw=1, pad=0)
    case = cases.make_conv_case(73, bias="f32", calib=True, out_dtype=np.int8, **geom)
    want, got = cases.run_oracle(case), cases.run_gpu(eng, case, "conv_i8_tc", 0)
    assert np.array_equal(want[:case.out_elems], got[:case.out_elems])
    case = cases.make_conv_case(74, **geom, **F16)
    want, got = cases.run_oracle(case).astype(np.float32), cases.run_gpu(eng, case, "conv_f16_tc", 0).astype(np.float32)
    n = case.out_elems
    assert np.abs(got[:n] - want[:n]).max() <= F16_TOL * np.abs(want[:n]).max()


@pytest.mark.parametrize("shift", [1, 2, 7])
@pytest.mark.parametrize("fused", [False, True])
def test_8bit_buffers_off_the_vector_alignment(eng, shift, fused):
    """Output and residual that start anywhere: whole vectors of features have to be stored by bytes, in this form and in the pixel-row kernel."""
    from cldnn_b200 import engine
    for geom, order in ((dict(N=3, C=64, K=131, H=7, W=7), abi.EPILOGUE_REF), (dict(N=2, C=160, K=128, H=9, W=11), abi.EPILOGUE_REF),
                        (dict(N=2, C=64, K=64, H=7, W=7, bias="f32", calib=True, eltw_calib=fused), abi.EPILOGUE_IMAD)):
        case = cases.make_conv_case(75, out_dtype=np.int8, fused=fused, **geom)
        case.p.epilogue_order = order
        want, n = cases.run_oracle(case), case.out_elems
        bufs = {k: eng.upload(v) for k, v in dict(weights=case.w, bias=case.bias, quant=case.quant, calib=case.calib, eltw_calib=case.ecal).items() if v is not None}
        src, k, ran = eng.upload(case.inp), eng.kernel("conv_i8_tc"), 0
        res = eng.upload(np.concatenate([np.zeros(shift, np.int8), case.eltw])) if fused else None
        for tune in [0, 2, 6, 10, 14, 18, 22] + list(range(I8_BASE, I8_BASE + VARIANTS)):
            p = cases.copy_params(case.p)
            p.tune = tune
            if not k.supports(p):
                continue
            out = eng.upload(np.full(n + shift, 77, np.int8))
            k.launch(p, engine.make_args(input0=src, input1=res.ptr + shift if fused else None, output=out.ptr + shift, **bufs))
            eng.sync()
            got = out.read(np.int8)
            assert eng.device_status() == 0 and (got[:shift] == 77).all()
            logical = cases.logical_out(case, got[shift:])
            assert np.array_equal(logical, cases.logical_out(case, want)), "tune %d" % tune
            ran += 1
        assert ran >= 10
