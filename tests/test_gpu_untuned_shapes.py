"""What an untuned convolution runs on: the tile shape the estimates prefer (feature tiles of 64 / 128 / 256, four epilogue groups, CTA
pairs, the feature-row form, the patch mode, the first layer's row form) against the CPU oracle, over sizes on either side of where the choice
changes; and the row form's answer to an fp16 image that is not finite."""
import numpy as np
import pytest

import cases
from cldnn_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


GEOMS = {
    "one_tile": dict(N=1, C=64, K=256, H=7, W=7, kh=1, kw=1, pad=0),
    "ragged_features": dict(N=2, C=96, K=200, H=13, W=11, kh=1, kw=1, pad=0),
    "odd_tiles_pair": dict(N=5, C=128, K=256, H=33, W=31),
    "strided": dict(N=3, C=160, K=320, H=29, W=29, kh=1, kw=1, pad=0, stride=2),
    "long_reduction": dict(N=2, C=512, K=136, H=7, W=7),
    "few_features_many_pixels": dict(N=7, C=32, K=24, H=80, W=81, kh=1, kw=1, pad=0),
    "patch": dict(N=2, C=64, K=64, H=28, W=27),
}
# fp32 sums of fp16 products, rounded once: half an ulp (2^-11) plus the fp32 sums' own error, as in the feature-row form's tests
F16_TOL = 2.0 ** -10


@pytest.mark.parametrize("name", sorted(GEOMS))
@pytest.mark.parametrize("fused", [False, True])
def test_untuned_8bit(eng, name, fused):
    case = cases.make_conv_case(91, out_dtype=np.uint8, fused=fused, **GEOMS[name])
    want, got, n = cases.run_oracle(case), cases.run_gpu(eng, case, "conv_i8_tc", 0), case.out_elems
    assert np.array_equal(want[:n], got[:n])


@pytest.mark.parametrize("name", sorted(GEOMS))
@pytest.mark.parametrize("fused", [False, True])
def test_untuned_fp16(eng, name, fused):
    case = cases.make_conv_case(92, in_dtype=np.float16, out_dtype=np.float16, quant=False, bias="f32", fused=fused, **GEOMS[name])
    want, got, n = cases.run_oracle(case).astype(np.float32), cases.run_gpu(eng, case, "conv_f16_tc", 0).astype(np.float32), case.out_elems
    assert np.abs(got[:n] - want[:n]).max() <= F16_TOL * np.abs(want[:n]).max()


@pytest.mark.parametrize("images", [1, 6])                  # below and above the row form's pixel count
def test_untuned_first_layer_8bit(eng, images):
    case = cases.make_conv_case(93, N=images, C=3, K=64, H=224, W=224, kh=7, kw=7, stride=2, pad=3, fmt="bfyx", f_align=1, out_fmt="byxf",
                                in_dtype=np.uint8, out_dtype=np.uint8)
    want, got, n = cases.run_oracle(case), cases.run_gpu(eng, case, "conv_i8_first", 0), case.out_elems
    assert np.array_equal(want[:n], got[:n])


def test_row_form_of_an_image_that_is_not_finite(eng):
    """Only pixels with an Inf or NaN among their own taps may be affected, as in the gather kernel, not whole windows."""
    case = cases.make_conv_case(94, N=2, C=3, K=64, H=136, W=136, fmt="bfyx", f_align=1, out_fmt="byxf", in_dtype=np.float16, out_dtype=np.float16,
                                quant=False, bias="f32", act=abi.ACT_NONE)
    x = case.inp.reshape(-1)
    rng = np.random.default_rng(95)
    at = rng.choice(x.size, 40, replace=False)
    x[at] = np.resize(np.array([np.inf, -np.inf, np.nan], np.float16), 40)
    n = case.out_elems
    gather = cases.run_gpu(eng, case, "conv_first_tc", 1)[:n].astype(np.float32)
    assert 0 < np.isnan(gather).sum() < n // 4
    scale = np.abs(gather[np.isfinite(gather)]).max()
    for tune in (0, 2, 3):
        got = cases.run_gpu(eng, case, "conv_first_tc", tune)[:n].astype(np.float32)
        for special in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(special(got), special(gather))
        finite = np.isfinite(gather)
        assert np.abs(got[finite] - gather[finite]).max() <= F16_TOL * scale
