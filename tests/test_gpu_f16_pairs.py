"""CTA pairs of the fp16 convolution (two pixel tiles per tensor-core instruction) against the CPU oracle: odd tile counts (a phantom tile), laps of the
stage and accumulator rings, every addressing mode, and what the pairs refuse."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
PAIRS = range(33, 39)
F16 = dict(in_dtype=np.float16, out_dtype=np.float16, quant=False, bias="f32")
# fp32 sums of fp16 products, rounded once: half an ulp (2^-11) plus the fp32 sums' own error, as in the feature-row form's tests
F16_TOL = 2.0 ** -10


@pytest.fixture(scope="module")
def eng():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


GEOMS = {
    # (geometry, variants that run)
    "two_tiles": (dict(N=1, C=64, K=256, H=16, W=16), 2),                        # one pair; im2col needs 128 KiB: tiled only
    "odd_tiles": (dict(N=5, C=128, K=256, H=17, W=19), 4),
    "pointwise": (dict(N=3, C=96, K=384, H=23, W=21, kh=1, kw=1, pad=0), 3),
    "strided": (dict(N=4, C=80, K=128, H=41, W=43, stride=2), 1),
    "laps": (dict(N=9, C=32, K=128, H=112, W=113), 2),                           # 890 tiles: six per CTA
    "long_reduction": (dict(N=2, C=512, K=512, H=14, W=14), 4),
}


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_against_the_oracle(eng, name):
    geom, expected = GEOMS[name]
    case = cases.make_conv_case(61, **geom, **F16)
    k, n, ran = eng.kernel("conv_f16_tc"), case.out_elems, 0
    want = cases.run_oracle(case).astype(np.float32)
    for tune in PAIRS:
        p = cases.copy_params(case.p)
        p.tune = tune
        if not k.supports(p):
            continue
        got = cases.run_gpu(eng, case, "conv_f16_tc", tune).astype(np.float32)
        assert np.abs(got[:n] - want[:n]).max() <= F16_TOL * np.abs(want[:n]).max(), "tune %d" % tune
        ran += 1
    assert ran == expected


def test_refusals(eng):
    k = eng.kernel("conv_f16_tc")
    for geom in (dict(N=1, C=64, K=200, H=28, W=28), dict(N=1, C=64, K=128, H=9, W=9), dict(N=2, C=64, K=128, H=28, W=28, fused=True)):
        case = cases.make_conv_case(62, **geom, **F16)
        for tune in list(PAIRS) + [39]:
            case.p.tune = tune
            assert not k.supports(case.p)


def test_many_launches_in_a_row(eng):
    """Pairs that follow one another at once, each set up while the one before still runs: its tensor memory, barriers and last commits must be
    through before the pair leaves."""
    case = cases.make_conv_case(63, **GEOMS["odd_tiles"][0], **F16)
    from cldnn_b200 import engine
    n, es = case.out_elems, 2
    want = cases.run_oracle(case).astype(np.float32)
    src, w, bias, outs = eng.upload(case.inp), eng.upload(case.w), eng.upload(case.bias), [eng.alloc(n * es) for _ in range(6)]
    runs = []
    for i, out in enumerate(outs):
        p = cases.copy_params(case.p)
        p.tune = 33 + 2 + i % 4                                # im2col and tiled, 128 and 256 features
        runs.append(eng.kernel("conv_f16_tc").prepare(p, engine.make_args(input0=src, output=out, weights=w, bias=bias)))
    for _ in range(30):
        for r in runs:
            r.run()
    eng.sync()
    assert eng.device_status() == 0
    for out in outs:
        got = out.read(np.float16, n).astype(np.float32)
        assert np.abs(got - want[:n]).max() <= F16_TOL * np.abs(want[:n]).max()
