"""Convolutions in groups whose feature tiles lie inside a group: each group's slice of the input features against its own weights, compared with
the reference-order build (optimize_data off) of the same layer.  Slices that end inside a chunk of the reduction, several tiles per group,
and groups that keep the block-diagonal form beside them."""
import numpy as np
import pytest

from cldnn_b200 import cldnn as cl

pytestmark = pytest.mark.gpu

# groups, features in and out per group, map, filter, images; the last three do not qualify (features per group, slices off 16 bytes)
CASES = {
    "alexnet_conv2": (2, 48, 128, 27, 5, 2),
    "long_slices": (2, 192, 128, 13, 3, 5),
    "two_tiles_per_group": (3, 32, 256, 9, 3, 1),
    "pointwise": (4, 80, 128, 11, 1, 3),
    "many_tiles": (2, 16, 128, 61, 3, 9),
    "dense_192": (2, 192, 192, 13, 3, 1),
    "dense_40": (2, 40, 64, 8, 3, 2),
    "dense_off_16_bytes": (2, 36, 128, 8, 3, 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("half", [False, True])
def test_against_the_reference_order(name, half):
    groups, cin, cout, size, filt, images = CASES[name]
    eng, rng, dt = cl.engine(0), np.random.default_rng(41), cl.data_types
    total_in, total_out = groups * cin, groups * cout
    lay = cl.layout(dt.f16 if half else dt.u8, cl.format.bfyx, cl.tensor(images, total_in, size, size))
    geometry = dict(input_offset=(-(filt // 2), -(filt // 2)), with_activation=True, groups=groups)
    if half:
        x = rng.standard_normal((images, total_in, size, size)).astype(np.float16)
        w = (rng.standard_normal((total_out, cin, filt, filt)) / np.sqrt(cin * filt * filt)).astype(np.float16)
        consts = [("w", w), ("b", (rng.standard_normal(total_out) * 0.1).astype(np.float16))]
        conv = cl.convolution("conv", "input", "w", "b", **geometry)
    else:
        x = rng.integers(0, 256, (images, total_in, size, size), dtype=np.uint8)
        consts = [("w", rng.integers(-127, 128, (total_out, cin, filt, filt), dtype=np.int8)), ("b", rng.integers(-4096, 4097, total_out, dtype=np.int32)),
                  ("q", rng.uniform(2.0 ** -14, 2.0 ** -10, total_out).astype(np.float32))]
        conv = cl.convolution("conv", "input", "w", "b", "q", output_data_type=dt.u8, **geometry)
    mems = [(id, cl.memory.from_numpy(eng, a)) for id, a in consts]
    got = {}
    for optimize in (False, True):
        net = cl.network(eng, cl.topology(cl.input_layout("input", lay), *[cl.data(id, m) for id, m in mems], conv),
                         cl.build_options(optimize_data=optimize, outputs=["conv"]))
        net.set_input_data("input", cl.memory.from_numpy(eng, x))
        net.execute()
        got[optimize] = net.get_output("conv").to_numpy().astype(np.float32)
    if half:
        # one rounding to half of fp32 sums in another order
        assert np.abs(got[True] - got[False]).max() <= 2.0 ** -10 * np.abs(got[False]).max()
    else:
        assert np.array_equal(got[True], got[False])


@pytest.fixture(scope="module")
def raw():
    from cldnn_b200 import engine
    e = engine.Engine(0)
    yield e
    e.close()


# (groups, features in per group, out per group, map, filter, stored features of the weights, tuning variants that run)
SLICES = {"alexnet_conv2": (2, 48, 128, 27, 5, 64), "pointwise": (4, 80, 128, 11, 1, 128), "three_groups": (3, 40, 256, 14, 3, 64), "whole_chunks": (2, 64, 128, 14, 3, 64)}


@pytest.mark.parametrize("name", sorted(SLICES))
def test_a_group_that_is_not_finite_stays_by_itself(raw, name):
    """Inf and NaN among one group's input features: a chunk of the reduction that reaches past the slice of the group before must not bring them in."""
    import cases
    from cldnn_b200 import abi
    groups, cin, cout, size, filt, stored = SLICES[name]
    case = cases.make_conv_case(43, N=3, C=groups * cin, K=groups * cout, H=size, W=size, kh=filt, kw=filt, pad=filt // 2, groups=groups, in_dtype=np.float16,
                                out_dtype=np.float16, quant=False, bias="f32", act=abi.ACT_NONE, f_align=32)
    w = np.zeros((groups * cout, filt, filt, stored), np.float16)
    w[..., :cin] = case.w_logical.transpose(0, 2, 3, 1)
    p, n = case.p, case.out_elems
    case.w = w.reshape(-1)
    p.w_px, p.w_py, p.w_po = stored, stored * filt, stored * filt * filt
    x = case.inp.reshape(3, size, size, -1)
    for bad in range(groups):
        y = x.copy()
        y[:, :, :, bad * cin:(bad + 1) * cin:3] = np.resize(np.array([np.inf, np.nan, -np.inf], np.float16), y[:, :, :, bad * cin:(bad + 1) * cin:3].shape)
        case.inp = y.reshape(-1)
        want = cases.logical_out(case, cases.run_oracle(case)).astype(np.float32)
        rest = np.arange(groups * cout) // cout != bad
        assert np.isfinite(want[:, rest]).all() and not np.isfinite(want[:, ~rest]).all()
        k, ran = raw.kernel("conv_f16_tc"), []
        for tune in range(k.tune_count(p)):
            q = cases.copy_params(p)
            q.tune = tune
            if not k.supports(q):
                continue
            got = cases.logical_out(case, cases.run_gpu(raw, case, "conv_f16_tc", tune)).astype(np.float32)
            assert np.abs(got[:, rest] - want[:, rest]).max() <= 2.0 ** -10 * np.abs(want[:, rest]).max(), "group %d tune %d" % (bad, tune)
            assert not np.isfinite(got[:, ~rest]).all()
            ran.append(tune)
        assert 0 in ran and any(13 <= t < 33 for t in ran) and any(0 < t < 13 for t in ran)
        assert name == "three_groups" or any(t >= 33 for t in ran)


def test_slices_of_many_groups_are_whole_chunks(raw):
    """Beyond four groups a slice that ends inside a chunk is refused rather than mixed with the next group; whole chunks run."""
    import cases
    case = cases.make_conv_case(44, N=1, C=6 * 48, K=6 * 128, H=9, W=9, groups=6, in_dtype=np.float16, out_dtype=np.float16, quant=False, bias="f32")
    k = raw.kernel("conv_f16_tc")
    assert case.p.w_px == 64 and not k.supports(case.p)
    w = np.ascontiguousarray(case.w_logical.transpose(0, 2, 3, 1))
    case.w = w.reshape(-1)
    case.p.w_px, case.p.w_py, case.p.w_po = 48, 48 * 3, 48 * 9
    want, got = cases.run_oracle(case).astype(np.float32), cases.run_gpu(raw, case, "conv_f16_tc", 0).astype(np.float32)
    assert np.abs(got - want).max() <= 2.0 ** -10 * np.abs(want).max()
