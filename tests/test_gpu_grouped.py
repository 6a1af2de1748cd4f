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
