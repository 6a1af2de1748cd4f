"""The work that users of this framework have it do, as cases that can be measured: whole networks and single
convolution layers, built and executed through the topology / network interface (cldnn_b200/cldnn.py) with the
optimising build and otherwise default options, as a program does that has not tuned for its own sizes.

A program keeps one engine for its life; each state below is one network of that program with its constants, its input
and its output memory."""
import functools
import math

import numpy as np
import torch

from cldnn_b200 import cldnn as cl
from cldnn_b200 import topologies

MAX_OPS = 1.97e12           # ResNet-50 at batch 256, the largest listed case
MAX_LAYER_VALUES = 40e6     # values in and out of a drawn layer, as of the largest single layers of the networks


def _network(name, model, batch, io="device", image=224):
    return {"name": name, "model": model, "batch": batch, "image": image, "io": io}


def _layer(name, dtype, batch, features_in, features_out, size, filter, stride):
    return {"name": name, "model": "layer", "dtype": dtype, "batch": batch, "features_in": features_in, "features_out": features_out,
            "size": size, "filter": filter, "stride": stride}


def listed():
    return [
        # one int8 convolution by itself, the smallest call a program makes: latency
        _layer("conv_int8_28x28_b1", "int8", 1, 128, 128, 28, 3, 1),
        # one layer of the VGG16 sweep, fp16, on data in the caller's planar layout
        _layer("conv_fp16_28x28_b32", "fp16", 32, 512, 512, 28, 3, 1),
        # an online request: one image arrives in host memory, its class probabilities are read back
        _network("resnet50_int8_b1_request", "resnet50_int8", 1, "host"),
        # a single image already on the GPU, the network with the most launches for the least work
        _network("mobilenet_v2_int8_b1", "mobilenet_v2_int8", 1),
        # a small, odd batch as a batching server collects it
        _network("resnet50_int8_b13", "resnet50_int8", 13),
        _network("alexnet_fp16_b5", "alexnet_fp16", 5, image=227),
        # ordinary batches
        _network("resnet50_int8_b64", "resnet50_int8", 64),
        _network("mobilenet_v2_int8_b128", "mobilenet_v2_int8", 128),
        _network("vgg16_fp16_b32", "vgg16_fp16", 32),
        # large batches: offline throughput
        _network("alexnet_int8_b256", "alexnet_int8", 256, image=227),
        _network("alexnet_fp16_b256", "alexnet_fp16", 256, image=227),
        _network("resnet50_int8_b256", "resnet50_int8", 256),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    if rng.random() < 0.3:
        size, filter = rng.choice((7, 13, 14, 17, 27, 28, 35, 55, 56, 112)), rng.choice((1, 3, 3, 5))
        case = _layer(None, rng.choice(("int8", "fp16")), 1, _log_int(rng, 16, 512), _log_int(rng, 16, 512), size, filter, rng.choice((1, 1, 2)))
        per_image = (case["features_in"] + case["features_out"]) * size * size
        most = max(1, min(256, int(MAX_LAYER_VALUES / per_image), int(MAX_OPS / work(case)["flops"])))
        case["batch"] = _log_int(rng, 1, most)
    else:
        model = rng.choice(("resnet50_int8", "resnet50_int8", "mobilenet_v2_int8", "vgg16_fp16", "alexnet_fp16", "alexnet_int8"))
        most = {"resnet50_int8": 250, "mobilenet_v2_int8": 200, "vgg16_fp16": 32, "alexnet_fp16": 250, "alexnet_int8": 250}[model]
        image = 227 if model.startswith("alexnet") else (224 if model == "vgg16_fp16" else rng.choice((160, 192, 224, 224)))
        case = _network(None, model, _log_int(rng, 1, most), "host" if rng.random() < 0.2 else "device", image)
    del case["name"]
    return case


# ---- the topologies ----------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _model(model, image):
    """A model's primitives and constants: a program loads them once, whatever batch it then runs."""
    return getattr(topologies, model)(1, image=image)


def _layer_spec(case):
    rng = np.random.default_rng(7)
    s, dt = topologies.Spec(), cl.data_types
    k, c, f = case["features_out"], case["features_in"], case["filter"]
    int8 = case["dtype"] == "int8"
    s.input_id = "input"
    s.input_layout = cl.layout(dt.u8 if int8 else dt.f16, cl.format.bfyx, cl.tensor(1, c, case["size"], case["size"]))
    s.add(cl.input_layout("input", s.input_layout))
    geometry = dict(stride=(case["stride"], case["stride"]), input_offset=(-(f // 2), -(f // 2)), with_activation=True)
    if int8:
        s.const("conv_w", rng.integers(-127, 128, size=(k, c, f, f), dtype=np.int8))
        s.const("conv_b", rng.integers(-4096, 4097, size=k, dtype=np.int32))
        s.const("conv_q", rng.uniform(2.0 ** -14, 2.0 ** -10, size=k).astype(np.float32))
        s.add(cl.convolution("conv", "input", "conv_w", "conv_b", "conv_q", output_data_type=dt.i8, **geometry))
    else:
        s.const("conv_w", (rng.standard_normal((k, c, f, f)) * np.sqrt(2.0 / (c * f * f))).astype(np.float16))
        s.const("conv_b", (rng.standard_normal(k) * 0.05).astype(np.float16))
        s.add(cl.convolution("conv", "input", "conv_w", "conv_b", **geometry))
    s.outputs = ["conv"]
    return s


def _spec(case):
    """The case's primitives; only the input layout depends on the batch."""
    base = _layer_spec(case) if case["model"] == "layer" else _model(case["model"], case["image"])
    s, lay = topologies.Spec(), base.input_layout
    s.input_id, s.outputs, s.consts = base.input_id, list(base.outputs), base.consts
    s.input_layout = cl.layout(lay.data_type, lay.format, cl.tensor(case["batch"], lay.size.feature, lay.size.x, lay.size.y))
    s.prims = [cl.input_layout(s.input_id, s.input_layout) if p.kind == "input_layout" else p for p in base.prims]
    return s


# ---- preparing and running ---------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _engine():
    return cl.engine(torch.cuda.current_device())


class _DeviceView:
    """A framework memory as other libraries see it: its address, shape and element type.  A tensor made from it keeps this
    object, and with it the memory."""

    def __init__(self, mem):
        self.memory, lay = mem, mem.get_layout()
        shape = (lay.size.batch, lay.size.feature, lay.size.y, lay.size.x)
        self.__cuda_array_interface__ = {"shape": shape, "typestr": np.dtype(lay.np_dtype()).str, "data": (mem.device_ptr(), False), "version": 3}


class _State:
    pass


def prepare(case, seed):
    s, spec, eng = _State(), _spec(case), _engine()
    topo, s.constants = spec.realise(eng)
    s.net = cl.network(eng, topo, cl.build_options(optimize_data=True, outputs=spec.outputs))
    s.output_ids, lay = spec.outputs, spec.input_layout
    shape = (lay.size.batch, lay.size.feature, lay.size.y, lay.size.x)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    # 8-bit images over their whole range, fp16 ones normalised
    s.images = torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=gen) if lay.data_type == cl.data_types.u8 else \
        torch.randn(shape, dtype=torch.float32, device="cuda", generator=gen).half()
    s.host = case.get("io") == "host"
    if s.host:
        s.images = s.images.cpu().numpy()
        s.input = cl.memory.allocate(eng, lay)
    else:
        torch.cuda.synchronize()
        s.input = cl.memory.attach(eng, lay, s.images.data_ptr())
        s.memories = {o: s.net.get_output(o) for o in s.output_ids}
        s.outputs = {o: torch.as_tensor(_DeviceView(m), device="cuda") for o, m in s.memories.items()}
    s.net.set_input_data(spec.input_id, s.input)
    return s


def run(s):
    if s.host:
        s.input.write_flat(s.images)
        s.net.execute()
        return {o: s.net.get_output(o).to_numpy() for o in s.output_ids}
    s.net.execute()
    return s.outputs


# ---- what a pass cannot do without -------------------------------------------------------------------------------------

def work(case):
    if case["model"] == "layer":
        c, k, f, n = case["features_in"], case["features_out"], case["filter"], case["batch"]
        out = (case["size"] + 2 * (f // 2) - f) // case["stride"] + 1
        value = 1 if case["dtype"] == "int8" else 2
        constants = k * c * f * f * value + k * (8 if value == 1 else 2)
        return {"bytes": value * n * (c * case["size"] ** 2 + k * out * out) + constants, "flops": 2 * n * k * out * out * c * f * f}
    spec = _spec(case)
    ops, _ = topologies.conv_ops(spec)
    lay = spec.input_layout
    image = lay.size.feature * lay.size.y * lay.size.x * np.dtype(lay.np_dtype()).itemsize
    outputs = 1000 * (2 + 2 if lay.data_type == cl.data_types.f16 else 4 + 1)        # probabilities and logits
    return {"bytes": sum(c.nbytes for c in spec.consts.values()) + case["batch"] * (image + outputs), "flops": case["batch"] * ops}


def tolerance(case):
    """Four times what the reference-order kernels (optimize_data off: other order of the sums, fp32 accumulation as well)
    differ by on the same fp16 network or layer; the 8-bit networks are integers up to the logits."""
    if case["model"] == "layer":
        return "exact" if case["dtype"] == "int8" else {"rel": 2.5e-4, "max": 2e-2}
    if case["model"].endswith("int8"):
        return {"rel": 1e-5}                # the fp32 softmax behind the exact logits
    if case["model"] == "vgg16_fp16":
        return {"rel": 2e-2, "max": 0.8}    # probabilities from fp16 logits of a few tens: exp() of their rounding
    return {"rel": 1.2e-3, "max": 1e-2}
