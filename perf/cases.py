"""The work this framework is used for, as cases that can be timed and compared.

Each case is one pass through the public entry points, as a program that uses the framework calls them:

* ``infer``  -- a ``conv.Conv2d`` / ``conv.Conv3d`` module in evaluation mode (bias, ReLU and 2x2 pool fused);
* ``train``  -- forward, backward and a weight update of such a module: new weights on every pass, as in a training loop;
* ``call``   -- the reference's functional operators on tensors in torch order: weights are given with every call;
* ``stack``  -- the VGG-16 convolution stack, called layer by layer or replayed as a CUDA graph.

Sizes are those of the repository's configurations, tests and benchmark, or round and ragged neighbours of them.
"""
import math

import torch

from pytorch_winoconv_b200 import conv, dwm, engine, matrix_conv, matrix_conv3d

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
LEARNING_RATE = 1e-7


def _case(name, kind, dtype, n, c, k, size, kernel, stride=1, **more):
    """``size``: input extent per spatial dimension, ``kernel``: taps per dimension (padding is kernel // 2)."""
    size = tuple(size)
    case = {"kind": kind, "dtype": dtype, "n": n, "c": c, "k": k, "nd": len(size), "d": size[0] if len(size) == 3 else 1,
            "h": size[-2], "w": size[-1], "kernel": kernel, "stride": stride, "bias": True, "relu": False, "pool": False,
            "channels_last": True}
    case.update(more)
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # one image through a middle layer: what a latency-bound service waits for, the launch path more than the kernel
        _case("infer_n1_c64_56_f16", "infer", "f16", 1, 64, 64, (56, 56), 3, relu=True),
        # a few images of an odd size through an odd number of channels: detection or segmentation crops in bfloat16
        _case("infer_n3_c72_k120_ragged_bf16", "infer", "bf16", 3, 72, 120, (37, 51), 3),
        # the 256-channel layer of the benchmark at a serving batch
        _case("infer_n32_c256_28_f16", "infer", "f16", 32, 256, 256, (28, 28), 3, relu=True),
        # an RGB stem: 7x7 at stride 2 on images as a loader delivers them (torch's contiguous order)
        _case("infer_stem_7x7s2_n32_f16", "infer", "f16", 32, 3, 64, (224, 224), 7, 2, relu=True, channels_last=False),
        # a large kernel, the case the DWM decomposition is there for
        _case("infer_5x5_n32_c128_56_f16", "infer", "f16", 32, 128, 128, (56, 56), 5),
        # video / volumes
        _case("infer_3d_n8_c64_16x56_f16", "infer", "f16", 8, 64, 64, (16, 56, 56), 3),
        # single precision, where the caller asks for fp32 results
        _case("infer_n8_c64_56_f32", "infer", "f32", 8, 64, 64, (56, 56), 3),
        # the reference's own operator: float tensors in torch order, the filter given with each call
        _case("dwm2d_5x5_n8_c64_56_f32", "call", "f32", 8, 64, 64, (56, 56), 5, channels_last=False),
        # one training step of a middle layer: forward, three gradients, new weights
        _case("train_n32_c128_28_f16", "train", "f16", 32, 128, 128, (28, 28), 3),
        # one training step of a downsampling layer in bfloat16
        _case("train_3x3s2_n16_c64_k128_56_bf16", "train", "bf16", 16, 64, 128, (56, 56), 3, 2, bias=False),
        # the stack at batch 1, replayed as a graph: the lowest latency a user can get
        _stack("vgg16_n1_graph_f16", 1, 224, True),
        # the stack at a throughput batch
        _stack("vgg16_n64_f16", 64, 224, False),
    ]


def _stack(name, n, hw, graph, dtype="f16"):
    case = {"kind": "stack", "dtype": dtype, "n": n, "h": hw, "w": hw, "graph": graph}
    if name is not None:
        case["name"] = name
    return case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo=1, hi=512):
    """Mostly multiples of 8, as networks have them; one in four as it comes (RGB, odd counts)."""
    c = _log_int(rng, lo, hi)
    return c if rng.random() < 0.25 else max(8, (c + 4) // 8 * 8)


#: the most multiply-adds x 2 (direct convolution) of a drawn case, and the most elements of its input and output
MOST = {"infer": (4e11, 1.2e8), "infer_f32": (4e10, 3e7), "call": (2e10, 2e7), "train": (4e10, 4e7)}


def draw(rng):
    kind = rng.choice(["infer"] * 5 + ["infer_f32", "call", "call", "train", "train", "stack"])
    if kind == "stack":
        return _stack(None, _log_int(rng, 1, 48), 32 * rng.randint(2, 7), rng.random() < 0.5, rng.choice(["f16", "f16", "bf16"]))
    flops_most, elements_most = MOST[kind]
    while True:
        dtype = "f32" if kind == "infer_f32" else rng.choice(["f32", "f16"]) if kind == "call" else rng.choice(["f16", "f16", "bf16"])
        nd = 3 if rng.random() < 0.2 else 2
        if nd == 2:
            h = _log_int(rng, 7, 224)
            size = (h, h if rng.random() < 0.5 else max(7, int(h * rng.uniform(0.6, 1.6))))
            kernel = rng.choice([1, 3, 3, 3, 3, 5, 5, 7, 9])
        else:
            h = _log_int(rng, 7, 64)
            size = (_log_int(rng, 4, 32), h, h if rng.random() < 0.5 else max(7, int(h * rng.uniform(0.6, 1.6))))
            kernel = rng.choice([1, 3, 3, 3, 5]) if dtype != "f32" else rng.choice([1, 3])
        stride = 2 if rng.random() < 0.2 else 1
        c, k = _channels(rng), _channels(rng, 8)
        if kind == "train":
            c = max(8, c)       # a layer that sees images has no data gradient: middle layers
        case = _case(None, kind.split("_")[0], dtype, _log_int(rng, 1, 64), c, k, size, kernel, stride,
                     bias=rng.random() < 0.6, channels_last=kind != "call" and rng.random() < 0.8)
        if kind != "call" and kind != "train":
            case["relu"] = rng.random() < 0.5
            case["pool"] = nd == 2 and stride == 1 and rng.random() < 0.2
        x, y = _in_out_elements(case)
        if _flops(case) <= flops_most and x + y <= elements_most:
            return case


def _out_extents(case):
    p, r, s = case["kernel"] // 2, case["kernel"], case["stride"]
    sp = [case["d"], case["h"], case["w"]][3 - case["nd"]:]
    return [(e + 2 * p - r) // s + 1 for e in sp]


def _in_out_elements(case):
    x = case["n"] * case["c"] * case["d"] * case["h"] * case["w"]
    out = _out_extents(case)
    if case["pool"]:
        out = [e // 2 for e in out]
    return x, case["n"] * case["k"] * math.prod(out)


def _flops(case):
    return 2.0 * case["n"] * case["k"] * case["c"] * case["kernel"] ** case["nd"] * math.prod(_out_extents(case))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(shape, dtype, gen):
    """Images in [0, 1) for a first layer, rectified normal values behind one."""
    if shape[1] < 8:
        return torch.rand(shape, generator=gen, device="cuda").to(dtype)
    return torch.randn(shape, generator=gen, device="cuda").clamp_min_(0).to(dtype)


def _kaiming(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda") * math.sqrt(2.0 / math.prod(shape[1:]))


def prepare(case, seed):
    gen = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "stack":
        weights = [_kaiming((k, c, 3, 3), gen).to(dtype) for c, k in engine.VGG16_CHANNELS]
        stack = engine.VGG16ConvStack(weights, case["n"], case["h"], case["w"])
        x = torch.rand((case["n"], case["h"], case["w"], 3), generator=gen, device="cuda").to(dtype)
        if case["graph"]:
            stack.capture(x)
        return {"kind": "stack", "stack": stack, "x": x, "graph": case["graph"]}
    nd, r, s = case["nd"], case["kernel"], case["stride"]
    sp = [case["d"], case["h"], case["w"]][3 - nd:]
    x = _activations((case["n"], case["c"], *sp), dtype, gen)
    if case["channels_last"]:
        x = x.contiguous(memory_format=torch.channels_last if nd == 2 else torch.channels_last_3d)
    weight = _kaiming((case["k"], case["c"], *([r] * nd)), gen)
    bias = torch.randn(case["k"], generator=gen, device="cuda") * 0.1 if case["bias"] else None
    if case["kind"] == "call":
        if case["dtype"] == "f32":
            op = dwm.dwm2d if nd == 2 else dwm.dwm3d
        else:
            op = matrix_conv.conv16 if nd == 2 else matrix_conv3d.conv16
        return {"kind": "call", "op": op, "x": x, "weight": weight, "bias": bias, "stride": (s,) * nd, "padding": (r // 2,) * nd}
    module_type = conv.Conv2d if nd == 2 else conv.Conv3d
    options = {"pool": 2} if case["pool"] else {}
    module = module_type(case["c"], case["k"], r, stride=s, padding=r // 2, bias=case["bias"], device="cuda",
                         compute_dtype=dtype, activation="relu" if case["relu"] else None, **options)
    with torch.no_grad():
        module.weight.copy_(weight)
        if bias is not None:
            module.bias.copy_(bias)
    if case["kind"] == "infer":
        return {"kind": "infer", "module": module.eval(), "x": x}
    gy = torch.randn((case["n"], case["k"], *_out_extents(case)), generator=gen, device="cuda").to(dtype)
    gy = gy.contiguous(memory_format=torch.channels_last if nd == 2 else torch.channels_last_3d)
    return {"kind": "train", "module": module.train(), "x": x.requires_grad_(True), "gy": gy}


def run(state):
    kind = state["kind"]
    if kind == "infer":
        with torch.no_grad():
            return state["module"](state["x"])
    if kind == "call":
        return state["op"](state["x"], state["weight"], state["bias"], stride=state["stride"], padding=state["padding"])
    if kind == "stack":
        return state["stack"].replay(state["x"]) if state["graph"] else state["stack"](state["x"])
    module, x = state["module"], state["x"]
    x.grad = None
    module.zero_grad(set_to_none=True)
    y = module(x)
    y.backward(state["gy"])
    with torch.no_grad():
        for p in module.parameters():
            p.add_(p.grad, alpha=-LEARNING_RATE)
    return {"y": y.detach(), "grad_x": x.grad, "grad": [p.grad for p in module.parameters()],
            "parameters": [p.detach() for p in module.parameters()]}


def work(case):
    """Direct-convolution multiply-adds x 2 (a Winograd pass does fewer), each input read and each output written once."""
    element = 4 if case["dtype"] == "f32" else 2
    if case["kind"] == "stack":
        flops = elements = 0
        h, w = case["h"], case["w"]
        for i, (c, k) in enumerate(engine.VGG16_CHANNELS):
            flops += 2.0 * case["n"] * k * c * 9 * h * w
            elements += k * c * 9 + case["n"] * c * h * w
            if i in engine.VGG16_POOL_AFTER:
                h, w = h // 2, w // 2
            elements += case["n"] * k * h * w
        return {"bytes": float(element * elements), "flops": flops}
    x, y = _in_out_elements(case)
    weights = case["k"] * case["c"] * case["kernel"] ** case["nd"]
    flops = _flops(case)
    if case["kind"] == "infer":
        return {"bytes": float(element * (x + y + weights)), "flops": flops}
    if case["kind"] == "call":
        return {"bytes": float(element * x + 4 * (y + weights)), "flops": flops}
    # x, grad_y in, y, grad_x out; fp32 weights read, their gradient written, the update read and written
    return {"bytes": float(element * 2 * (x + y) + 4 * 4 * weights), "flops": 3 * flops}


def tolerance(case):
    """Relative 2-norm error of another correct implementation at the same precision.

    16-bit operands and results: a Winograd transform rounds its transformed operands to the 16-bit type once more, so
    two implementations with different tilings differ by one to three units of its rounding (2**-11, 2**-8); a stack of
    13 layers by about the square root of 13 times that.  fp32: sums of up to some ten thousand products."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    rel = 2e-3 if case["dtype"] == "f16" else 1.5e-2
    return {"rel": min(0.03, rel * 3)} if case["kind"] == "stack" else {"rel": rel}
