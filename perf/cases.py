"""Performance cases of the library: what its users have it do, through the Python mirror of the C ABI.

Three kinds of work:
  conv     one forward call of a convolution plan (``ConvPlan.launch`` / ``launch_fused``) on tensors in device memory;
  rmsnorm  one ``rmsnorm_forward`` call, plain or with the residual add;
  chain    one pass of the ResNet-50-shaped ``ConvChain``, launch by launch (``enqueue``) or as a replayed CUDA graph.
Plans, workspaces, converted weights and captured graphs are what a program keeps between calls, so ``prepare`` makes
them; ``run`` is the call itself."""
import importlib
import math

import torch

from __graft_entry__ import load_package

gie = load_package()
chain_module = importlib.import_module(gie.__name__ + ".chain")

PRECISIONS = {"fp32": gie.FP32, "fp16": gie.FP16, "bf16": gie.BF16, "tf32": gie.TF32, "fp8": gie.FP8_E4M3}
STORAGE = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16, "tf32": torch.float32, "fp8": torch.float8_e4m3fn}
RESULT = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16, "tf32": torch.float32, "fp8": torch.float16}
RMSNORM_TYPES = {"fp32": 0, "fp16": 1, "bf16": 2}


def conv(name, precision, batch, channels, height, width, filters, kernel, stride=1, layout="nchw", residual=False, prepacked=False):
    case = {"kind": "conv", "precision": precision, "batch": batch, "channels": channels, "height": height, "width": width,
            "filters": filters, "kernel": kernel, "stride": stride, "layout": layout, "residual": residual, "prepacked": prepacked}
    return dict(case, name=name) if name else case


def rmsnorm(name, dtype, rows, hidden, residual):
    case = {"kind": "rmsnorm", "dtype": dtype, "rows": rows, "hidden": hidden, "residual": residual}
    return dict(case, name=name) if name else case


def chain(name, precision, batch, image, layout, graph):
    case = {"kind": "chain", "precision": precision, "batch": batch, "image": image, "layout": layout, "graph": graph}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one layer of a mid-size network at a serving batch, everything as the operator API has it: NCHW tensors, OIHW weights
        conv("conv fp16 3x3 14x14 b32", "fp16", 32, 256, 14, 14, 256, 3),
        # a single image through a deep 3x3 layer: few output pixels, long reduction, launch latency
        conv("conv fp16 3x3 7x7 b1", "fp16", 1, 512, 7, 7, 512, 3),
        # a channel-reducing pointwise layer: bound by reading its input once
        conv("conv bf16 1x1 28x28 b64", "bf16", 64, 512, 28, 28, 128, 1),
        # a down-sampling layer
        conv("conv fp16 3x3/2 56x56 b16", "fp16", 16, 128, 56, 56, 256, 3, stride=2),
        # a residual layer between channel-contiguous tensors with sizes that fit no tile: odd maps, ragged channels
        conv("conv bf16 ragged nhwc residual", "bf16", 6, 144, 35, 45, 200, 3, layout="nhwc", residual=True, prepacked=True),
        # strict FP32 for a single image
        conv("conv fp32 3x3 56x56 b1", "fp32", 1, 64, 56, 56, 64, 3),
        # FP32 tensors on the tensor cores, an odd map and a wide kernel
        conv("conv tf32 5x5 27x27 b16", "tf32", 16, 96, 27, 27, 192, 5),
        # quantised inputs
        conv("conv fp8 3x3 14x14 b32", "fp8", 32, 256, 14, 14, 256, 3),
        # a decoding step's normalisation: a handful of tokens
        rmsnorm("rmsnorm bf16 16x4096", "bf16", 16, 4096, True),
        # the same over a prompt or a training batch
        rmsnorm("rmsnorm bf16 8192x4096", "bf16", 8192, 4096, True),
        # a whole network over a small batch, launched layer by layer on the operator API's tensor contract
        chain("chain fp16 nchw b4", "fp16", 4, 224, "nchw", False),
        # a whole network at full batch, captured as one graph, in the layout made for chains
        chain("chain fp16 nhwc b256", "fp16", 256, 224, "nhwc", True),
    ]


def between(rng, low, high):
    """A whole number, its logarithm spread evenly."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def channel_count(rng, low, high):
    """Mostly the multiples of 64 or 16 that networks have, now and then any number."""
    c = between(rng, low, high)
    unit = rng.choice([1, 16, 64, 64])
    return max(unit, (c + unit // 2) // unit * unit)


def draw(rng):
    kind = rng.choice(["conv"] * 7 + ["rmsnorm"] * 2 + ["chain"])
    if kind == "rmsnorm":
        while True:
            rows, hidden = between(rng, 1, 16384), between(rng, 128, 16384)
            unit = rng.choice([1, 64, 64, 256])
            hidden = max(unit, hidden // unit * unit)
            if rows * hidden <= 1 << 26:
                return rmsnorm(None, rng.choice(["bf16", "bf16", "fp16", "fp32"]), rows, hidden, rng.random() < 0.7)
    if kind == "chain":
        return chain(None, rng.choice(["fp16", "bf16"]), between(rng, 1, 128), rng.choice([128, 160, 192, 224, 256]),
                     rng.choice(["nchw", "nhwc"]), rng.random() < 0.6)
    while True:
        precision = rng.choice(["fp16"] * 4 + ["bf16"] * 3 + ["fp32", "tf32", "fp8"])
        if rng.random() < 0.1 and precision in ("fp16", "bf16"):  # a first layer over images
            side = between(rng, 64, 256) // 2 * 2
            return conv(None, precision, between(rng, 1, 64), 3, side, side, 64, 7, stride=2)
        kernel = rng.choice([1, 1, 3, 3, 3, 5])
        stride = rng.choice([1, 1, 1, 2])
        height = between(rng, 7, 112)
        width = height if rng.random() < 0.6 else between(rng, 7, 112)
        channels, filters = channel_count(rng, 16, 1024), channel_count(rng, 16, 1024)
        batch = between(rng, 1, 256)
        layout, residual, prepacked = "nchw", False, False
        if precision in ("fp16", "bf16"):
            residual, prepacked = rng.random() < 0.25, rng.random() < 0.4
            layout = "nhwc" if channels % 16 == 0 and rng.random() < 0.4 else "nchw"
        case = conv(None, precision, batch, channels, height, width, filters, kernel, stride, layout, residual, prepacked)
        w = work(case)
        if 1e7 <= w["flops"] <= (2e10 if precision == "fp32" else 3e11) and w["bytes"] <= 8e8:
            return case


def out_size(case):
    pad = case["kernel"] // 2
    return ((case["height"] + 2 * pad - case["kernel"]) // case["stride"] + 1, (case["width"] + 2 * pad - case["kernel"]) // case["stride"] + 1)


def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def uniform(n, bound, g):
    return (torch.rand(n, device="cuda", generator=g) * 2 - 1) * bound


def prepare(case, seed):
    g = generator(seed)
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "rmsnorm":
        dtype = STORAGE[case["dtype"]]
        shape = (case["rows"], case["hidden"])
        x = torch.randn(shape, device="cuda", generator=g).to(dtype)
        gamma = (1 + 0.02 * torch.randn(case["hidden"], device="cuda", generator=g)).to(dtype)
        state = {"case": case, "stream": stream, "x": x, "gamma": gamma, "y": torch.empty_like(x)}
        if case["residual"]:
            state["residual"] = torch.randn(shape, device="cuda", generator=g).to(dtype)
            state["residual_out"] = torch.empty_like(x)
        return state
    if case["kind"] == "chain":
        c = chain_module.ConvChain(case["batch"], PRECISIONS[case["precision"]], case["image"], seed=seed, layout=case["layout"])
        c.input.copy_(torch.randn(c.input.numel(), device="cuda", generator=g))
        if case["graph"]:
            c.capture(torch.cuda.Stream())
        return {"case": case, "stream": stream, "chain": c}
    k = case["kernel"]
    storage, result = STORAGE[case["precision"]], RESULT[case["precision"]]
    nhwc = case["layout"] == "nhwc"
    flags = (gie.FLAG_INPUT_NHWC | gie.FLAG_OUTPUT_NHWC if nhwc else 0) | (gie.FLAG_RESIDUAL if case["residual"] else 0) \
        | (gie.FLAG_WEIGHTS_PREPACKED if case["prepacked"] else 0)
    problem = gie.ConvProblem(case["batch"], case["channels"], case["height"], case["width"], case["filters"], k, k, case["stride"],
                              case["stride"], k // 2, k // 2, precision=PRECISIONS[case["precision"]], has_bias=True, relu=True, flags=flags)
    plan = gie.ConvPlan(problem)
    fan_in = case["channels"] * k * k
    x = torch.randn(case["batch"] * case["channels"] * case["height"] * case["width"], device="cuda", generator=g)
    if case["channels"] > 4:
        x = torch.relu_(x)  # what the layer before it hands on; a first layer sees images
    x = x.to(storage)
    # (an 8-bit weight tensor is stored scaled to use its range)
    w = uniform(case["filters"] * fan_in, 1.0 if case["precision"] == "fp8" else math.sqrt(6.0 / fan_in), g).to(storage)
    bias = uniform(case["filters"], 0.1, g).to(torch.float32 if case["precision"] == "fp8" else storage)
    if case["prepacked"]:
        packed = torch.empty(plan.prepacked_weight_bytes, dtype=torch.uint8, device="cuda")
        plan.prepack_weights(w.data_ptr(), packed.data_ptr(), stream)
        w = packed
    p, q = out_size(case)
    shape = (case["batch"], p, q, case["filters"]) if nhwc else (case["batch"], case["filters"], p, q)
    y = torch.empty(shape, dtype=result, device="cuda")
    workspace = torch.empty(max(plan.workspace_bytes, 256), dtype=torch.uint8, device="cuda")  # (torch's blocks are 512-byte aligned)
    state = {"case": case, "stream": stream, "plan": plan, "x": x, "w": w, "bias": bias, "y": y, "workspace": workspace}
    if case["residual"]:
        state["residual"] = torch.randn(shape, device="cuda", generator=g).to(result)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "conv":
        plan, y, ws = state["plan"], state["y"], state["workspace"]
        if "residual" in state:
            plan.launch_fused(state["x"].data_ptr(), state["w"].data_ptr(), state["bias"].data_ptr(), state["residual"].data_ptr(), y.data_ptr(),
                              ws.data_ptr(), ws.numel(), state["stream"])
        else:
            plan.launch(state["x"].data_ptr(), state["w"].data_ptr(), state["bias"].data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(),
                        state["stream"])
        return y
    if kind == "rmsnorm":
        c = state["case"]
        if c["residual"]:
            gie.rmsnorm_forward(c["rows"], c["hidden"], 1e-6, RMSNORM_TYPES[c["dtype"]], state["x"].data_ptr(), state["gamma"].data_ptr(),
                                state["y"].data_ptr(), state["residual"].data_ptr(), state["residual_out"].data_ptr(), stream=state["stream"])
            return state["y"], state["residual_out"]
        gie.rmsnorm_forward(c["rows"], c["hidden"], 1e-6, RMSNORM_TYPES[c["dtype"]], state["x"].data_ptr(), state["gamma"].data_ptr(),
                            state["y"].data_ptr(), stream=state["stream"])
        return state["y"]
    network = state["chain"]
    if state["case"]["graph"]:
        network.replay()
    else:
        network.enqueue(state["stream"])
    return network.output


def chain_shapes(case):
    """(layer shapes, output elements) of a chain without building it."""
    ops, slots = chain_module.resnet50_chain(case["batch"], PRECISIONS[case["precision"]], case["image"])
    c, h, w = slots[len(slots) - 1]
    return [op.shape for op in ops if op.kind == "conv"], case["batch"] * c * h * w


def work(case):
    if case["kind"] == "rmsnorm":
        size = torch.empty(0, dtype=STORAGE[case["dtype"]]).element_size()
        n = case["rows"] * case["hidden"]
        return {"bytes": ((4 if case["residual"] else 2) * n + case["hidden"]) * size, "flops": (5 if case["residual"] else 4) * n}
    if case["kind"] == "chain":
        # the image and the weights in, the last tensor out; what lies between belongs to the way it is computed
        shapes, out = chain_shapes(case)
        weights = sum(s.w_elems + s.out_channels for s in shapes)
        return {"bytes": 2 * (shapes[0].x_elems + weights + out), "flops": sum(s.flops for s in shapes)}
    p, q = out_size(case)
    k = case["kernel"]
    size = torch.empty(0, dtype=STORAGE[case["precision"]]).element_size()
    size_out = torch.empty(0, dtype=RESULT[case["precision"]]).element_size()
    # a pointwise layer with a stride reads only the pixels it lands on
    pixels = p * q if k == 1 else case["height"] * case["width"]
    x = case["batch"] * case["channels"] * pixels
    w = case["filters"] * case["channels"] * k * k
    y = case["batch"] * case["filters"] * p * q
    return {"bytes": (x + w) * size + y * size_out * (2 if case["residual"] else 1) + case["filters"] * (4 if case["precision"] == "fp8" else size),
            "flops": 2 * y * case["channels"] * k * k}


def tolerance(case):
    """One rounding to the output's type where sums are taken in FP32 in another order; a chain carries 53 of them."""
    if case["kind"] == "chain":
        return {"rel": 5e-3 if case["precision"] == "fp16" else 2.5e-2}
    kind = case["dtype"] if case["kind"] == "rmsnorm" else case["precision"]
    # TF32 multiplies 11-bit values exactly and sums them in FP32, as many as the reduction is long
    return {"rel": {"fp32": 1e-5, "tf32": 5e-5, "fp16": 1e-3, "fp8": 1e-3, "bf16": 1e-2}[kind]}
