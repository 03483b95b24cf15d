"""The work this framework is used for, as cases to time: int8 fc, conv2d, depthwise_conv2d and sparse_conv2d layers
called one by one, and the two whole networks.

`listed()` gives the fixed cases, `draw(rng)` more of the same ranges; `prepare` builds what a program holds before it
calls (prepared layers, device tensors), `run` is one pass through the package's public calls.
"""
import functools
import importlib
import math

import numpy as np
import torch

plb = importlib.import_module("paddle-lite_b200")
networks = importlib.import_module("paddle-lite_b200.networks")
sparse_format = importlib.import_module("paddle-lite_b200.sparse_format")

ACTS = {"none": plb.ACT_NONE, "relu": plb.ACT_RELU, "relu6": plb.ACT_RELU6, "leaky": plb.ACT_LEAKY}
ALPHA = {"none": 0.0, "relu": 0.0, "relu6": 6.0, "leaky": 0.1}
ACT_SCALE = 4.0 / 127  # int8 activations: real values of about unit variance, clipped at four deviations
NET_SCALE = {"resnet50": (4.09e9, 25.6e6), "mobilenet_v1": (0.57e9, 4.2e6)}  # multiply-adds per image, weights


def listed():
    return [
        # classifier head of a network run on one image: the smallest call, latency only
        dict(name="fc_one_row", kind="fc", m=1, k=2048, n=1000, act="none", out="f32"),
        # a hidden layer at a serving batch
        dict(name="fc_256", kind="fc", m=256, k=4096, n=4096, act="relu6", out="f32"),
        # large fully-connected layer with requantised output: the tensor-core bound end
        dict(name="fc_4096", kind="fc", m=4096, k=4096, n=4096, act="relu6", out="i8"),
        # one 3x3 layer on one image in the layout of the reference's kernels, dequantised output
        dict(name="conv3x3_one_image", kind="conv", batch=1, cin=64, cout=64, h=56, w=56, k=3, stride=1, act="relu",
             out="f32", layout="nchw"),
        # an ordinary 3x3 layer of a batch in the same layout
        dict(name="conv3x3_nchw", kind="conv", batch=64, cin=128, cout=128, h=28, w=28, k=3, stride=1, act="relu",
             out="i8", layout="nchw"),
        # sizes that fit nothing: channels and pixels that are no multiples of a tile or of a vector
        dict(name="conv3x3_ragged", kind="conv", batch=9, cin=75, cout=100, h=61, w=45, k=3, stride=2, act="leaky",
             out="i8", layout="nchw"),
        # a depthwise layer of a mobile network, channels-last as between int8 layers
        dict(name="depthwise", kind="dw", batch=128, c=128, h=56, w=56, k=3, stride=1, act="relu", out="i8",
             layout="nhwc"),
        # pruned pointwise layers (four of five weights zero), both precisions
        dict(name="sparse_i8", kind="sparse", dtype="i8", batch=256, cin=512, cout=512, h=14, w=14, density=0.2,
             semi=False, act="relu", out="i8"),
        dict(name="sparse_f32", kind="sparse", dtype="f32", batch=256, cin=128, cout=128, h=56, w=56, density=0.2,
             semi=False, act="relu", out="f32"),
        # whole networks from fp32 images to logits: one image, a small batch, a full batch
        dict(name="resnet50_1", kind="net", net="resnet50", batch=1),
        dict(name="mobilenet_v1_32", kind="net", net="mobilenet_v1", batch=32),
        dict(name="resnet50_128", kind="net", net="resnet50", batch=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, lo, hi, step):
    """A size of the range: half of them multiples of `step`, half any."""
    v = _log(rng, lo, hi)
    return min(hi, max(lo, (v + step // 2) // step * step)) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["fc", "conv", "conv", "dw", "sparse", "net"])
    act = rng.choice(["none", "relu", "relu", "relu6", "leaky"])
    out = rng.choice(["i8", "f32"])
    if kind == "net":
        net = rng.choice(sorted(NET_SCALE))
        return dict(kind=kind, net=net, batch=_log(rng, 1, 128 if net == "resnet50" else 256))
    if kind == "fc":
        k = _ragged(rng, 512, 4096, 32) // 4 * 4  # rows of whole words: what the layer takes
        return dict(kind=kind, m=_log(rng, 1, 4096), k=k, n=_ragged(rng, 100, 4096, 16), act=act, out=out)
    h = _log(rng, 7, 112)
    w = h if rng.random() < 0.6 else min(112, max(7, int(h * rng.uniform(0.6, 1.6))))
    if kind == "conv":
        k, stride = rng.choice([1, 3, 3, 5]), rng.choice([1, 1, 2])
        layout = rng.choice(["nchw", "nchw", "nhwc"])
        cin, cout = _ragged(rng, 16, 512, 32), _ragged(rng, 16, 512, 32)
        if layout == "nhwc":
            cin = max(32, cin // 32 * 32)  # channels-last tensors come in rows of whole 32-byte groups
        c = dict(kind=kind, batch=_log(rng, 1, 128), cin=cin, cout=cout, h=h, w=w, k=k, stride=stride, act=act, out=out,
                 layout=layout)
    elif kind == "dw":
        layout = rng.choice(["nhwc", "nhwc", "nchw"])
        ch = _ragged(rng, 16, 1024, 32)
        if layout == "nhwc":
            ch = ch // 16 * 16
        c = dict(kind=kind, batch=_log(rng, 1, 256), c=ch, h=h, w=w, k=rng.choice([3, 3, 3, 5]),
                 stride=rng.choice([1, 1, 2]), act=act, out=out, layout=layout)
    else:
        dtype = rng.choice(["i8", "f32"])
        c = dict(kind=kind, dtype=dtype, batch=_log(rng, 1, 256), cin=_ragged(rng, 32, 1024, 32),
                 cout=_ragged(rng, 32, 1024, 32), h=h, w=w, density=round(rng.uniform(0.1, 0.3), 2),
                 semi=rng.random() < 0.4, act=act, out="f32" if dtype == "f32" else out)
    # no larger than the largest listed layers of the kind
    most_bytes, most_flops = (850e6, 6e9) if kind == "sparse" else (420e6, 150e9)
    while c["batch"] > 1 and (work(c)["bytes"] > most_bytes or work(c)["flops"] > most_flops):
        c["batch"] = (c["batch"] + 1) // 2
    return c


def _out_hw(case):
    p = case["k"] // 2
    return tuple((case[d] + 2 * p - case["k"]) // case["stride"] + 1 for d in "hw")


def work(case):
    kind = case["kind"]
    if kind == "net":  # images in, weights once, logits out
        macs, weights = NET_SCALE[case["net"]]
        return {"bytes": case["batch"] * (3 * 224 * 224 + 1000) * 4 + weights, "flops": 2 * macs * case["batch"]}
    eb = 1 if case["out"] == "i8" else 4
    if kind == "fc":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": m * k + k * n + m * n * eb + 8 * n, "flops": 2 * m * k * n}
    if kind == "sparse":
        cin, cout, pix = case["cin"], case["cout"], case["batch"] * case["h"] * case["w"]
        xb, nnz = (1 if case["dtype"] == "i8" else 4), int(cin * cout * case["density"])
        return {"bytes": pix * (cin * xb + cout * eb) + nnz * (xb + 4) + 8 * cout, "flops": 2 * nnz * pix}
    ho, wo = _out_hw(case)
    cin, cout, taps = case.get("cin", case.get("c")), case.get("cout", case.get("c")), case["k"] ** 2
    per_out = taps * (cin if kind == "conv" else 1)
    return {"bytes": case["batch"] * (case["h"] * case["w"] * cin + ho * wo * cout * eb) + cout * per_out + 8 * cout,
            "flops": 2 * case["batch"] * ho * wo * cout * per_out}


def tolerance(case):
    # int8 results come from exact integer sums and one rounding; fp32 results from exact integer sums and one fused
    # multiply-add (int8 layers) or from fp32 sums (sparse fp32 layers)
    return {"rel": 1e-5} if case["kind"] == "net" or case["out"] == "f32" else "exact"


@functools.lru_cache(maxsize=None)
def _model(net):
    """The quantised network a program has loaded: fixed weights; activation scales to seven bits, so that they do not
    depend on the order in which the calibration pass sums."""
    q = networks.build_quantized(networks.SPECS[net](), seed=1234, calib_images=4, device="cuda")
    scales = {}
    for name, s in q["scales"].items():
        m, e = math.frexp(float(s))
        scales[name] = np.float32(math.ldexp(round(m * 128) / 128, e))
    return dict(q, scales=scales)


def _activations(shape, gen):
    """int8 activations behind a ReLU."""
    x = torch.randn(shape, generator=gen, device="cuda").clamp_(min=0).mul_(1 / ACT_SCALE).round_().clamp_(max=127)
    return x.to(torch.int8)


def _per_channel(w):
    q, ws = sparse_format.quantize_per_channel(w.reshape(w.shape[0], -1))
    return q.reshape(w.shape), ws


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    ctx = plb.Context(0)
    state = {"kind": kind, "ctx": ctx}
    if kind == "net":
        state["runner"] = networks.Runner(plb, ctx, _model(case["net"]), case["batch"])
        state["x"] = torch.randn(state["runner"].image_shape, generator=gen, device="cuda")
        return state
    act, alpha, i8 = ACTS[case["act"]], ALPHA[case["act"]], case["out"] == "i8"
    dt = torch.int8 if i8 else torch.float32
    if kind == "fc":
        m, k, n = case["m"], case["k"], case["n"]
        wt, ws = _per_channel(rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
        bias = rng.standard_normal(n).astype(np.float32) * np.float32(0.1)
        std = 0.02 * math.sqrt(k / 3)
        state["layer"] = plb.Fc(ctx, np.ascontiguousarray(wt.T), ws, 1 / 127, bias, act, alpha,
                                out_scale=4 * std / 127 if i8 else None)
        state["x"] = torch.randint(-127, 128, (m, k), generator=gen, device="cuda", dtype=torch.int8)
        state["y"] = torch.empty((m, n), dtype=dt, device="cuda")
        return state
    h, w = case["h"], case["w"]
    if kind == "sparse":
        cin, cout = case["cin"], case["cout"]
        wf = rng.standard_normal((cout, cin), dtype=np.float32) * np.float32(math.sqrt(2 / (cin * case["density"])))
        if case["semi"]:  # pairs of output channels share their zeros
            mask = np.repeat(rng.random(((cout + 1) // 2, cin)) < case["density"], 2, axis=0)[:cout]
        else:
            mask = rng.random((cout, cin)) < case["density"]
        wf = wf * mask
        bias = rng.standard_normal(cout).astype(np.float32) * np.float32(0.1)
        scales = {}
        if case["dtype"] == "i8":
            wf, ws = sparse_format.quantize_per_channel(wf)
            scales = dict(wscale=ws, in_scale=ACT_SCALE, out_scale=ACT_SCALE if i8 else None)
            state["x"] = _activations((case["batch"], cin, h, w), gen)
        else:
            state["x"] = torch.randn((case["batch"], cin, h, w), generator=gen, device="cuda").clamp_(min=0)
        e = sparse_format.encode(wf, h * w, semi=case["semi"])
        state["layer"] = plb.SparseConv(ctx, e["nonzero_weights"], e["oc_nonzeros"], e["diffs"], e["first_ic"],
                                        e["flag_semi"], cin=cin, cout=cout, in_hw=(h, w), bias=bias, act=act,
                                        alpha=alpha, **scales)
        state["y"] = torch.empty((case["batch"], cout, h, w), dtype=dt, device="cuda")
        return state
    k, nhwc = case["k"], case["layout"] == "nhwc"
    cin, cout = case.get("cin", case.get("c")), case.get("cout", case.get("c"))
    groups = cin if kind == "dw" else 1
    wf = rng.standard_normal((cout, cin // groups, k, k), dtype=np.float32)
    wq, ws = _per_channel(wf * np.float32(math.sqrt(2 / (cin // groups * k * k))))
    bias = rng.standard_normal(cout).astype(np.float32) * np.float32(0.1)
    state["layer"] = plb.Conv(ctx, wq, ws, ACT_SCALE, bias, in_hw=(h, w), stride=(case["stride"],) * 2,
                              pads=(k // 2,) * 4, groups=groups, act=act, alpha=alpha,
                              out_scale=ACT_SCALE if i8 else None)
    ho, wo = _out_hw(case)
    state["nhwc"] = nhwc
    state["x"] = _activations((case["batch"], h, w, cin) if nhwc else (case["batch"], cin, h, w), gen)
    state["y"] = torch.empty((case["batch"], ho, wo, cout) if nhwc else (case["batch"], cout, ho, wo), dtype=dt,
                             device="cuda")
    return state


def run(state):
    if state["kind"] == "net":
        return state["runner"].forward(state["x"])
    if state.get("nhwc"):
        return state["layer"].run_nhwc(state["x"], out=state["y"])
    return state["layer"].run(state["x"], out=state["y"])
