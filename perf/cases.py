"""Performance cases of the convolution library, through its public Python
entry points (each a thin veneer over the C ABI).

Kinds:

* ``dropin``    the plugin ABI of include/conv2d.h as the reference harness
                drives it: getParamsize, getkernelInfo, the four launch slots,
                weights untransformed on every call, caller-owned workspaces.
                Any filter / stride / padding it accepts.
* ``epilogue``  inference with a transformed filter kept across calls: conv +
                bias + residual + ReLU in one call, as a ResNet block needs it.
* ``variant``   one conv with another precision of the GEMM stage, everything
                per call.
* ``batch``     the uneven layers of a network stage replayed as one CUDA
                graph.

Sizes are those of the repository's own workloads (bench.py, tests/): the small
layer N8 C64 H32 K64, the large layer N128 C256 H28 K256, the precision-sweep
layer N64 C256 H14 K256, the ResNet-50 layers of bench.py's implicit-GEMM leg,
the 12-layer set, and the cost model's shape space (N 1 to 128, channels 16 to
1024 with multiples of 48, H and W 7 to 112) for the drawn ones.
"""
import importlib

import torch

wino = importlib.import_module("2024pra_conv_b200")

# Direct-conv FLOPs of the largest listed case: no drawn case exceeds them.
MAX_FLOPS = 2.0 * 128 * 256 * 28 * 28 * 256 * 9
# ... nor its input + output elements by more than this.
MAX_ELEMS = 2.0 * 128 * 256 * 28 * 28 * 1.6


def _dropin(name, n, c, h, w, k, r=3, stride=1, pad=1):
    return {"name": name, "kind": "dropin", "n": n, "c": c, "h": h, "w": w, "k": k, "r": r,
            "stride": stride, "pad": pad}


def listed():
    return [
        # one image through a late-stage layer: interactive inference, where
        # launches and the length of the reduction count, not throughput
        _dropin("dropin n1 c256 14x14", 1, 256, 14, 14, 256),
        # the small layer of the tests and of the reference-style harness
        _dropin("dropin n8 c64 32x32", 8, 64, 32, 32, 64),
        # the precision-sweep layer: a mid-network batch
        _dropin("dropin n64 c256 14x14", 64, 256, 14, 14, 256),
        # bench.py's single large layer
        _dropin("dropin n128 c256 28x28", 128, 256, 28, 28, 256),
        # last ResNet stage: odd image, many channels
        _dropin("dropin n32 c512 7x7", 32, 512, 7, 7, 512),
        # ragged: odd height and width, channels that are multiples of 48
        _dropin("dropin n8 c48 45x61 k144", 8, 48, 45, 61, 144),
        # downsampling 3x3 between stages (outside the Winograd contract)
        _dropin("dropin 3x3 s2 n32 c128", 32, 128, 56, 56, 128, stride=2),
        # bottleneck expansion 1x1
        _dropin("dropin 1x1 n32 c64 k256", 32, 64, 56, 56, 256, r=1, pad=0),
        # network stem: 7x7 stride 2 over RGB images
        _dropin("dropin 7x7 s2 n32 c3", 32, 3, 224, 224, 64, r=7, stride=2, pad=3),
        # residual block inference: filter transformed once, conv + bias +
        # residual + ReLU per call
        {"name": "epilogue n32 c128 28x28", "kind": "epilogue", "n": 32, "c": 128, "h": 28, "w": 28, "k": 128},
        # bf16 GEMM stage on the precision-sweep layer
        {"name": "variant bf16 n64 c256 14x14", "kind": "variant", "variant": "bf16", "n": 64, "c": 256,
         "h": 14, "w": 14, "k": 256},
        # the 12 uneven ResNet layers as one graph replay
        {"name": "batch resnet set n32", "kind": "batch", "n": 32, "first": 0, "count": 12, "odd": 0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _chan(rng, lo=16, hi=1024):
    """Channels: a power of two or a multiple of 48, log-uniform."""
    if rng.random() < 0.5:
        p = 16
        ps = []
        while p <= hi:
            if p >= lo:
                ps.append(p)
            p *= 2
        return rng.choice(ps)
    return max(lo, _log_int(rng, max(48, lo), min(hi, 960)) // 48 * 48)


def _elems(case):
    st = case.get("stride", 1)
    return case["n"] * (case["c"] * case["h"] * case["w"] + case["k"] * case["h"] * case["w"] / (st * st))


def draw(rng):
    while True:
        kind = rng.choices(["dropin", "general", "epilogue", "variant", "batch"], [10, 6, 3, 2, 2])[0]
        if kind == "batch":
            # a run of the layer set at another batch size; "odd" adds to each H and W
            return {"kind": "batch", "n": _log_int(rng, 1, 32), "first": rng.randrange(0, 8),
                    "count": rng.randrange(2, 5), "odd": rng.choice([0, 0, 1, 2])}
        n = _log_int(rng, 1, 128)
        h = _log_int(rng, 7, 112)
        w = h if rng.random() < 0.6 else _log_int(rng, 7, 112)
        case = {"kind": kind, "n": n, "c": _chan(rng), "h": h, "w": w, "k": _chan(rng)}
        if kind == "general":
            case["kind"] = "dropin"
            f = rng.choice(["3s2", "3s2", "1s1", "1s1", "1s2", "7s2"])
            if f == "3s2":
                case.update(r=3, stride=2, pad=1)
            elif f == "7s2":
                side = _log_int(rng, 64, 256)
                case.update(n=min(n, 32), c=3, h=side, w=side, k=rng.choice([32, 64, 96]), r=7, stride=2, pad=3)
            else:
                case.update(r=1, stride=int(f[2]), pad=0)
        elif kind == "dropin":
            case.update(r=3, stride=1, pad=1)
        elif kind == "variant":
            case["variant"] = rng.choice(["bf16", "f16", "f16_hilo", "f8"])
            if case["variant"] == "f8":
                case["c"] = (case["c"] + 31) // 32 * 32
        if _direct_flops(case) <= MAX_FLOPS and _elems(case) <= MAX_ELEMS:
            return case


def _out_hw(case):
    r, st, pad = case.get("r", 3), case.get("stride", 1), case.get("pad", 1)
    return (case["h"] - r + 2 * pad) // st + 1, (case["w"] - r + 2 * pad) // st + 1


def _direct_flops(case):
    oh, ow = _out_hw(case)
    return 2.0 * case["n"] * case["k"] * oh * ow * case["c"] * case.get("r", 3) ** 2


def _batch_layers(case):
    picks = wino.RESNET_LAYER_SET[case["first"]:case["first"] + case["count"]]
    return [{"kind": "layer", "n": case["n"], "c": c, "h": h + case["odd"], "w": h + case["odd"], "k": k}
            for (c, k, h) in picks]


def work(case):
    """Bytes: input, weights, output (bias and residual) once each, fp16.
    FLOPs: the F(2x2,3x3) multiply-adds for 3x3 / stride 1 / pad 1 (the direct
    count / 2.25, what the library's rooflines are drawn with), the direct
    count otherwise."""
    if case["kind"] == "batch":
        ws = [work(l) for l in _batch_layers(case)]
        return {key: sum(w[key] for w in ws) for key in ("bytes", "flops")}
    n, c, k, r = case["n"], case["c"], case["k"], case.get("r", 3)
    oh, ow = _out_hw(case)
    nbytes = 2.0 * (n * c * case["h"] * case["w"] + k * c * r * r + n * k * oh * ow)
    if case["kind"] == "epilogue":
        nbytes += 2.0 * n * k * oh * ow + 4.0 * k
    wino_shape = r == 3 and case.get("stride", 1) == 1
    return {"bytes": nbytes, "flops": _direct_flops(case) / (2.25 if wino_shape else 1.0)}


def _tensors(case, gen):
    """x: ReLU outputs of the layer before (half zeros; images for the stem);
    weights at He scale."""
    n, c, k, r = case["n"], case["c"], case["k"], case.get("r", 3)
    x = torch.randn((n, c, case["h"], case["w"]), device="cuda", generator=gen)
    x = (x if c == 3 else x.relu_()).half()
    w = (torch.randn((k, c, r, r), device="cuda", generator=gen) * (2.0 / (c * r * r)) ** 0.5).half()
    return x, w


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "batch":
        return [_tensors(l, gen) for l in _batch_layers(case)]
    x, w = _tensors(case, gen)
    if case["kind"] != "epilogue":
        return x, w
    oh, ow = _out_hw(case)
    bias = torch.randn(case["k"], device="cuda", generator=gen) * 0.5
    res = torch.randn((case["n"], case["k"], oh, ow), device="cuda", generator=gen).relu_().half()
    return x, w, bias, res


_VARIANTS = {"f16": wino.VAR_F16, "bf16": wino.VAR_BF16, "f8": wino.VAR_F8, "f16_hilo": wino.VAR_F16_HILO}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b, outs = wino.Batch(), []
        for layer, (x, w) in zip(_batch_layers(case), _inputs(case, seed)):
            ws = torch.empty(wino.fused_workspace_bytes(layer["n"], layer["c"], layer["h"], layer["w"]),
                             dtype=torch.uint8, device="cuda")
            y = torch.empty((layer["n"], layer["k"], layer["h"], layer["w"]), dtype=torch.float16, device="cuda")
            b.add(x, wino.filter_transform(w), layer["k"], y, workspace=ws)
            outs.append(y)
        torch.cuda.synchronize()
        b.capture()
        return {"case": case, "batch": b, "outs": outs}
    n, c, h, w_, k = (case[f] for f in ("n", "c", "h", "w", "k"))
    if kind == "dropin":
        x, w = _inputs(case, seed)
        return {"case": case, "x": x, "w": w, "ws": wino.DropinWorkspaces(n, c, h, w_, k, x.device)}
    if kind == "epilogue":
        x, w, bias, res = _inputs(case, seed)
        ws = torch.empty(wino.fused_workspace_bytes(n, c, h, w_), dtype=torch.uint8, device="cuda")
        return {"case": case, "x": x, "u": wino.filter_transform(w), "bias": bias, "res": res, "ws": ws}
    x, w = _inputs(case, seed)
    ws = torch.empty(wino.variant_workspace_bytes(_VARIANTS[case["variant"]], n, c, h, w_, k) + 256,
                     dtype=torch.uint8, device="cuda")
    return {"case": case, "x": x, "w": w, "ws": ws}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].launch()
        return state["outs"]
    if kind == "dropin":
        return wino.dropin_conv2d(state["x"], state["w"], ws=state["ws"], stride=case["stride"], pad=case["pad"])
    if kind == "epilogue":
        return wino.conv2d_fused_epilogue(state["x"], state["u"], case["k"], bias=state["bias"],
                                          residual=state["res"], relu=True, workspace=state["ws"])
    return wino.conv2d_variant(state["x"], state["w"], _VARIANTS[case["variant"]], workspace=state["ws"])


def _conv64(x, w, stride, pad):
    """FP64 convolution as a sum of shifted channel contractions (plain
    matmuls), a few images at a time to bound memory."""
    n, c, h, w_ = x.shape
    k, _, r, s = w.shape
    oh, ow = (h - r + 2 * pad) // stride + 1, (w_ - s + 2 * pad) // stride + 1
    y = torch.empty((n, k, oh, ow), dtype=torch.float64, device=x.device)
    wd = w.double()
    step = max(1, int(2e8 // (c * h * w_ + (c + 2 * k) * oh * ow)))
    for i in range(0, n, step):
        xp = torch.nn.functional.pad(x[i:i + step].double(), (pad, pad, pad, pad))
        acc = torch.zeros((xp.shape[0], k, oh * ow), dtype=torch.float64, device=x.device)
        for a in range(r):
            for b in range(s):
                win = xp[:, :, a:a + (oh - 1) * stride + 1:stride, b:b + (ow - 1) * stride + 1:stride]
                acc += torch.matmul(wd[:, :, a, b], win.reshape(win.shape[0], c, oh * ow))
        y[i:i + step] = acc.view(-1, k, oh, ow)
    return y


def exact(case, seed):
    if case["kind"] == "batch":
        return [_conv64(x, w, 1, 1) for x, w in _inputs(case, seed)]
    if case["kind"] == "epilogue":
        x, w, bias, res = _inputs(case, seed)
        return torch.relu(_conv64(x, w, 1, 1) + bias.double().view(1, -1, 1, 1) + res.double())
    x, w = _inputs(case, seed)
    return _conv64(x, w, case.get("stride", 1), case.get("pad", 1))
