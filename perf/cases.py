"""The work this library is asked to do, as cases that can be timed and checked.

Every case goes through the public operators of ``cctconv`` (and ``cctconv.graph`` for a
whole stack), the way a program that convolves fields calls them.  ``listed`` names one
case of each kind of call; ``draw`` gives others of the same kinds over the sizes, borders,
samplings and precisions that the kind meets in use.  ``exact`` restates each operator in
FP64 with plain torch.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cct-core_b200"))
import cctconv as C  # noqa: E402
from cctconv import _lib  # noqa: E402
from cctconv.graph import LayerStack  # noqa: E402

BORDERS = {"zero": C.BorderZero, "clamp": C.BorderClamp, "cyclic": C.BorderCyclic,
           "valid": C.BorderValid, "full": C.BorderFull}
PRECISIONS = {"fp32": _lib.PREC_FP32, "bf16x3": _lib.PREC_BF16X3, "bf16x6": _lib.PREC_BF16X6}


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # One 256x256 ScalarField and one 5x5 kernel: the smallest step of a field graph, a
        # call whose latency is what counts.
        plane("plane_5x5_256", 256, 256, 0, 0, 5, "zero", "convolve"),
        # A large VectorField through one small kernel: what a memory-bound smoothing or
        # gradient step over many planes costs.
        plane("planes_5x5_1024x256", 256, 256, 1024, 0, 5, "zero", "convolve"),
        # Frames of an uneven size with edge replication, the border that image work takes.
        plane("planes_7x7_clamp_ragged", 301, 403, 64, 0, 7, "clamp", "xcorr"),
        # One camera image against a bank of oriented 11x11 kernels, one output plane each.
        plane("bank_11x11_480x640", 480, 640, 0, 16, 11, "clamp", "xcorr"),
        # A wide blur that the operator may take through the FFT: 2048x2048 by 63x63, cyclic,
        # the kernel itself a field that can change from step to step.
        plane("blur_63x63_2048", 2048, 2048, 0, 0, 63, "cyclic", "convolve"),
        # One pyramid level of a three-plane 1080p frame and the way back: DownsampleOutput(2),
        # then UpsampleInput(2), 5x5.
        {"name": "pyramid_1080p", "kind": "pyramid", "rows": 1080, "cols": 1920, "planes": 3, "R": 5, "step": 2,
         "border": "zero"},
        # Separable 9 + 9 taps over eight 1080p frames.
        {"name": "separable_9_1080p", "kind": "separable", "rows": 1080, "cols": 1920, "planes": 8, "R": 9, "S": 9,
         "border": "zero", "op": "convolve"},
        # A ColorField (RGBA bytes) of a 1080p movie through a 5x5 kernel.
        {"name": "color_5x5_1080p", "kind": "color", "rows": 1080, "cols": 1920, "R": 5, "border": "clamp"},
        # One training step of a convolution layer: projectFrame, backProjectFrame and the
        # weight gradient, in FP32 and in split BF16.
        {"name": "layer_fp32_16x32x64_5x5", "kind": "layer", "precision": "fp32", "B": 16, "C": 32, "K": 64,
         "rows": 64, "cols": 64, "R": 5},
        {"name": "layer_bf16x3_16x32x64_5x5", "kind": "layer", "precision": "bf16x3", "B": 16, "C": 32, "K": 64,
         "rows": 64, "cols": 64, "R": 5},
        # One small uneven field through one filter bank: inference on a single sample.
        {"name": "frame_small_ragged", "kind": "frame", "dir": "project", "precision": "bf16x3", "B": 1, "C": 16,
         "K": 16, "rows": 57, "cols": 43, "R": 3, "border": "clamp", "sampling": "none", "step": 1, "relu": True},
        # The eight-layer stack at batch 8, one graph step from a new input to the last field.
        {"name": "stack8_bf16x6_b8", "kind": "stack", "precision": "bf16x6", "B": 8, "rows": 224, "cols": 224, "C": 3,
         "R": 3, "width": 64, "layers": 8},
    ]


def plane(name, rows, cols, planes, fplanes, R, border, op):
    """planes / fplanes 0: a ScalarField / a scalar filter."""
    return {"name": name, "kind": "plane", "rows": rows, "cols": cols, "planes": planes, "fplanes": fplanes, "R": R,
            "border": border, "op": op}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "planes", "planes", "bank", "blur", "pyramid", "separable", "color", "layer", "layer",
                       "frame", "frame", "stack"])
    op = rng.choice(["convolve", "xcorr"])
    if kind == "single":
        c = plane("", _log_int(rng, 24, 512), _log_int(rng, 24, 512), 0, 0, rng.choice([3, 5, 7, 9]),
                  rng.choice(["zero", "clamp", "cyclic", "valid", "full"]), op)
    elif kind == "planes":
        rows, cols = _log_int(rng, 32, 1200), _log_int(rng, 32, 1600)
        if rng.random() < 0.4:
            cols = max(32, cols & ~15)
        most = max(1, 24_000_000 // (rows * cols))
        c = plane("", rows, cols, _log_int(rng, 1, min(1024, most)), 0, rng.choice([3, 3, 5, 5, 7, 9]),
                  rng.choice(["zero", "zero", "clamp", "cyclic", "valid"]), op)
    elif kind == "bank":
        rows, cols, R = _log_int(rng, 96, 800), _log_int(rng, 96, 1000), rng.choice([9, 11, 13, 15, 17, 21])
        most = int(max(1, 600e6 // (rows * cols * R * R)))
        if rng.random() < 0.6:
            c = plane("", rows, cols, 0, min(most, rng.choice([4, 6, 8, 12, 16, 24])), R,
                      rng.choice(["zero", "clamp", "cyclic"]), op)
        else:
            c = plane("", rows, cols, min(most, _log_int(rng, 1, 32)), 0, R, rng.choice(["zero", "clamp", "cyclic"]), op)
    elif kind == "blur":
        rows, cols = _log_int(rng, 256, 2048), _log_int(rng, 256, 2048)
        if rng.random() < 0.4:
            rows = cols = rng.choice([256, 512, 1024, 2048])
        c = plane("", rows, cols, 0, 0, rng.choice([25, 31, 41, 47, 63]), rng.choice(["zero", "clamp", "cyclic"]), op)
    elif kind == "pyramid":
        step = rng.choice([2, 2, 2, 3])
        rows, cols = step * _log_int(rng, 20, 600), step * _log_int(rng, 20, 900)
        c = {"kind": "pyramid", "rows": rows, "cols": cols, "planes": rng.choice([1, 1, 3, 4]),
             "R": rng.choice([3, 5, 5, 7]), "step": step, "border": rng.choice(["zero", "cyclic"])}
    elif kind == "separable":
        rows, cols = _log_int(rng, 64, 1200), _log_int(rng, 64, 1920)
        c = {"kind": "separable", "rows": rows, "cols": cols, "planes": min(rng.choice([1, 3, 8, 16]), max(1, 16_000_000 // (rows * cols))),
             "R": rng.choice([3, 5, 7, 9, 11, 15]), "S": rng.choice([3, 5, 7, 9, 11, 15]),
             "border": rng.choice(["zero", "zero", "clamp", "cyclic"]), "op": op}
    elif kind == "color":
        c = {"kind": "color", "rows": _log_int(rng, 100, 1080), "cols": _log_int(rng, 100, 1920), "R": rng.choice([3, 5, 7]),
             "border": rng.choice(["zero", "clamp", "cyclic"])}
    elif kind == "layer":
        c = {"kind": "layer", "precision": rng.choice(["fp32", "bf16x3"]), "B": rng.choice([1, 2, 4, 8, 16]),
             "C": rng.choice([3, 8, 16, 24, 32, 48, 64]), "K": rng.choice([8, 16, 24, 32, 48, 64]),
             "rows": _log_int(rng, 16, 100), "cols": _log_int(rng, 16, 100), "R": rng.choice([3, 5, 5, 7])}
        _shrink(c, 6.8e9)
    elif kind == "frame":
        sampling = rng.choice(["none", "none", "none", "down", "up"])
        c = {"kind": "frame", "dir": rng.choice(["project", "back"]), "precision": rng.choice(["fp32", "bf16x3", "bf16x6"]),
             "B": rng.choice([1, 1, 2, 4, 8]), "C": rng.choice([1, 3, 8, 16, 32, 64]), "K": rng.choice([4, 8, 16, 32, 64, 96]),
             "rows": 2 * _log_int(rng, 8, 64), "cols": 2 * _log_int(rng, 8, 64), "R": rng.choice([1, 3, 3, 5, 7, 9]),
             "border": rng.choice(["zero", "clamp", "cyclic"] if sampling == "down" else
                                  ["zero", "cyclic"] if sampling == "up" else ["zero", "clamp", "cyclic", "valid", "full"]),
             "sampling": sampling, "step": 1 if sampling == "none" else 2, "relu": rng.random() < 0.5}
        if sampling == "none":
            c["rows"] += rng.choice([0, 1])
            c["cols"] += rng.choice([0, 1])
        _shrink(c, 3e9)
    else:
        c = {"kind": "stack", "precision": rng.choice(["fp32", "bf16x3", "bf16x6"]), "B": rng.choice([1, 2, 4, 8]),
             "rows": 16 * rng.randint(4, 10), "cols": 16 * rng.randint(4, 10), "C": rng.choice([1, 3]), "R": rng.choice([3, 3, 5]),
             "width": rng.choice([16, 32, 48, 64]), "layers": rng.choice([2, 3, 4, 6])}
        while work(c)["flops"] > (4e9 if c["precision"] == "fp32" else 2.4e10) and c["B"] > 1:
            c["B"] //= 2
        while work(c)["flops"] > (4e9 if c["precision"] == "fp32" else 2.4e10):
            c["width"] = max(8, c["width"] // 2)
            c["layers"] = max(2, c["layers"] - 1)
    c.pop("name", None)
    return c


def _shrink(c, flops):
    """Halves the batch, then the planes, until one convolution of the case fits the bound."""
    while 2.0 * c["B"] * c["C"] * c["K"] * c["R"] ** 2 * c["rows"] * c["cols"] > flops:
        if c["B"] > 1:
            c["B"] //= 2
        elif c["K"] >= c["C"]:
            c["K"] //= 2
        else:
            c["C"] //= 2


# ------------------------------------------------------------------------ inputs and passes
def _sampling(c):
    return {"none": C.NoSamplingConvolution, "down": C.DownsampleOutputConvolution(c["step"]),
            "up": C.UpsampleInputConvolution(c["step"])}[c["sampling"]]


def _stack_layers(c):
    """Widths double every second layer; DownsampleOutput(2) after layers 2, 4 and 6; ReLU
    between layers."""
    n = c["layers"]
    return [(c["width"] << (i // 2), c["R"], 2 if i in (1, 3, 5) and i < n - 1 else 1, i < n - 1) for i in range(n)]


def _tensors(c, seed):
    """The case's inputs as FP32 (bytes for a ColorField) CUDA tensors, from the seed."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0):
        return torch.randn(shape, device="cuda", generator=gen) * std

    def uniform(*shape):
        return torch.rand(shape, device="cuda", generator=gen) * 2 - 1

    kind = c["kind"]
    if kind == "plane":
        field = (c["planes"],) if c["planes"] else ()
        filt = (c["fplanes"],) if c["fplanes"] else ()
        R = c["R"]
        x = uniform(*field, c["rows"], c["cols"])
        if R >= 25:  # a wide blur: a normalised Gaussian with a little of its own in every tap
            a = torch.arange(R, device="cuda", dtype=torch.float32) - R // 2
            w = torch.exp(-a * a / (2 * (R / 6.3) ** 2))
            f = w[:, None] * w[None, :] * (1 + 0.05 * uniform(R, R))
            return x * 0.5 + 0.5, f / f.sum()
        return x, uniform(*filt, R, R)
    if kind == "pyramid":
        R = c["R"]
        return uniform(c["planes"], c["rows"], c["cols"]), uniform(R, R) / R, uniform(R, R) / R
    if kind == "separable":
        return uniform(c["planes"], c["rows"], c["cols"]), uniform(c["R"]), uniform(c["S"])
    if kind == "color":
        x = torch.randint(0, 256, (c["rows"], c["cols"], 4), device="cuda", generator=gen, dtype=torch.uint8)
        f = torch.rand((c["R"], c["R"]), device="cuda", generator=gen)
        return x, f / f.sum()
    if kind == "layer":
        B, Cn, K, H, W, R = (c[k] for k in ("B", "C", "K", "rows", "cols", "R"))
        x, f = normal(B * Cn, H, W), normal(K * Cn, R, R, std=math.sqrt(2.0 / (Cn * R * R)))
        h = R // 2
        # the weight gradient of a zero-border layer reads the zero-extended field
        return x, f, normal(B * K, H, W), torch.nn.functional.pad(x, (h, h, h, h))
    if kind == "frame":
        B, Cn, K, R = (c[k] for k in ("B", "C", "K", "R"))
        n_in, n_out = (Cn, K) if c["dir"] == "project" else (K, Cn)
        return normal(B * n_in, c["rows"], c["cols"]), normal(K * Cn, R, R, std=math.sqrt(2.0 / (n_in * R * R)))
    # stack: the input field and a filter bank for each layer
    planes, filters = c["C"], []
    for k, R, _, _ in _stack_layers(c):
        filters.append(normal(k * planes, R, R, std=math.sqrt(2.0 / (planes * R * R))))
        planes = k
    return uniform(c["B"] * c["C"], c["rows"], c["cols"]), filters


def prepare(case, seed):
    t = _tensors(case, seed)
    state = {"case": case, "t": t}
    if case["kind"] == "stack":
        x, filters = t
        stack = LayerStack((case["rows"], case["cols"], case["C"]), case["B"], _stack_layers(case),
                           PRECISIONS[case["precision"]])
        stack.set_filters([f.cpu().numpy() for f in filters])
        state |= {"t": (x,), "stack": stack, "in": stack.input, "out": stack.output}
    return state


def run(state):
    c, t = state["case"], state["t"]
    kind = c["kind"]
    if kind == "plane":
        op = C.convolve if c["op"] == "convolve" else C.crossCorrelate
        return op(t[0], t[1], BORDERS[c["border"]])
    if kind == "pyramid":
        down = C.convolve(t[0], t[1], BORDERS[c["border"]], C.DownsampleOutputConvolution(c["step"]))
        return down, C.convolve(down, t[2], BORDERS[c["border"]], C.UpsampleInputConvolution(c["step"]))
    if kind == "separable":
        op = C.convolveSeparable if c["op"] == "convolve" else C.crossCorrelateSeparable
        return op(t[0], t[1], t[2], BORDERS[c["border"]])
    if kind == "color":
        return C.convolve(t[0], t[1], BORDERS[c["border"]])
    if kind == "layer":
        x, f, dy, xp = t
        B, p = c["B"], PRECISIONS[c["precision"]]
        y = C.projectFrameBlockReduceSum(x, f, C.BorderZero, batchSize=B, precision=p)
        dx = C.backProjectFrameBlockReduceSum(dy, f, C.BorderZero, batchSize=B, precision=p)
        df = C.filterAdjointBlockReduceSum(xp, dy, C.BorderValid, batchSize=B, precision=p)
        return y, dx, df
    if kind == "frame":
        op = C.projectFrameBlockReduceSum if c["dir"] == "project" else C.backProjectFrameBlockReduceSum
        return op(t[0], t[1], BORDERS[c["border"]], _sampling(c), c["B"], PRECISIONS[c["precision"]], c["relu"])
    state["in"].copy_(t[0])
    state["stack"].step()
    return state["out"].clone()  # the next step writes the stack's own field again


# --------------------------------------------------------------------- what a pass must do
def _out_size(n, R, border, down=1, up=1):
    n = n * up
    n = n - R + 1 if border == "valid" else n + R - 1 if border == "full" else n
    return -(-n // down)


def work(case):
    """Bytes: every input once, every output once.  Flops: two per tap that carries a value;
    a wide kernel at most the transforms of a real FFT there and back and of the kernel."""
    c, kind = case, case["kind"]
    rows, cols, R = c["rows"], c["cols"], c["R"]
    if kind == "plane":
        oh, ow = (_out_size(n, R, c["border"]) for n in (rows, cols))
        pin, pf = max(1, c["planes"]), max(1, c["fplanes"])
        pout = max(pin, pf)
        flops = 2.0 * pout * oh * ow * R * R
        fft = 2.5 * rows * cols * math.log2(rows * cols)
        return {"bytes": 4.0 * (pin * rows * cols + pf * R * R + pout * oh * ow), "flops": min(flops, (pin + pf + pout) * fft)}
    if kind == "pyramid":
        p, s = c["planes"], c["step"]
        small, full = p * rows * cols / (s * s), p * rows * cols
        # the coarse field is an output of one call and an input of the next
        return {"bytes": 4.0 * (2 * full + 2 * small + 2 * R * R), "flops": 2.0 * 2 * small * R * R}
    if kind == "separable":
        n = c["planes"] * rows * cols
        return {"bytes": 4.0 * (2 * n + c["R"] + c["S"]), "flops": 2.0 * n * (c["R"] + c["S"])}
    if kind == "color":
        return {"bytes": 8.0 * rows * cols + 4.0 * R * R, "flops": 3 * 2.0 * rows * cols * R * R}
    if kind == "layer":
        B, Cn, K = c["B"], c["C"], c["K"]
        x, dy, f = B * Cn * rows * cols, B * K * rows * cols, K * Cn * R * R
        xp = B * Cn * (rows + R - 1) * (cols + R - 1)
        return {"bytes": 4.0 * (x + 2 * f + dy + dy + x + xp + dy + f), "flops": 3 * 2.0 * B * rows * cols * f}
    if kind == "frame":
        B, Cn, K = c["B"], c["C"], c["K"]
        n_in, n_out = (Cn, K) if c["dir"] == "project" else (K, Cn)
        down, up = (c["step"] if c["sampling"] == s else 1 for s in ("down", "up"))
        oh, ow = (_out_size(n, R, c["border"], down, up) for n in (rows, cols))
        return {"bytes": 4.0 * (B * n_in * rows * cols + K * Cn * R * R + B * n_out * oh * ow),
                "flops": 2.0 * B * oh * ow * K * Cn * R * R / (up * up)}
    n, h, w, flops, weights = c["C"], rows, cols, 0.0, 0
    for k, size, down, _ in _stack_layers(c):
        h, w = -(-h // down), -(-w // down)
        flops += 2.0 * c["B"] * h * w * k * n * size * size
        weights += k * n * size * size
        n = k
    # the input, every filter bank and the last field; the fields between may stay on the chip
    return {"bytes": 4.0 * (c["B"] * c["C"] * rows * cols + weights + c["B"] * n * h * w), "flops": flops}


# --------------------------------------------------------------------------- FP64 restatement
def _extend(x, R, S, border):
    """x (..., H, W) with the border that an R x S filter reads around it."""
    if border == "valid":
        return x
    for dim, size in ((-2, R), (-1, S)):
        h = size - 1 if border == "full" else size // 2
        n = x.shape[dim]
        i = torch.arange(-h, n + h, device=x.device)
        if border == "clamp":
            x = x.index_select(dim, i.clamp(0, n - 1))
        elif border == "cyclic":
            x = x.index_select(dim, i % n)
        else:
            pad = (0, 0, h, h) if dim == -2 else (h, h)
            x = torch.nn.functional.pad(x, pad)
    return x


def _insert(x, up):
    if up == 1:
        return x
    y = x.new_zeros(x.shape[:-2] + (x.shape[-2] * up, x.shape[-1] * up))
    y[..., ::up, ::up] = x
    return y


def _planes64(x, f, border, flip, down=1, up=1):
    """Plane-by-plane: x (..., H, W), f (R, S) or (P, R, S)."""
    x, f = x.double(), f.double()
    R, S = f.shape[-2:]
    if flip:
        f = f.flip(-2, -1)
    x = _extend(_insert(x, up), R, S, border)
    oh, ow = x.shape[-2] - R + 1, x.shape[-1] - S + 1
    y = None
    for r in range(R):
        for s in range(S):
            v = x[..., r:r + oh:down, s:s + ow:down]
            w = f[..., r, s, None, None]
            if y is None:
                y = v * w
            else:
                y.addcmul_(v, w.expand(y.shape) if w.dim() < y.dim() else w)
    return y


def _bank64(x, f, B, border, flip, down=1, up=1):
    """x (B*N, H, W), f (M, N, R, S): out[b, m] = sum over n, the fused filter-bank form."""
    x, f = x.double(), f.double()
    M, N, R, S = f.shape
    if flip:
        f = f.flip(-2, -1)
    x = _extend(_insert(x.reshape(B, N, *x.shape[-2:]), up), R, S, border)
    oh, ow = x.shape[-2] - R + 1, x.shape[-1] - S + 1
    y = 0
    for r in range(R):
        for s in range(S):
            v = x[..., r:r + oh:down, s:s + ow:down]
            shape = v.shape[-2:]
            y = y + torch.matmul(f[:, :, r, s], v.reshape(B, N, -1))
    return y.reshape(B * M, *shape)


def _forward_bank(f, K, Cn):
    return f.reshape(K, Cn, *f.shape[-2:])


def exact(case, seed):
    c, kind = case, case["kind"]
    t = _tensors(c, seed)
    if kind == "color":
        return None
    if kind == "plane":
        return _planes64(t[0], t[1], c["border"], c["op"] == "convolve")
    if kind == "pyramid":
        down = _planes64(t[0], t[1], c["border"], True, down=c["step"])
        return down, _planes64(down, t[2], c["border"], True, up=c["step"])
    if kind == "separable":
        flip = c["op"] == "convolve"
        return _planes64(_planes64(t[0], t[1][None, :], c["border"], flip), t[2][:, None], c["border"], flip)
    if kind == "layer":
        x, f, dy, xp = t
        B, Cn, K, H, W, R = (c[k] for k in ("B", "C", "K", "rows", "cols", "R"))
        bank = _forward_bank(f, K, Cn)
        y = _bank64(x, bank, B, "zero", False)
        dx = _bank64(dy, bank.transpose(0, 1), B, "zero", True)
        g, xp = dy.double().reshape(B, K, H * W), xp.double().reshape(B, Cn, H + R - 1, W + R - 1)
        df = torch.empty((K, Cn, R, R), device=x.device, dtype=torch.float64)
        for r in range(R):
            for s in range(R):
                v = xp[:, :, r:r + H, s:s + W].reshape(B, Cn, H * W)
                df[:, :, r, s] = torch.matmul(g, v.transpose(1, 2)).sum(0)
        return y, dx, df.reshape(K * Cn, R, R)
    if kind == "frame":
        bank = _forward_bank(t[1], c["K"], c["C"])
        back = c["dir"] == "back"
        down, up = (c["step"] if c["sampling"] == s else 1 for s in ("down", "up"))
        y = _bank64(t[0], bank.transpose(0, 1) if back else bank, c["B"], c["border"], back, down, up)
        y = y.clamp_min(0) if c["relu"] else y
        return y[0] if y.shape[0] == 1 else y
    y, filters = t
    planes = c["C"]
    for f, (k, _, down, relu) in zip(filters, _stack_layers(c)):
        # the device's FP32 copy of the filter is the filter; fields stay in FP64
        y = _bank64(y, _forward_bank(f, k, planes), c["B"], "zero", False, down)
        y = y.clamp_min(0) if relu else y
        planes = k
    return y
