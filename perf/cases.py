"""The work a program has this framework do, as a list of cases for timing and comparison.

Each case is one call (or one forward and backward) through a public entry point:
`bridct_b200.torch_api` for CUDA tensors, `bridct_b200.ragged.RaggedBatch` for mixed shapes and
`bridct_b200.bridct_numpy.Plan` for host arrays.  The workloads are those of `bench.py` where it has
one: the 8x8 block batch of a 4096x4096 image, 1024 arrays of 64x64, the 2048 x 256^2 sweep of
magnitudes, one 1024x1024 array, blocks inside an image, and the mixed-shape batch.

`draw` spreads over every supported shape (each axis a power of two from 8 to 1024), the three
modes, the execution forms and batch sizes from one array to the size of the largest listed case.
"""
import math

import numpy as np
import torch

from bridct_b200 import torch_api
from bridct_b200.bridct_numpy import Plan as HostPlan
from bridct_b200.ragged import RaggedBatch, two_pass

AXES = (8, 16, 32, 64, 128, 256, 512, 1024)
FORWARD, INVERSE, ROUNDTRIP = 0, 1, 2

# A luminance quantization table as used with 8x8 blocks: small steps at low frequencies.
QUANT = [[16.0 + 4.0 * (r + c) + 1.5 * r * c for c in range(8)] for r in range(8)]


def listed():
    return [
        # The smallest call: one array of the 64x64 configuration, latency alone.
        {"name": "one64", "kind": "plan", "h": 64, "w": 64, "mode": FORWARD, "batch": 1, "form": "sj"},
        # The block transform of a 4096x4096 image, blocks stored one after another.
        {"name": "blocks8", "kind": "plan", "h": 8, "w": 8, "mode": FORWARD, "batch": 262144, "form": "sj"},
        # A DCT layer in a training step: forward and gradient of 1024 arrays of 64x64.
        {"name": "train64", "kind": "train", "h": 64, "w": 64, "batch": 1024},
        # Spectra of a large data set of 256x256 arrays whose magnitudes span twelve decades.
        {"name": "sweep256", "kind": "plan", "h": 256, "w": 256, "mode": FORWARD, "batch": 2048, "form": "sj"},
        # One large image: a single 1024x1024 array.
        {"name": "one1024", "kind": "plan", "h": 1024, "w": 1024, "mode": FORWARD, "batch": 1, "form": "sj"},
        # Reconstruction of a stack of wide images from their spectra.
        {"name": "inverse512x1024", "kind": "plan", "h": 512, "w": 1024, "mode": INVERSE, "batch": 24, "form": "sj"},
        # Normalized round trip of an odd number of tall tiles (an accuracy check over a data set).
        {"name": "roundtrip256x64", "kind": "plan", "h": 256, "w": 64, "mode": ROUNDTRIP, "batch": 777, "form": "sj"},
        # Patches taken where they lie in wider rows (a view, no copy), an odd number of them.
        {"name": "patches16x64", "kind": "strided", "h": 16, "w": 64, "mode": INVERSE, "batch": 3001, "margin": 8},
        # A codec step on a full-HD luminance plane: every 8x8 block transformed where it lies and quantized.
        {"name": "frame1080q", "kind": "image", "h": 1080, "w": 1920, "mode": FORWARD, "quant": True, "margin": 0},
        # A batch of arrays of mixed shapes and directions, its two-pass classes in merged passes.
        {"name": "ragged1024", "kind": "ragged", "count": 1024, "top": 1024, "schedule": "merged", "mix": 1},
        # The tensor-core precision form on a batch of 256x256 arrays.
        {"name": "bf16x3_256", "kind": "plan", "h": 256, "w": 256, "mode": FORWARD, "batch": 256, "form": "tc_bf16x3"},
        # A host array through the NumPy plan: copy in, transform, copy out.
        {"name": "host512", "kind": "host", "h": 512, "w": 512, "mode": FORWARD},
    ]


# Most elements of one drawn case, so that none costs more than the largest listed one: the plain
# form's largest listed batch where a line has at most 256 points, and less for longer lines, round
# trips and the slower forms.
_MOST = {"sj": 1 << 25, "tc_bf16x3": 1 << 23, "tc_tf32x3": 1 << 22, "tc_fp8": 1 << 21}


def _most_plain(h, w, mode):
    return 2048 * 256 * 256 if max(h, w) <= 256 and mode != ROUNDTRIP else _MOST["sj"]


def _batch(rng, elements, most):
    """A batch of log-uniform size between one array and `most` elements."""
    top = max(1, most // elements)
    return max(1, min(top, int(round(math.exp(rng.uniform(0.0, math.log(top)))))))


def draw(rng):
    h, w = rng.choice(AXES), rng.choice(AXES)
    mode = rng.choice((FORWARD, FORWARD, INVERSE, INVERSE, ROUNDTRIP))
    kind = rng.choice(("plan",) * 11 + ("train", "train", "strided", "strided", "image", "image", "ragged", "form", "form", "host"))
    if kind == "train":
        return {"kind": "train", "h": h, "w": w, "batch": _batch(rng, h * w, _MOST["sj"] // 2)}
    if kind == "strided":
        return {"kind": "strided", "h": h, "w": w, "mode": mode, "batch": _batch(rng, h * w, _MOST["sj"]),
                "margin": 4 * rng.randint(1, 8)}
    if kind == "image":
        return {"kind": "image", "h": 8 * rng.randint(16, 512), "w": 8 * rng.randint(16, 512), "mode": mode,
                "quant": mode != ROUNDTRIP and rng.random() < 0.5, "margin": 4 * rng.randint(0, 8)}
    if kind == "ragged":
        return {"kind": "ragged", "count": int(round(math.exp(rng.uniform(math.log(16), math.log(640))))),
                "top": rng.choice((256, 512, 1024)), "schedule": rng.choice(("queue", "merged")),
                "mix": rng.randint(2, 1 << 20)}
    if kind == "form":
        form = rng.choice(("tc_bf16x3", "tc_bf16x3", "tc_tf32x3", "tc_fp8"))
        return {"kind": "plan", "h": h, "w": w, "mode": rng.choice((FORWARD, INVERSE)),
                "batch": _batch(rng, h * w, _MOST[form]), "form": form}
    if kind == "host":
        return {"kind": "host", "h": h, "w": w, "mode": mode}
    return {"kind": "plan", "h": h, "w": w, "mode": mode, "batch": _batch(rng, h * w, _most_plain(h, w, mode)),
            "form": "sj"}


# ---- inputs ------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _values(batch, h, w, mode, seed):
    """What a transform meets: centred 8-bit pixels for blocks, samples whose magnitude varies from
    array to array (1e-6 to 1e6) for forward transforms of arrays, and spectra that fall off with
    the frequency for inverse transforms."""
    g = _gen(seed)
    if mode != INVERSE and h == 8 and w == 8:
        return torch.randint(0, 256, (batch, h, w), generator=g, device="cuda").float() - 128.0
    x = torch.randn((batch, h, w), generator=g, device="cuda")
    if mode == INVERSE:
        r = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
        c = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
        x *= 64.0 / (1.0 + r + c)
    elif batch >= 256:
        x *= torch.pow(10.0, torch.rand((batch, 1, 1), generator=g, device="cuda") * 12.0 - 6.0)
    return x


def _frame(case, seed):
    """A float plane of centred 8-bit samples (or quantized spectra for the inverse) with row margin."""
    h, w, m = case["h"], case["w"], case["margin"]
    g = _gen(seed)
    wide = torch.randint(0, 256, (h, w + m), generator=g, device="cuda").float() - 128.0
    if case["mode"] == INVERSE:
        wide = torch.round(wide / 16.0)
    return wide[:, :w]


def _items(case):
    """Shapes and directions of a mixed batch: each axis a power of two up to `top`."""
    r = np.random.default_rng(case["mix"])
    axes = [a for a in AXES if a <= case["top"]]
    out = []
    for _ in range(case["count"]):
        h, w = (int(axes[int(r.integers(len(axes)))]) for _ in range(2))
        out.append((h, w, int(r.integers(2))))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plan":
        x = _values(case["batch"], case["h"], case["w"], case["mode"], seed)
        if case["batch"] == 1:
            x = x[0]
        plan = torch_api.Plan(case["h"], case["w"], form=case["form"])
        call = (plan.forward, plan.inverse, plan.roundtrip)[case["mode"]]
        return {"kind": kind, "call": call, "x": x, "out": torch.empty_like(x)}
    if kind == "train":
        x = _values(case["batch"], case["h"], case["w"], FORWARD, seed).requires_grad_()
        g = _values(case["batch"], case["h"], case["w"], INVERSE, seed + 7919)
        return {"kind": kind, "x": x, "g": g}
    if kind == "strided":
        m = case["margin"]
        wide = torch.zeros((case["batch"], case["h"], case["w"] + 2 * m), device="cuda")
        view = wide[:, :, m:m + case["w"]]
        view.copy_(_values(case["batch"], case["h"], case["w"], case["mode"], seed))
        plan = torch_api.Plan(case["h"], case["w"])
        call = (plan.forward, plan.inverse, plan.roundtrip)[case["mode"]]
        return {"kind": kind, "call": call, "x": view, "out": torch.empty(view.shape, device="cuda")}
    if kind == "image":
        x = _frame(case, seed)
        return {"kind": kind, "x": x, "mode": case["mode"], "quant": QUANT if case["quant"] else None,
                "out": torch.empty((case["h"], case["w"]), device="cuda")}
    if kind == "ragged":
        items = _items(case)
        schedule = None
        if case["schedule"] == "merged":
            names = {f"{h}x{w}/{m}": "merged" for h, w, m in items if two_pass(h, w, m)}
            schedule = {"classes": names, "streams": 2}
        batch = RaggedBatch(items, schedule=schedule)
        x = torch.randn(batch.span, generator=_gen(seed), device="cuda")
        return {"kind": kind, "batch": batch, "x": x, "y": torch.empty_like(x)}
    if kind == "host":
        r = np.random.default_rng(seed)
        x = r.standard_normal((case["h"], case["w"]), dtype=np.float32)
        plan = HostPlan(case["h"], case["w"])
        call = (plan.forward, plan.inverse, plan.roundtrip)[case["mode"]]
        return {"kind": kind, "plan": plan, "call": call, "x": x, "out": np.empty_like(x)}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind in ("plan", "strided", "host"):
        return state["call"](state["x"], out=state["out"])
    if kind == "train":
        y = torch_api.dct2(state["x"])
        return y, torch.autograd.grad(y, state["x"], state["g"])[0]
    if kind == "image":
        return torch_api.image_blocks8(state["x"], state["mode"], quant=state["quant"], out=state["out"])
    return state["batch"].apply(state["x"], state["y"])


# ---- the work and the exact results ------------------------------------------------------------

def _lines(n):
    """Floating operations of one n-point transform (split radix, scaled outputs)."""
    return 2.0 * n * math.log2(n)


def work(case):
    """Each element read once and written once; per axis a fast transform of every line."""
    kind = case["kind"]
    if kind == "ragged":
        items = _items(case)
        return {"bytes": 8 * sum(h * w for h, w, _ in items),
                "flops": sum(w * _lines(h) + h * _lines(w) for h, w, _ in items)}
    h, w = case["h"], case["w"]
    if kind == "image":
        return {"bytes": 8 * h * w, "flops": h * w / 64 * 16 * _lines(8) * (2 if case["mode"] == ROUNDTRIP else 1)}
    batch = case.get("batch", 1)
    times = 2 if kind == "train" or case["mode"] == ROUNDTRIP else 1
    return {"bytes": (16 if kind == "train" else 8) * batch * h * w,
            "flops": times * batch * (w * _lines(h) + h * _lines(w))}


def _matrix(n):
    k = torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    j = torch.arange(n, device="cuda", dtype=torch.float64)[None, :]
    c = torch.cos(math.pi * k * (2 * j + 1) / (2 * n)) * math.sqrt(2.0 / n)
    c[0] *= math.sqrt(0.5)
    return c


def _transform(x, mode):
    """The orthonormal 2D DCT-II (or DCT-III, or both in turn) over the last two axes, in float64."""
    x = x.double()
    ch, cw = _matrix(x.shape[-2]), _matrix(x.shape[-1])
    if mode != INVERSE:
        x = ch @ x @ cw.T
    if mode != FORWARD:
        x = ch.T @ x @ cw
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "host":
        r = np.random.default_rng(seed)
        x = torch.from_numpy(r.standard_normal((case["h"], case["w"]), dtype=np.float32)).cuda()
        return _transform(x, case["mode"]).cpu().numpy()
    if kind == "image":
        if case["quant"]:
            return None     # rounded values: no number to be near to
        x = _frame(case, seed)
        h, w = x.shape
        b = x.reshape(h // 8, 8, w // 8, 8).transpose(1, 2)
        return _transform(b, case["mode"]).transpose(1, 2).reshape(h, w)
    if kind == "ragged":
        items = _items(case)
        span = sum(h * w for h, w, _ in items)
        x = torch.randn(span, generator=_gen(seed), device="cuda")
        y = torch.empty(span, device="cuda", dtype=torch.float64)
        at = 0
        for h, w, m in items:
            y[at:at + h * w] = _transform(x[at:at + h * w].view(h, w), m).reshape(-1)
            at += h * w
        return y
    if kind == "train":
        x = _values(case["batch"], case["h"], case["w"], FORWARD, seed)
        g = _values(case["batch"], case["h"], case["w"], INVERSE, seed + 7919)
        return _transform(x, FORWARD), _transform(g, INVERSE)
    x = _values(case["batch"], case["h"], case["w"], case["mode"], seed)
    y = _transform(x, case["mode"])
    return y[0] if case["batch"] == 1 and kind == "plan" else y
