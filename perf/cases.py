"""The work that programs built on sapa_b200 have it do, as cases to time: the SAPA-B and SAPA-D attention operators and
the two modules around them, through the public entry points, inference and training, from one small image to the largest.

A case is a dict of plain values:

    op      "fused" (sapa_fused), "separate" (qk, softmax, av: the reference's own sequence), "pyramid" (a chain of SAPA
            modules, each doubling the resolution), "module" (one SAPA module), "deform" (deform_sapa_fused) or
            "deform_module" (one SAPADeform module)
    train   forward and backward (gradients of all inputs and parameters) instead of inference
    dtype   "f32", "f16", "bf16"; "amp" = float32 parameters and features under torch.autocast(bfloat16)
    B, C, d, H, W   images, value channels, query / key channels, low-resolution height and width (for the modules d is
            embedding_dim and the guidance has C channels too); levels = modules in the pyramid; sigma = standard
            deviation of the sampling offsets in low-resolution pixels
"""
import math

import torch

import sapa_b200

K, S, GROUPS, POINTS = 5, 2, 4, 9
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "amp": torch.float32}


def listed():
    return [
        # one small feature map, as in the operator's smallest use (latency of a single call)
        {"name": "small_infer_f32", "op": "fused", "train": False, "dtype": "f32", "B": 1, "C": 64, "d": 32, "H": 16, "W": 16},
        # the headline workload: one decoder level of a batch, inference
        {"name": "infer_f32", "op": "fused", "train": False, "dtype": "f32", "B": 8, "C": 256, "d": 64, "H": 64, "W": 64},
        # batched serving at a large feature size, 16-bit
        {"name": "infer_bf16_batch", "op": "fused", "train": False, "dtype": "bf16", "B": 64, "C": 256, "d": 64, "H": 128, "W": 128},
        # one huge image (remote sensing, pathology): planes of megabytes per channel
        {"name": "infer_bf16_plane", "op": "fused", "train": False, "dtype": "bf16", "B": 1, "C": 256, "d": 64, "H": 1024, "W": 1024},
        # a training step through the operator
        {"name": "train_f32", "op": "fused", "train": True, "dtype": "f32", "B": 8, "C": 256, "d": 64, "H": 64, "W": 64},
        # a detector's pyramid level (800 x 1344 input at stride 32): rows of no convenient length, 16-bit training
        {"name": "train_bf16_ragged", "op": "fused", "train": True, "dtype": "bf16", "B": 2, "C": 256, "d": 32, "H": 25, "W": 42},
        # programs that keep the reference's own sequence of operators
        {"name": "separate_train_f16", "op": "separate", "train": True, "dtype": "f16", "B": 4, "C": 128, "d": 32, "H": 32, "W": 32},
        # segmentation decoder: three chained upsampling modules on projected encoder features
        {"name": "pyramid_infer_bf16", "op": "pyramid", "train": False, "dtype": "bf16", "B": 16, "C": 256, "d": 32, "H": 16, "W": 16, "levels": 3},
        # a training step of the module in mixed precision
        {"name": "module_train_amp", "op": "module", "train": True, "dtype": "amp", "B": 8, "C": 256, "d": 32, "H": 32, "W": 32},
        # the deformable operator: inference, and a training step
        {"name": "deform_infer_f32", "op": "deform", "train": False, "dtype": "f32", "B": 8, "C": 256, "d": 64, "H": 64, "W": 64, "sigma": 0.5},
        {"name": "deform_train_bf16", "op": "deform", "train": True, "dtype": "bf16", "B": 8, "C": 256, "d": 64, "H": 64, "W": 64, "sigma": 0.5},
        # the deformable module with its learned offsets, as it runs in a model
        {"name": "deform_module_infer_f16", "op": "deform_module", "train": False, "dtype": "f16", "B": 4, "C": 256, "d": 32, "H": 32, "W": 32},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# for each kind of case: the element types it is run in, and the most output elements (B * C * 2H * 2W) of a drawn one
_KINDS = {
    ("fused", False): (("f32", "f16", "bf16"), 1 << 29), ("fused", True): (("f32", "f16", "bf16"), 1 << 26),
    ("separate", False): (("f32", "f16", "bf16"), 1 << 25), ("separate", True): (("f32", "f16", "bf16"), 1 << 25),
    ("pyramid", False): (("f32", "f16", "bf16"), 1 << 26), ("module", False): (("f32", "f16", "bf16"), 1 << 26),
    ("module", True): (("f32", "amp"), 1 << 24),
    ("deform", False): (("f32", "f16", "bf16"), 1 << 25), ("deform", True): (("f32", "f16", "bf16"), 1 << 24),
    ("deform_module", False): (("f32", "f16", "bf16"), 1 << 25), ("deform_module", True): (("f32", "amp"), 1 << 23),
}


def draw(rng):
    op, train = rng.choice([("fused", False)] * 3 + [("fused", True)] * 2 + list(_KINDS)[2:])
    dtypes, most = _KINDS[op, train]
    case = {"op": op, "train": train, "dtype": rng.choice(dtypes)}
    grouped = op in ("module", "pyramid")            # GroupNorm(32, C)
    case["C"] = rng.choice((64, 96, 128, 192, 256, 320, 512) if grouped else (32, 48, 64, 96, 128, 192, 256, 320, 512))
    case["d"] = rng.choice((32, 64) if op == "deform_module" else (16, 32, 48, 64))
    if op == "pyramid":
        case["levels"] = rng.choice((2, 3))
    up = 4 ** case.get("levels", 1) * case["C"]
    room = most // up                                # low-resolution pixels of the whole batch
    side = min(256 if op == "fused" and not train else 128, math.isqrt(room))
    case["H"] = _spread(rng, 4, side)
    case["W"] = _spread(rng, max(4, case["H"] // 2), max(8, min(side, 2 * case["H"])))
    if rng.random() < 0.5:                           # half of them in multiples of eight, as padded inputs have them
        case["H"], case["W"] = (8 * max(1, round(x / 8)) for x in (case["H"], case["W"]))
    case["B"] = _spread(rng, 1, max(1, min(64, room // (case["H"] * case["W"]))))
    if op == "deform":
        case["sigma"] = rng.choice((0.25, 0.5, 1.0))
    return case


def _normal(gen, *shape, dtype, scale=1.0, shift=0.0):
    return (torch.randn(*shape, generator=gen, device=gen.device) * scale + shift).to(dtype)


def _module(case, gen, dtype):
    make = sapa_b200.SAPADeform if case["op"] == "deform_module" else sapa_b200.SAPA
    m = make(case["C"], embedding_dim=case["d"]).to(gen.device)
    with torch.no_grad():
        for name, p in m.named_parameters():         # projections as they are initialised, biases and norms as after some training
            scale, shift = (0.02, 0.0) if p.dim() > 1 else (0.1, 1.0 if "norm" in name and "weight" in name else 0.0)
            p.copy_(_normal(gen, *p.shape, dtype=p.dtype, scale=scale, shift=shift))
            p.requires_grad_(case["train"])
    return m.to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt, op = DTYPES[case["dtype"]], case["op"]
    B, C, d, H, W = (case[k] for k in ("B", "C", "d", "H", "W"))
    st = {"case": case}
    if op in ("fused", "separate", "deform"):
        st["inputs"] = [_normal(gen, B, d, S * H, S * W, dtype=dt, scale=0.5), _normal(gen, B, d, H, W, dtype=dt, scale=0.5),
                        _normal(gen, B, C, H, W, dtype=dt)]
        if op == "deform":
            st["inputs"].append(_normal(gen, B, 2 * GROUPS * POINTS, S * H, S * W, dtype=dt, scale=case["sigma"]))
    else:
        levels = case.get("levels", 1)
        st["modules"] = [_module(case, gen, dt) for _ in range(levels)]
        st["inputs"] = [_normal(gen, B, C, H << i, W << i, dtype=dt) for i in range(levels + 1)]    # x, then the guidances
    if case["train"]:
        st["inputs"] = [t.requires_grad_() for t in st["inputs"]]
        out = torch.bfloat16 if case["dtype"] == "amp" else dt
        st["grad"] = _normal(gen, B, C, S * H, S * W, dtype=out)
        st["wanted"] = st["inputs"] + [p for m in st.get("modules", ()) for p in m.parameters()]
    return st


def _forward(st):
    case, x = st["case"], st["inputs"]
    if case["op"] == "fused":
        return sapa_b200.sapa_fused(*x, K, S)
    if case["op"] == "separate":
        attn = torch.softmax(sapa_b200.qk(x[0], x[1], K, S), dim=1)
        return sapa_b200.av(attn, x[2], K, S)
    if case["op"] == "deform":
        return sapa_b200.deform_sapa_fused(*x, POINTS, S, GROUPS)
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=case["dtype"] == "amp"):
        out = x[0]
        for module, guidance in zip(st["modules"], x[1:]):
            out = module(guidance, out)
        return out


def run(state):
    if not state["case"]["train"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    return [out.detach()] + list(torch.autograd.grad(out, state["wanted"], state["grad"]))


def work(case):
    """Inputs read once and outputs written once; the multiply-adds of the window contractions (and projections), twice each."""
    es = 4 if case["dtype"] in ("f32", "amp") else 2
    op, train, B, C, d = (case[k] for k in ("op", "train", "B", "C", "d"))
    total = {"bytes": 0.0, "flops": 0.0}
    for level in range(case.get("levels", 1)):
        lo = B * (case["H"] << level) * (case["W"] << level)
        hi = S * S * lo
        elems = (lo + hi) * (C if op in ("module", "pyramid", "deform_module") else d) + C * lo
        if op in ("module", "pyramid", "deform_module"):
            elems -= C * lo                          # the value is the low-resolution feature itself
        offsets = 2 * GROUPS * POINTS * hi if op == "deform" else 0
        elems += offsets
        out = C * hi
        width = d * GROUPS if op == "deform_module" else d
        taps = 4 * POINTS if op.startswith("deform") else K * K
        flops = 2.0 * hi * taps * (width + C)
        if op in ("module", "pyramid", "deform_module"):
            flops += 2.0 * (lo + hi) * C * width
        if op == "deform_module":
            flops += 2.0 * lo * C * 2 * GROUPS * POINTS * S * S
        if train:                                    # inputs, the output's gradient; the output and a gradient per input
            total["bytes"] += es * (2 * elems) + (2 if case["dtype"] == "amp" else es) * 2 * out
            flops *= 3
        else:
            total["bytes"] += es * (elems + (out if level == case.get("levels", 1) - 1 or op != "pyramid" else 0))
        total["flops"] += flops
    return total


def tolerance(case):
    """What the element types give.  float32: sums of a few hundred products, exponentials, and gradients of those; where a
    module's convolutions are torch's they run in TensorFloat-32, as torch has it by default.  16 bits: operands, attention
    map and gradients are rounded to 11 or 8 bits on the way, in training several times.  The modules' gradients include
    those of the key bias and norm, sums over all pixels that cancel but for the borders."""
    module = case["op"] in ("module", "pyramid", "deform_module")
    if case["dtype"] == "f32":
        if module and case["train"]:
            return {"rel": 1e-2}
        return {"rel": 2e-3 if case["op"] == "deform_module" else 2e-5 if module else 1e-5}
    if module and case["train"]:
        return {"rel": 3e-2}
    step = 1e-3 if case["dtype"] == "f16" else 8e-3
    return {"rel": 2 * step if case["train"] else step}
