"""Projections that share their launches (sapa_project_list_forward), against float64 GroupNorm + convolution."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


class Record(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("x", "gamma", "beta", "weight", "bias", "out", "stats")] + \
               [(n, ctypes.c_int) for n in ("B", "C", "HW", "d", "groups")] + [("eps", ctypes.c_float)]


def _problem(gen, x, d, groups, bias, dtype, odd_weight):
    C = x.shape[1]
    draw = lambda *s, scale=1.0, shift=0.0: (torch.randn(*s, generator=gen, device="cuda") * scale + shift).to(dtype)
    w = draw(d * C + 1, scale=0.05)
    w = (w[1:] if odd_weight else w[:-1].clone()).view(d, C)           # a weight that starts on no 16-byte boundary is folded, not used as it is
    return {"x": x, "w": w, "b": draw(d, scale=0.5) if bias else None, "groups": groups,
            "gamma": draw(C, scale=0.3, shift=1.0) if groups else None, "beta": draw(C, scale=0.3) if groups else None}


# (B, C, H, W) of the two inputs; per projection: input, rows, groups, bias, pixel shuffle, odd weight
LISTS = {
    "module_with_norm": ([(2, 64, 16, 16), (2, 64, 8, 8)], [(0, 32, 32, True, 0, False), (1, 32, 32, True, 0, False)]),
    "no_norm_mixed_rows": ([(3, 96, 8, 20), (3, 96, 4, 10)], [(0, 48, 0, True, 0, False), (1, 48, 0, False, 0, True), (1, 288, 0, True, 10, False)]),
    "shared_statistics": ([(2, 128, 8, 12), (2, 128, 4, 6)], [(0, 64, 32, True, 0, False), (1, 64, 32, True, 0, False), (1, 16, 32, True, 6, False)]),
    "more_parts_than_a_launch": ([(1, 64, 4, 8), (1, 64, 8, 8)], [(0, 1024, 0, True, 0, False), (1, 768, 8, True, 0, False), (1, 16, 8, False, 0, False)]),
}


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2), (torch.float16, 2e-3)])
@pytest.mark.parametrize("name", LISTS)
def test_list_equals_separate_float64(name, dtype, tol):
    """tol: as for one projection (test_projection_gpu.py) - the arithmetic of a problem does not depend on its list."""
    from sapa_b200 import _lib
    handle = _lib.lib()
    gen = torch.Generator(device="cuda").manual_seed(7)
    inputs, problems = LISTS[name]
    xs = [torch.randn(*s, generator=gen, device="cuda").to(dtype) for s in inputs]
    made = [_problem(gen, xs[i], d, g, b, dtype, odd) for i, d, g, b, _, odd in problems]
    n, records, outs = len(made), (Record * len(made))(), []
    for r, q, (_, d, groups, _, shuffle, _) in zip(records, made, problems):
        B, C, H, W = q["x"].shape
        out = torch.empty((B, d // 4, 2 * H, 2 * W) if shuffle else (B, d, H, W), device="cuda", dtype=dtype)
        outs.append(out)
        for field, t in (("x", q["x"]), ("gamma", q["gamma"]), ("beta", q["beta"]), ("weight", q["w"]), ("bias", q["b"]), ("out", out)):
            setattr(r, field, t.data_ptr() if t is not None else None)
        r.B, r.C, r.HW, r.d, r.groups, r.eps = B, C, H * W, d, groups, 1e-5
    code = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype]
    need = handle.sapa_project_list_workspace(records, n, code)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    widths = (ctypes.c_int * n)(*[p[4] for p in problems])
    status = handle.sapa_project_list_forward(records, widths, n, ws.data_ptr(), need, code, code, torch.cuda.current_stream().cuda_stream)
    assert status == 0, handle.sapa_last_error()
    for q, out, (_, d, groups, _, shuffle, _) in zip(made, outs, problems):
        y = q["x"].double()
        if groups:
            y = F.group_norm(y, groups, q["gamma"].double(), q["beta"].double(), 1e-5)
        ref = F.conv2d(y, q["w"].double().view(d, -1, 1, 1), q["b"].double() if q["b"] is not None else None)
        if shuffle:
            ref = F.pixel_shuffle(ref, 2)
        assert float((out.double() - ref).abs().max() / ref.abs().max()) < tol


def _reference(q, groups, shuffle):
    y = q["x"].double()
    if groups:
        y = F.group_norm(y, groups, q["gamma"].double(), q["beta"].double(), 1e-5)
    ref = F.conv2d(y, q["w"].double().view(q["w"].shape[0], -1, 1, 1), q["b"].double() if q["b"] is not None else None)
    return F.pixel_shuffle(ref, 2) if shuffle else ref


@pytest.mark.parametrize("out_dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2), (torch.float16, 2e-3)])
def test_float32_lists_with_16_bit_outputs(out_dtype, tol):
    """Mixed precision: float32 products, rounded once when they are written."""
    from sapa_b200 import _lib
    handle = _lib.lib()
    gen = torch.Generator(device="cuda").manual_seed(11)
    inputs, problems = LISTS["shared_statistics"]
    xs = [torch.randn(*s, generator=gen, device="cuda") for s in inputs]
    made = [_problem(gen, xs[i], d, g, b, torch.float32, odd) for i, d, g, b, _, odd in problems]
    records, outs = (Record * len(made))(), []
    for r, q, (_, d, groups, _, shuffle, _) in zip(records, made, problems):
        B, C, H, W = q["x"].shape
        outs.append(torch.empty((B, d // 4, 2 * H, 2 * W) if shuffle else (B, d, H, W), device="cuda", dtype=out_dtype))
        for field, t in (("x", q["x"]), ("gamma", q["gamma"]), ("beta", q["beta"]), ("weight", q["w"]), ("bias", q["b"]), ("out", outs[-1])):
            setattr(r, field, t.data_ptr() if t is not None else None)
        r.B, r.C, r.HW, r.d, r.groups, r.eps = B, C, H * W, d, groups, 1e-5
    need = handle.sapa_project_list_workspace(records, len(made), 0)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    code = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[out_dtype]
    assert handle.sapa_project_list_forward(records, (ctypes.c_int * len(made))(*[p[4] for p in problems]), len(made), ws.data_ptr(), need, 0, code,
                                            torch.cuda.current_stream().cuda_stream) == 0, handle.sapa_last_error()
    for q, out, (_, _, groups, _, shuffle, _) in zip(made, outs, problems):
        ref = _reference(q, groups, shuffle)
        assert float((out.double() - ref).abs().max() / ref.abs().max()) < tol


@pytest.mark.parametrize("d,groups,shuffle,bias", [(32, 0, 10, True), (288, 0, 10, False), (288, 8, 0, True), (1024, 32, 10, True)])
@pytest.mark.parametrize("dtype,out_dtype,tol", [(torch.float32, torch.float32, 1e-5), (torch.float32, torch.bfloat16, 1e-2), (torch.bfloat16, torch.bfloat16, 1e-2),
                                                 (torch.float16, torch.float16, 2e-3)])
def test_one_projection_of_many_rows(d, groups, shuffle, bias, dtype, out_dtype, tol):
    """sapa_project_rows_forward: parts of up to 256 rows, sub-pixels, 16-bit outputs of float32; everything is folded."""
    from sapa_b200 import _lib
    handle = _lib.lib()
    gen = torch.Generator(device="cuda").manual_seed(d)
    B, C, H, W = 2, 96, 8, 10
    q = _problem(gen, torch.randn(B, C, H, W, generator=gen, device="cuda").to(dtype), d, groups, bias, dtype, False)
    out = torch.empty((B, d // 4, 2 * H, 2 * W) if shuffle else (B, d, H, W), device="cuda", dtype=out_dtype)
    codes = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}
    need = handle.sapa_project_rows_workspace(B, C, H * W, d, groups, codes[dtype])
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    pointer = lambda t: t.data_ptr() if t is not None else None
    status = handle.sapa_project_rows_forward(pointer(q["x"]), pointer(q["gamma"]), pointer(q["beta"]), pointer(q["w"]), pointer(q["b"]), pointer(out), shuffle,
                                              ws.data_ptr(), need, B, C, H * W, d, groups, 1e-5, codes[dtype], codes[out_dtype], torch.cuda.current_stream().cuda_stream)
    assert status == 0, handle.sapa_last_error()
    ref = _reference(q, groups, shuffle)
    assert float((out.double() - ref).abs().max() / ref.abs().max()) < tol
