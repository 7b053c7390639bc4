import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


def golden_cases(prefix):
    """Names of the golden cases whose reference-Python file exists, e.g. prefix 'b_' or 'd_'."""
    names = sorted(f[len("pyref_"):-4] for f in os.listdir(GOLDEN) if f.startswith("pyref_" + prefix) and f.endswith(".npz"))
    return names


class Golden:
    """One golden case: inputs (float32), metadata and the expected float64 outputs of the reference."""

    def __init__(self, name, source="pyref"):
        f = np.load(os.path.join(GOLDEN, f"pyref_{name}.npz"))
        self.name = name
        self.inputs = {k[3:]: f[k] for k in f.files if k.startswith("in_")}
        self.meta = {k[5:]: f[k].item() for k in f.files if k.startswith("meta_")}
        self.expected = {k[4:]: f[k] for k in f.files if k.startswith("out_")}
        self.cuda = None
        path = os.path.join(GOLDEN, f"cudaref_{name}.npz")
        if os.path.exists(path):
            c = np.load(path)
            self.cuda = {k: c[k] for k in c.files}


def rel_err(got, want):
    """max|got - want| / max|want| (norm-relative error used throughout the parity tests)."""
    got = np.asarray(got, dtype=np.float64)
    want = np.asarray(want, dtype=np.float64)
    return float(np.abs(got - want).max() / max(np.abs(want).max(), 1e-30))


@pytest.fixture(scope="session")
def oracle():
    from oracle import c_oracle
    c_oracle.build()
    return c_oracle


# ------------------------------------------------------------------ which kernel must serve which call
# Mirrors the dispatch rules of csrc/sapa_b.cu, csrc/sapa_tma.cu and csrc/sapa_gath_mma.cu so that a silent fall-back to a slower
# kernel fails a test instead of passing on the fall-back's (correct) numbers.  B images of H x W low-resolution pixels, C channels
# of the value (of the operand itself for sim, agg and gath), d of the query; `groups` of the B belong to one image.

def _ceil(a, b):
    return -(-a // b)


def _filled(W, cells, part, whole):
    """At least part / whole of the columns of strips of `cells` lie inside the image."""
    return whole * W >= part * _ceil(W, cells) * cells


def _rows_of_16_bytes(W, dtype_name):
    return W % (4 if dtype_name == "f32" else 8) == 0


def _wide_columns(W):
    """Tiles of 32 columns with at least three quarters of them inside the image, rows of 16 bytes."""
    return W % 8 == 0 and 4 * W >= 3 * 32 * -(-W // 32)


def _tiles(mode, W, dtype_name, B, H):
    """The K = 5, s = 2 kernel on tiles of a mode (fwd, bwd, sim, agg); None where the FP32-pipe kernels serve (float32, W % 4 != 0)."""
    if dtype_name == "f32":
        return f"sapa_tma_fused_f32_kernel<{mode}>" if W % 4 == 0 else None
    if W % 8 != 0:
        return f"sapa_tma_fused_16_kernel<ragged {mode}>"
    tiles = B * -(-W // 32) * -(-H // 4)
    return f"sapa_wide_16_kernel<{mode}>" if _wide_columns(W) and tiles >= 100 else f"sapa_tma_fused_16_kernel<{mode}>"


def _steps(columns, rows, extra, sms):
    """Steps of the busiest SM when `columns` of `rows` rows are cut into items (split_rows of csrc/umma_util.cuh)."""
    best = None
    for turn in range(_ceil(columns, sms), _ceil(columns, sms) + 5):
        want = min(turn * sms // columns, rows)
        r = _ceil(rows, want)
        total = _ceil(columns * _ceil(rows, r), sms) * (r + extra) + 3
        best = total if best is None else min(best, total)
    return best


def _agg_on_strips(W, dtype_name, B, H, C, groups):
    if dtype_name == "f32":
        import torch
        steps = _steps(B * _ceil(W, 16) * _ceil(C, 128), H, 1, torch.cuda.get_device_properties(0).multi_processor_count)
        return W % 4 == 0 and steps <= 0.7 + 5.1e-6 * B * H * W * (C + 99.0)
    return W % 8 == 0 and C >= 16 and W >= 16 and (_filled(W, 32, 3, 4) or groups * C * H * W >= 6e4)


def expected_fused_forward(K, s, W, dtype_name, B=1, H=1, C=8, d=8):
    if s != 2 or K not in (3, 5) or dtype_name == "f64":
        return None                                   # no fused kernel: the separate ops run
    if K == 3:
        return ["sapa_tile_kernel<fused>"]
    if not _rows_of_16_bytes(W, dtype_name) and (dtype_name == "f32" or W % 2 == 0):
        return ["sapa_mma_fused_kernel"]
    n = C * H * W
    if dtype_name == "f32":
        if _filled(W, 16, 3, 4) and C >= 48 and W * W * C >= (5e5 if C >= 96 else 7.5e5) and n >= 3e5:
            return ["sapa_strip_sim_kernel<softmax>", "sapa_strip_kernel"]
    elif W % 8 == 0 and d <= 64 and W >= 16 and C >= 24 and n >= 2e4 and (n <= 1e8 or C <= 64):
        return ["sapa_strip_fwd_kernel"]
    return [_tiles("fwd", W, dtype_name, B, H)]


def expected_gath(K, s, W, dtype_name, H=1, C=8, groups=1):
    if s != 2 or K not in (3, 5) or dtype_name == "f64":
        return "gath_generic_kernel"
    if K == 3 or (dtype_name == "f32" and W % 2 != 0):
        return "sapa_gath_kernel"
    if dtype_name != "f32" and W % 4 != 0:
        return "sapa_gath_mma_kernel<ragged>"
    n = groups * C * H * W
    if _rows_of_16_bytes(W, dtype_name):
        if dtype_name == "f32" and C >= 64 and _filled(W, 16, 3, 4) and n >= 6e4:
            return "sapa_gath_umma_kernel"
        if dtype_name != "f32" and C >= 32 and (n >= 3e4 if _filled(W, 32, 3, 4) else _filled(W, 32, 5, 8) and n >= 1e5):
            return "sapa_gath_umma_kernel"
    return "sapa_gath_wide_16_kernel" if dtype_name != "f32" and _wide_columns(W) else "sapa_gath_mma_kernel"


def _one(mode, generic, K, s, W, dtype_name, B, H):
    if s != 2 or K not in (3, 5) or dtype_name == "f64":
        return generic
    return [(_tiles(mode, W, dtype_name, B, H) if K == 5 else None) or f"sapa_tile_kernel<{mode}>"]


def expected_fused_backward(K, s, W, dtype_name, B=1, H=1, C=8, d=8):
    stage1 = _one("bwd", ["sim_generic_kernel", "softmax_bwd_generic_kernel", "agg_generic_kernel"], K, s, W, dtype_name, B, H)
    if K == 5 and s == 2 and dtype_name != "f64" and _rows_of_16_bytes(W, dtype_name):
        if dtype_name == "f32" and W >= 16 and C >= 64 and _filled(W, 16, 4, 5):
            stage1 = ["sapa_strip_sim_kernel<softmax_bwd>", "sapa_strip_kernel"]
        elif dtype_name != "f32" and W >= 24 and C >= 32 and _filled(W, 32, 5, 8):
            stage1 = ["sapa_strip_sim_16_kernel<softmax_bwd>", "sapa_strip_kernel"]
    return stage1 + [expected_gath(K, s, W, dtype_name, H, d), expected_gath(K, s, W, dtype_name, H, C)]


def expected_sim(K, s, W, dtype_name, B=1, H=1, C=8, groups=1):
    if K == 5 and s == 2 and dtype_name != "f64" and _rows_of_16_bytes(W, dtype_name):
        if dtype_name != "f32":
            return ["sapa_strip_sim_16_kernel<logits>"]
        if W >= 16 and _filled(W, 16, 3, 4) and groups * C * H * W >= 1e4:
            return ["sapa_strip_sim_kernel<logits>"]
    return _one("sim", ["sim_generic_kernel"], K, s, W, dtype_name, B, H)


def expected_agg(K, s, W, dtype_name, B=1, H=1, C=8, groups=1):
    if K == 5 and s == 2 and dtype_name != "f64" and _agg_on_strips(W, dtype_name, B, H, C, groups):
        return ["sapa_strip_kernel"]
    return _one("agg", ["agg_generic_kernel"], K, s, W, dtype_name, B, H)
