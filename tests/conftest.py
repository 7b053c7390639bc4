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
# kernel fails a test instead of passing on the fall-back's (correct) numbers.  B images of H x W low-resolution pixels.

def _wide_columns(W):
    """Tiles of 32 columns with at least three quarters of them inside the image, rows of 16 bytes."""
    return W % 8 == 0 and 4 * W >= 3 * 32 * -(-W // 32)


def _tensor_core(mode, W, dtype_name, B, H):
    """The K = 5, s = 2 kernel of a mode (fwd, bwd, sim, agg); None where the FP32-pipe kernels serve (float32, W % 4 != 0)."""
    if dtype_name == "f32":
        return f"sapa_tma_fused_f32_kernel<{mode}>" if W % 4 == 0 else None
    if W % 8 != 0:
        return f"sapa_tma_fused_16_kernel<ragged {mode}>"
    tiles = B * -(-W // 32) * -(-H // 4)
    return f"sapa_wide_16_kernel<{mode}>" if _wide_columns(W) and tiles >= 100 else f"sapa_tma_fused_16_kernel<{mode}>"


def expected_fused_forward(K, s, W, dtype_name, B=1, H=1):
    if s != 2 or K not in (3, 5) or dtype_name == "f64":
        return None                                   # no fused kernel: the separate ops run
    if K == 3:
        return ["sapa_tile_kernel<fused>"]
    if W % (4 if dtype_name == "f32" else 8) != 0 and (dtype_name == "f32" or W % 2 == 0):
        return ["sapa_mma_fused_kernel"]
    return [_tensor_core("fwd", W, dtype_name, B, H)]


def expected_gath(K, s, W, dtype_name):
    if s != 2 or K not in (3, 5) or dtype_name == "f64":
        return "gath_generic_kernel"
    if K == 3 or (dtype_name == "f32" and W % 2 != 0):
        return "sapa_gath_kernel"
    if dtype_name != "f32" and W % 4 != 0:
        return "sapa_gath_mma_kernel<ragged>"
    return "sapa_gath_wide_16_kernel" if dtype_name != "f32" and _wide_columns(W) else "sapa_gath_mma_kernel"


def _one(mode, generic, K, s, W, dtype_name, B, H):
    if s != 2 or K not in (3, 5) or dtype_name == "f64":
        return generic
    return [(_tensor_core(mode, W, dtype_name, B, H) if K == 5 else None) or f"sapa_tile_kernel<{mode}>"]


def expected_fused_backward(K, s, W, dtype_name, B=1, H=1):
    stage1 = _one("bwd", ["sim_generic_kernel", "softmax_bwd_generic_kernel", "agg_generic_kernel"], K, s, W, dtype_name, B, H)
    return stage1 + [expected_gath(K, s, W, dtype_name)] * 2


def expected_sim(K, s, W, dtype_name, B=1, H=1):
    return _one("sim", ["sim_generic_kernel"], K, s, W, dtype_name, B, H)


def expected_agg(K, s, W, dtype_name, B=1, H=1):
    return _one("agg", ["agg_generic_kernel"], K, s, W, dtype_name, B, H)
