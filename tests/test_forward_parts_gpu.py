"""The float32 forward through scratch in place of the attention map: as much of it as there is, in parts, and none."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(seed, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype).to(DEV)


def _part(q, k, v, out, scratch, B, d, C, H, W, begin, end, halo=0, image_rows=0):
    from sapa_b200 import _lib
    _lib.call("sapa_fused_forward_part", out.device, q, k, v, out, None, scratch, 0 if scratch is None else scratch.numel(), B, d, C, H, W, halo, halo,
              begin, end, image_rows, 5, 2, _lib.dtype_code(out))


def test_parts_equal_the_whole():
    """Scratch of all images, some, one, an even and an odd number of rows, two rows; bands of rows of their own."""
    from sapa_b200 import _lib
    from sapa_b200.functions import fused_forward_raw
    B, d, C, H, W = 5, 33, 130, 37, 76
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, scale=0.5), _rand(2, B, d, H, W, scale=0.5), _rand(3, B, C, H, W)
    whole = fused_forward_raw(q, k, v, 5, 2, True)[0]                # through the map that the backward wants
    assert torch.equal(fused_forward_raw(q, k, v, 5, 2, False)[0], whole)
    row = 25 * 4 * W * 4
    assert int(_lib.lib().sapa_fused_forward_scratch(B, d, C, H, W, H, 5, 2, 0)) == B * H * row
    for nbytes in (B * H * row, 3 * H * row + 100, H * row, H * row - 4, 11 * row, 2 * row):
        scratch = torch.full((nbytes,), 255, dtype=torch.uint8, device=DEV)          # NaN
        for bands in (((0, H),), ((0, 5), (5, 30), (30, H))):
            out = torch.empty_like(whole)
            for begin, end in bands:
                _part(q, k, v, out, scratch, B, d, C, H, W, begin, end)
            assert torch.equal(out, whole), (nbytes, bands)
    out = torch.empty_like(whole)
    for scratch in (None, torch.empty(2 * row - 16, dtype=torch.uint8, device=DEV)):      # too little: the kernel that needs none
        _part(q, k, v, out, scratch, B, d, C, H, W, 0, H)
        assert float((out.double() - whole.double()).norm() / whole.double().norm()) < 4e-6      # two kernels, 2e-6 each from float64
    assert _lib.wait_timeout_flags(DEV) == 0


def test_scratch_is_bounded():
    import sapa_b200 as sp
    B, d, C, H, W = 4, 4, 48, 512, 512
    q, k, v = _rand(1, B, d, 2 * H, 2 * W), _rand(2, B, d, H, W), _rand(3, B, C, H, W)
    with torch.no_grad():
        sp.sapa_fused(q, k, v, 5, 2)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        out = sp.sapa_fused(q, k, v, 5, 2)
        assert torch.cuda.max_memory_allocated() - before <= out.numel() * 4 + (256 << 20) + (1 << 20)      # the map has 420 MB


def test_a_call_that_just_fits():
    """Memory for the output and little more (the map has 118 MB): the kernel that needs no scratch."""
    import sapa_b200 as sp
    B, d, C, H, W = 8, 16, 64, 192, 192
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, scale=0.5), _rand(2, B, d, H, W, scale=0.5), _rand(3, B, C, H, W)
    with torch.no_grad():
        want = sp.sapa_fused(q, k, v, 5, 2).cpu()
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + want.numel() * 4 + (40 << 20)) / total)
        try:
            out = sp.sapa_fused(q, k, v, 5, 2)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
    assert float((out.cpu().double() - want.double()).norm() / want.double().norm()) < 4e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(64, 8, 8, 512), (96, 8, 200, 64), (72, 8, 2800, 512)], ids=lambda s: "C%d_d%d_%dx%d" % s)
def test_a_slab_goes_the_way_of_its_image(shape, dtype):
    """Flat and tall images, which a slab by itself would take for square ones: told the image's height, its bits are the image's."""
    from sapa_b200 import _lib
    from sapa_b200.functions import fused_forward_raw
    C, d, H, W = shape
    if dtype == torch.float32:
        flat = H * 4 < W                  # two launches do not pay for a few rows
        assert _lib.lib().sapa_fused_forward_wants_map(1, d, C, H, W, 5, 2, 0) == (0 if flat else 1 if W * W * C >= 5e5 else 0)
    q, k, v = _rand(1, 1, d, 2 * H, 2 * W, scale=0.5, dtype=dtype), _rand(2, 1, d, H, W, scale=0.5, dtype=dtype), _rand(3, 1, C, H, W, dtype=dtype)
    whole = fused_forward_raw(q, k, v, 5, 2, False)[0]
    ran = set(_lib.last_kernels())
    if dtype == torch.bfloat16 and H * W * C > 1e8:
        assert ran == {"sapa_wide_16_kernel<fwd>"}
    for lo, rows in ((2, min(16, H - 4)), (H - 2 - min(16, H - 4), min(16, H - 4)), (3, 1), (4, 2)):
        hi, pad = slice(2 * lo, 2 * (lo + rows)), slice(lo - 2, lo + rows + 2)
        out = torch.empty(1, C, 2 * rows, 2 * W, dtype=dtype, device=DEV)
        nbytes = int(_lib.lib().sapa_fused_forward_scratch(1, d, C, rows, W, H, 5, 2, _lib.dtype_code(out)))
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=DEV) if nbytes else None
        _part(q[:, :, hi].contiguous(), k[:, :, pad].contiguous(), v[:, :, pad].contiguous(), out, scratch, 1, d, C, rows, W, 0, rows, halo=2, image_rows=H)
        assert torch.equal(out, whole[:, :, hi]) and (set(_lib.last_kernels()) == ran or "strip" not in _lib.last_kernels()[0])
