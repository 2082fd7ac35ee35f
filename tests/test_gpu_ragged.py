"""Convolution families on padded time-contiguous rows of any length: the block-Toeplitz family (kind 4), the Toeplitz family
(kind 3) and the long-row family (kind 2) at lengths that are no multiple of 8, against the float32 CUDA-core family.  What lies between a row's end
and the next row holds NaNs in the inputs and must stay untouched in the output.  Tolerance: the path's 2e-2 per operator
(bf16 rounding points shared by both families, one differing flip moves a value by 2^-8 of itself)."""
import pytest
import torch

from m2_b200 import ops
from tests.golden import cases as C
from tests.helpers import build_mixer
from tests.test_gpu_parity import TOL_BF16, flip_tolerant_error

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def run_both(kind, L, D, B, residual, u_dtype, seed):
    cfg = dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=B, order=32, residual=residual, seed=seed)
    m, _ = build_mixer(cfg, DEV)
    g = torch.Generator().manual_seed(L + B)
    Lp = (L + 7) // 8 * 8 + 8

    def rows(c, scale, dtype):
        t = torch.full((c, B, Lp), float("nan"), dtype=dtype, device=DEV)
        t[:, :, :L] = (scale * torch.randn((c, B, L), generator=g)).to(DEV).to(dtype)
        return t[:, :, :L].permute(1, 2, 0)
    xin, u = rows(3 * D, 0.6, torch.bfloat16), rows(D, 1.0, u_dtype)
    yu = u_dtype == torch.bfloat16
    filters = [m.filter_fn] + ([m.filter_fn2] if residual else [])
    biases = [f.conv_bias() for f in filters]
    out0 = torch.empty((D, B, L), dtype=torch.bfloat16, device=DEV).permute(1, 2, 0)
    u0 = u.bfloat16() if yu else u.float()
    with torch.no_grad():
        ops.longconv_fwd(xin.contiguous(), u0.contiguous() if residual else None, m.short_filter.weight, m.short_filter.bias,
                         [f.spectrum(L, True, 0) for f in filters], biases, kind=0, bf16_rounding=True, out=out0)
        buf = torch.full((D, B, Lp), float("nan"), dtype=torch.bfloat16, device=DEV)
        out = buf[:, :, :L].permute(1, 2, 0)
        ops.longconv_fwd(xin, u if residual else None, m.short_filter.weight, m.short_filter.bias,
                         [f.spectrum(L, True, kind) for f in filters], None if kind in (3, 4) else biases, kind=kind,
                         bf16_rounding=True, out=out, yu_bf16=yu)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.isnan(buf[:, :, L:].float()).all() and torch.isfinite(out.float()).all()
    return flip_tolerant_error(out, out0)


@pytest.mark.parametrize("L,D,B", [(1, 3, 2), (7, 8, 1), (16, 5, 17), (100, 8, 9), (128, 300, 3), (127, 8, 130), (128, 40, 128),
                                   (129, 8, 1), (256, 8, 65), (300, 24, 33), (384, 8, 40), (513, 8, 16), (640, 8, 20),
                                   (900, 8, 18), (1000, 320, 5), (1023, 8, 2), (1024, 8, 17)])
@pytest.mark.parametrize("residual,u_dtype", [(True, torch.float16), (True, torch.bfloat16), (False, torch.bfloat16)])
def test_block_toeplitz_family(L, D, B, residual, u_dtype):
    e = run_both(4, L, D, B, residual, u_dtype, 91)
    print("kind4-vs-kind0: %.3e" % e)
    assert e < TOL_BF16, e


@pytest.mark.parametrize("L", [1, 7, 8, 9, 15, 17, 33, 65, 100, 127, 128])
@pytest.mark.parametrize("B", [1, 48, 63, 129])
@pytest.mark.parametrize("residual", [True, False])
def test_toeplitz_family_at_any_length(L, B, residual):
    e = run_both(3, L, 16, B, residual, torch.float16, 94)
    print("kind3-vs-kind0: %.3e" % e)
    assert e < TOL_BF16, e


@pytest.mark.parametrize("L,D,B", [(131, 8, 2), (1531, 16, 3), (2045, 24, 2), (2049, 8, 2), (8191, 8, 3), (8193, 4, 1), (32767, 4, 1)])
@pytest.mark.parametrize("residual,u_dtype", [(True, torch.float16), (True, torch.bfloat16), (False, torch.bfloat16)])
def test_long_row_family_at_any_length(L, D, B, residual, u_dtype):
    e = run_both(2, L, D, B, residual, u_dtype, 92)
    print("kind2-vs-kind0: %.3e" % e)
    assert e < TOL_BF16, e
