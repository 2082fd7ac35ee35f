"""Float32 kernels at the edges of their tiles, against the one-element kernels that take what they do not (strides that are
no multiple of four elements, time-contiguous rows) and against 64-bit arithmetic."""
import pytest
import torch

from m2_b200 import ops
from tests.golden import cases as C
from tests.helpers import build_mixer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rand(*shape, seed=1, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (scale * torch.randn(shape, generator=g)).to(DEV)


@pytest.mark.parametrize("B,L,D", [(1, 1, 1), (2, 2, 9), (1, 3, 33), (3, 8, 40), (2, 13, 8), (2, 33, 16), (1, 64, 65), (8, 128, 768), (2, 129, 24),
                                   (1, 511, 20), (4, 512, 96), (1, 1000, 12), (1, 1025, 10), (1, 2047, 8), (1, 2048, 17)])
@pytest.mark.parametrize("residual", [True, False])
def test_long_convolution(B, L, D, residual):
    m, _ = build_mixer(dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=B, order=32, residual=residual, seed=17), DEV)
    xin, u = rand(B, L, 3 * D, scale=0.6), rand(B, L, D, seed=2)
    filters = [m.filter_fn] + ([m.filter_fn2] if residual else [])

    def run(x, v):
        wide = torch.full((B, L, D + 1), float("nan"), device=DEV)
        with torch.no_grad():
            ops.longconv_fwd(x, v if residual else None, m.short_filter.weight, m.short_filter.bias,
                             [f.spectrum(L, False, 0) for f in filters], [f.conv_bias() for f in filters], kind=0, bf16_rounding=False,
                             out=wide[..., :D])
        assert torch.isnan(wide[..., D]).all()
        return wide[..., :D].double()

    def along_time(t):
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    y, ref = run(xin, u), run(along_time(xin), along_time(u))
    # 2 lg(2L) + 6 float32 roundings on each side, each below 2^-24 of the values' norm
    assert (y - ref).norm() / ref.norm() < 2 ** -24 * 2 * (2 * max(1, L).bit_length() + 8), (y - ref).norm() / ref.norm()
