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


def unaligned(x):
    """The same values in rows an odd number of elements apart."""
    buf = torch.empty((*x.shape[:-1], x.shape[-1] + 1), device=DEV)
    buf[..., :-1] = x
    return buf[..., :-1]


def near(y, ref, k):
    # k products of N(0, 1) numbers summed in float32: each rounding is below 2^-24 of a partial sum of size <= sqrt(k)
    err = (y.double() - ref).norm() / ref.norm()
    assert err < 2 ** -24 * max(4.0, k ** 0.5), err


@pytest.mark.parametrize("B,L,K,N", [(1, 1, 4, 1), (1, 64, 16, 64), (3, 43, 20, 65), (2, 64, 12, 128), (1, 129, 768, 190), (8, 128, 768, 2304),
                                     (5, 401, 64, 257), (4, 512, 1536, 768)])
def test_linear(B, L, K, N):
    x, w, b = rand(B, L, K), rand(N, K, seed=2), rand(N, seed=3)
    y = ops.linear_fwd(x, w, b)
    assert torch.equal(y, ops.linear_fwd(x, w, b, force_simt=True))
    near(y, torch.nn.functional.linear(x.double(), w.double(), b.double()), K)
    wide = torch.full((B, L, N + 3), float("nan"), device=DEV)
    ops.linear_fwd(x.transpose(0, 1).contiguous().transpose(0, 1), w, b, out=wide[..., :N])
    assert torch.equal(wide[..., :N], y) and torch.isnan(wide[..., N:]).all()


@pytest.mark.parametrize("m,nb,p,q", [(1, 2, 4, 4), (64, 4, 16, 64), (65, 2, 20, 66), (200, 3, 36, 130), (2048, 4, 768, 192), (1000, 4, 192, 1536)])
def test_blockdiag_and_glu(m, nb, p, q):
    x, w, b = rand(m, nb * p), rand(nb, q, p, seed=2), rand(nb * q, seed=3)
    y = ops.blockdiag_fwd(x, w, b, nb * p, nb * q)
    assert torch.equal(y, ops.blockdiag_fwd(unaligned(x), w, b, nb * p, nb * q))
    near(y, torch.einsum("mkp,kqp->mkq", x.double().view(m, nb, p), w.double()).reshape(m, nb * q) + b.double(), p)
    if nb % 2 == 0:
        h = ops.blockdiag_glu_fwd(x, w, nb * q // 2)
        assert torch.equal(h, ops.blockdiag_glu_fwd(unaligned(x), w, nb * q // 2))


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


@pytest.mark.parametrize("B,L,D", [(1, 1, 4), (2, 8, 8), (3, 65, 100), (2, 130, 768), (1, 63, 68), (2, 9, 7)])
@pytest.mark.parametrize("channels_contiguous", [True, False])
def test_row_copies(B, L, D, channels_contiguous):
    u = rand(B, L, D, scale=300.0)
    u[0, 0, 0] = 1e6                                     # saturates in fp16
    if not channels_contiguous:
        u = u.transpose(1, 2).contiguous().transpose(1, 2)
    Lp = (L + 7) // 8 * 8
    tm = torch.full((D, B, Lp), float("nan"), dtype=torch.float16, device=DEV)
    rows = torch.full((B, Lp, D), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.time_major_f16(u, out=tm[:, :, :L], rows=rows[:, :L])
    assert torch.equal(tm[:, :, :L], u.clamp(-65504, 65504).half().permute(2, 0, 1)) and torch.isnan(tm[:, :, L:]).all()
    assert torch.equal(rows[:, :L], u.bfloat16()) and torch.isnan(rows[:, L:]).all()
