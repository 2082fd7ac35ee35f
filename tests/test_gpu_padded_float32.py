"""Float32 long convolution (kind 0) on padded time-contiguous rows of bf16 activations: tensor-core products of fp16 pairs, at the
edges of blocks, tiles of sequences and lengths, against 64-bit arithmetic and the CUDA-core transform on token rows."""
import pytest
import torch

from m2_b200 import ops
from tests.test_gpu_precision import DEV, error, exact, mixer

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status():
    yield
    torch.cuda.synchronize()
    assert ops.device_status() == 0


def conv(m, xin, u, padded, nf=2):
    """Padded rows with NaNs behind every sequence, or token rows."""
    B, L, D = xin.shape[0], xin.shape[1], xin.shape[2] // 3
    out = None
    if padded:
        Lp = (L + 7) // 8 * 8 + 8
        rows = torch.full((4 * D, B, Lp), float("nan"), dtype=torch.bfloat16, device=DEV)
        t = rows[:, :, :L].permute(1, 2, 0)
        t[..., :3 * D] = xin
        ub = torch.full((D, B, Lp), float("nan"), dtype=u.dtype, device=DEV)
        ub[:, :, :L] = u.permute(2, 0, 1)
        xin, u, out = t[..., :3 * D], ub[:, :, :L].permute(1, 2, 0), t[..., 3 * D:]
    f = [m.filter_fn, m.filter_fn2][:nf]
    with torch.no_grad():
        y = ops.longconv_fwd(xin, u if nf == 2 else None, m.short_filter.weight, m.short_filter.bias, [g.spectrum(L, True, 0) for g in f],
                             [g.conv_bias() for g in f], kind=0, bf16_rounding=True, out=out, rows_padded=padded)
    if padded:
        assert torch.isnan(rows[3 * D:, :, L:].float()).all()
    return y.clone()


@pytest.mark.parametrize("B,L,D", [(1, 1, 3), (9, 2, 8), (17, 7, 5), (130, 8, 4), (1, 37, 768), (8, 64, 300), (3, 127, 40), (129, 128, 2), (1, 129, 200),
                                   (7, 255, 8), (33, 256, 8), (2, 257, 149), (40, 300, 4), (3, 641, 16), (17, 1023, 8), (2, 1024, 160), (9, 1531, 8),
                                   (1, 1921, 5), (1, 2047, 8), (10, 2048, 6)])
@pytest.mark.parametrize("u_dtype", [torch.float32, torch.bfloat16, None])
def test_padded_rows(B, L, D, u_dtype):
    m, xin, u = mixer(L, D, B)
    u = u.to(u_dtype or torch.float32)
    y, ref = conv(m, xin, u, True, 2 if u_dtype else 1), conv(m, xin, u, False, 2 if u_dtype else 1)
    # both sides are within some 40 roundings of 2^-24 of the float32 results; with a spacing of 2^-8 at three bf16 roundings
    # 3 * 2 * 40 * 2^-16 = 4e-3 of the results may fall the other way, by a step (more where terms cancel: 1e-2 allowed)
    assert (y != ref).float().mean() < 1e-2 or (y != ref).sum() < 3
    assert error(y, ref.double()) < 1e-2 ** 0.5 * 2 ** -8
    if u_dtype == torch.float32 and y.numel() > 20000:
        with torch.no_grad():
            e, e0 = error(y, exact(m, xin, u)), error(ref, exact(m, xin, u))
        print("%.5e %.5e" % (e0, e))
        assert e < 1.001 * e0


def test_values_of_any_size():
    """Sequences are scaled one by one: their results do not depend on one another; what is not finite makes its row NaN, as in a transform."""
    m, xin, u = mixer(300, 16, 6)
    want = conv(m, xin, u, True)
    xin[1] *= 2.0 ** 40
    u[1] *= 2.0 ** 100
    xin[2] *= 2.0 ** -40
    u[3, 17, 2], xin[4, 5, 3], xin[5, 9, 32 + 4] = float("inf"), float("nan"), float("-inf")
    y, ref = conv(m, xin, u, True), conv(m, xin, u, False)
    assert torch.equal(y[0], want[0])
    assert torch.equal(torch.isfinite(y[:5]), torch.isfinite(ref[:5])) and not torch.isfinite(y[5, 9, 4]).any()
    for b in (1, 2):
        assert error(y[b], ref[b].double()) < 1e-2 ** 0.5 * 2 ** -8


@pytest.mark.parametrize("L", [129, 1531])
def test_exact_sums_stay_exact(L):
    """A filter of one tap, at values half way between two bf16 values: whatever scaled the sums would push them over."""
    m, xin, u = mixer(L, 8, 6)
    k = torch.zeros_like(m.filter_fn.time_filter(L, True))
    k[:, 0] = 1.0
    spec, zero = ops.filter_spectrum(k, L, 0), torch.zeros(8, device=DEV)
    u.copy_(1 + 2.0 ** -8)
    u[:, ::2].mul_(-1)
    rows = torch.zeros((4 * 8, 6, (L + 7) // 8 * 8), dtype=torch.bfloat16, device=DEV)
    t = rows[:, :, :L].permute(1, 2, 0)                       # the gate is zero: the residual convolution alone
    y = ops.longconv_fwd(t[..., :3 * 8], rows.new_zeros((8, 6, rows.shape[2]), dtype=torch.float32)[:, :, :L].copy_(u.permute(2, 0, 1)).permute(1, 2, 0),
                         m.short_filter.weight, torch.zeros_like(m.short_filter.bias), [spec, spec], [zero, zero], kind=0, bf16_rounding=True,
                         out=t[..., 3 * 8:], rows_padded=True)
    assert torch.equal(y.float(), u.sign())


@pytest.mark.parametrize("B,L", [(6, 1531), (40, 301)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_module_takes_padded_rows(B, L, dtype):
    """The mixer at lengths where it lays its rows out so: one call and single launches."""
    assert ops.longconv_padded(B, L, 256) and ops.longconv_pick(B, L, torch.bfloat16, 256) == 0
    m, _, u = mixer(L, 256, B)
    u = u.to(dtype)

    def run():
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return m(u)[0]
    y = run()
    ops.NVTX = True
    try:
        assert torch.equal(run(), y)
    finally:
        ops.NVTX = False
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        xin = torch.nn.functional.linear(u, m.in_linear.weight, m.in_linear.bias)
        ref = torch.nn.functional.linear(conv(m, xin.contiguous(), u, False), m.out_linear.weight, m.out_linear.bias)
    assert error(y, ref.double()) < 2e-2
