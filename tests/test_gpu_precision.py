"""How far the convolution families are from 64-bit arithmetic, and that lengths which are computed in float32 are.

On the same bf16 in_linear output the families differ in what they hold in fp16: kind 0 nothing, kinds 3 and 4 taps and the
residual input, kinds 1 and 2 spectra and the signal between transform stages too."""
import pytest
import torch

from m2_b200 import ops
from m2_b200.encoder import M2BertConfig, M2BertModel
from tests.golden import cases as C
from tests.helpers import build_mixer

DEV = "cuda:0"


def test_float32_lengths_are_picked_float32():
    """Kind 0 wherever no tensor-core family serves rows of seq_len steps as they are; elsewhere never."""
    for D in (8, 192, 256, 768, 1536):
        for B in (1, 3, 47, 48, 63, 64, 200):
            for L in [*range(1, 140), 255, 256, 258, 511, 1000, 1001, 1023, 1024, 1531, 2044, 2047, 2048, 2049, 8190, 8192, 32767, 32768]:
                pick = ops.longconv_pick(B, L, torch.bfloat16, D)
                assert (pick == 0) == (ops.longconv_kind_batch(B, L, torch.bfloat16, D) == 0), (B, L, D, pick)
                assert ops.reads_time_major(B, L, D) == (pick != 0 and L % 8 == 0)


def mixer(L, D, B, seed=5):
    m, _ = build_mixer(dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=B, order=32, residual=True, seed=seed), DEV)
    g = torch.Generator().manual_seed(L)
    u = torch.nn.functional.layer_norm(torch.randn((B, L, D), generator=g), (D,)).to(DEV)
    xin = (0.6 * torch.randn((B, L, 3 * D), generator=g)).to(DEV).bfloat16()
    return m, xin, u


def exact(m, xin, u):
    """The middle of the mixer in float64 on the taps that every family is given, without any rounding on the way."""
    B, L, D = u.shape
    x = torch.nn.functional.conv1d(xin.double().transpose(1, 2), m.short_filter.weight.bfloat16().double(),
                                   m.short_filter.bias.bfloat16().double(), padding=2, groups=3 * D)[..., :L]
    x1, x2, v = x.split(D, 1)

    def conv(a, f):
        k = f.time_filter(L, True).double()
        n = k.shape[1]
        return torch.fft.irfft(torch.fft.rfft(a, n=n) * torch.fft.rfft(k, n=n), n=n)[..., :L] + a * f.bias.double()[:, None]
    return (conv(v * x1, m.filter_fn) * x2 + conv(u.double().transpose(1, 2), m.filter_fn2)).transpose(1, 2)


def run(m, kind, xin, u, time_contiguous=False):
    """One family; kind 0 on token rows, or (time_contiguous) its stage-by-stage kernel, which takes any layout."""
    B, L, D = u.shape
    filters = [m.filter_fn, m.filter_fn2]
    specs = [f.spectrum(L, True, kind) for f in filters]
    biases = None if kind in (3, 4) else [f.conv_bias() for f in filters]
    out = None
    if kind in (2, 3, 4):
        Lp = (L + 7) // 8 * 8
        rows = torch.empty((4 * D, B, Lp), dtype=torch.bfloat16, device=DEV)[:, :, :L].permute(1, 2, 0)
        tm = torch.empty((D, B, Lp), dtype=torch.float16, device=DEV)[:, :, :L]
        xin, u, out = rows[..., :3 * D].copy_(xin), ops.time_major_f16(u, out=tm).permute(1, 2, 0), rows[..., 3 * D:]
    elif time_contiguous:
        xin, u = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (xin, u))
    with torch.no_grad():
        return ops.longconv_fwd(xin, u, m.short_filter.weight, m.short_filter.bias, specs, biases, kind=kind, bf16_rounding=True, out=out)


def error(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


@pytest.mark.gpu
@pytest.mark.parametrize("L,D,B,kinds", [(37, 768, 3, (3, 4)), (64, 768, 8, (3, 4)), (100, 768, 8, (1, 3, 4)), (128, 768, 1, (1, 3, 4)),
                                         (128, 768, 64, (1, 3, 4)), (132, 768, 4, (2, 4)), (512, 768, 2, (2, 4)), (1024, 768, 2, (2, 4))])
def test_families_against_64_bits(L, D, B, kinds):
    m, xin, u = mixer(L, D, B)
    with torch.no_grad():
        ref = exact(m, xin, u)
        e = {k: error(run(m, k, xin, u), ref) for k in (0, *kinds)}
    print({k: "%.4e" % v for k, v in e.items()})
    # bf16 results: a rounding to nearest is off by at most 2^-9 of the value, and there are four on the way
    assert e[0] < 2 ** -8
    # the Toeplitz families (fp16 taps, no transform) are the nearest of those that hold anything in 16 bits, so a length that
    # moved to them from kind 1 or 2 lost nothing; they are measurably behind kind 0, whose lengths stay with it
    for k in kinds:
        if k in (3, 4):
            assert e[0] < e[k] < 1.03 * e[0]
            assert all(e[k] < e[j] for j in kinds if j in (1, 2))


@pytest.mark.gpu
@pytest.mark.parametrize("B,L,D", [(1, 1, 8), (2, 2, 9), (3, 5, 33), (2, 17, 768), (3, 37, 768), (1, 63, 65), (2, 127, 192), (3, 131, 40),
                                   (2, 513, 96), (6, 1531, 256), (1, 2047, 24), (1, 2048, 17)])
@pytest.mark.parametrize("u_dtype", [torch.float32, torch.bfloat16, None])
def test_float32_rows_against_the_stage_by_stage_kernel(B, L, D, u_dtype):
    """The register-pass kernel on bf16 rows: same butterflies, same rounding points.  Only the compiler's choice of which product
    of a sum goes into the FMA may differ: some 20 roundings of 2^-24 on each side, against a spacing of 2^-8 at three bf16
    roundings, flip about 3 * 2 * 20 * 2^-16 = 2e-3 of the results by one step (more where terms cancel: 1e-2 allowed)."""
    m, xin, u = mixer(L, D, B)
    wide = torch.full((B, L, D + 1), float("nan"), dtype=torch.bfloat16, device=DEV)

    def conv(x, v, out):
        f = [m.filter_fn, m.filter_fn2][:1 if u_dtype is None else 2]
        with torch.no_grad():
            return ops.longconv_fwd(x, v if u_dtype else None, m.short_filter.weight, m.short_filter.bias, [g.spectrum(L, True, 0) for g in f],
                                    [g.conv_bias() for g in f], kind=0, bf16_rounding=True, out=out)
    u = u.to(u_dtype or torch.float32)
    y = conv(xin, u, wide[..., :D])
    ref = conv(*(t.transpose(1, 2).contiguous().transpose(1, 2) for t in (xin, u)), None)
    assert torch.isnan(wide[..., D]).all()
    assert (y != ref).float().mean() < 1e-2 or y.numel() < 1000 and (y != ref).sum() < 3
    assert error(y, ref.double()) < 1e-2 ** 0.5 * 2 ** -8


@pytest.mark.gpu
@pytest.mark.parametrize("B,L", [(1, 1), (3, 37), (2, 64), (2, 131), (2, 514), (1, 1531)])
def test_whole_encoder_at_float32_lengths(B, L):
    """One native call and the layers one by one: the same kernels on the same values."""
    torch.manual_seed(L)
    l_max = max(64, 1 << (L - 1).bit_length())
    model = M2BertModel(M2BertConfig(vocab_size=96, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                                     max_position_embeddings=l_max, long_conv_l_max=l_max, hyena_filter_order=16)).eval().to(DEV)
    ids = torch.randint(0, 96, (B, L), device=DEV)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        whole = model(ids)[0]
        assert model._plans.plans and next(iter(model._plans.plans.values())).args.kind == 0
        handle = model.encoder.register_forward_hook(lambda *a: None)
        assert torch.equal(whole, model(ids)[0])
        handle.remove()
    assert ops.device_status() == 0


@pytest.mark.gpu
def test_mixer_takes_half_inputs_at_float32_lengths():
    m, _, u = mixer(37, 256, 2)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        assert torch.equal(m(u.half())[0], m(u.half().float())[0])


@pytest.mark.gpu
@pytest.mark.parametrize("kind,L,D,B", [(3, 128, 128, 64), (4, 128, 128, 2), (4, 128, 256, 40), (4, 128, 128, 64), (4, 256, 768, 8)])
def test_operands_beyond_fp16(kind, L, D, B):
    """v * x1 and the residual input saturate at 65504 in the Toeplitz families: nothing finite becomes Inf, whichever kernel the
    batch takes; where they stay below, the result is the float32 family's; and a NaN does not get lost."""
    m, xin, u = mixer(L, D, B)
    with torch.no_grad():
        m.short_filter.weight.zero_()
        m.short_filter.weight[:, 0, 2] = 1.0
        m.short_filter.bias.zero_()
    xin = xin.contiguous()
    # at step 5 the product of channel 0 is beyond fp16 and that of channel 1 just inside it
    xin[:, 5, 0], xin[:, 5, 2 * D] = 512.0, 256.0
    xin[:, 5, 1], xin[:, 5, 2 * D + 1] = 255.0, 256.0
    u[:, 7, 2] = 1e5                                      # saturates in the fp16 copy
    y, ref = run(m, kind, xin, u).float(), run(m, 0, xin, u).float()
    assert torch.isfinite(y).all() and torch.isfinite(ref).all()
    keep = [c for c in range(D) if c not in (0, 2)]
    # taps that differ by 2^-12 make some of the three bf16 roundings fall the other way, a step of 2^-8 of the value each; where
    # a few large steps make up a channel's norm all three may do so on them
    err = (y - ref)[..., keep].norm(dim=1) / ref[..., keep].norm(dim=1)
    assert err.max() < 3 * 2 ** -8
    xin[0, 5, 3] = float("nan")
    y = run(m, kind, xin, u).float()
    assert torch.isnan(y[0, :, 3]).any() and torch.isfinite(y[..., 4:]).all()
    assert ops.device_status() == 0
