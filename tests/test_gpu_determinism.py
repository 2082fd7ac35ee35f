"""Race and bounds checks without a sanitizer: every launching entry point is run twice on the same inputs into
output buffers that sit inside a larger allocation filled with a canary pattern; the two results must be equal bit
for bit (a data race or an uninitialised read shows up as a difference sooner or later) and the canaries before
and after the output must be untouched (an out-of-bounds write shows up there).  Needs a B200."""
import ctypes as C_

import pytest
import torch

from m2_b200 import _lib, ops
from m2_b200.encoder import M2BertConfig, M2BertModel
from tests.golden import cases as C
from tests.helpers import build_glu, build_mixer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GUARD = 4096          # elements of canary on each side


def guarded(shape, dtype):
    """A tensor of `shape` carved out of a larger canary-filled buffer; returns (view, check)."""
    n = 1
    for d in shape:
        n *= d
    raw = torch.empty(n + 2 * GUARD, dtype=torch.int16 if dtype in (torch.bfloat16, torch.float16) else torch.int32, device=DEV)
    raw.fill_(0x5A5A if raw.dtype == torch.int16 else 0x5A5A5A5A)
    view = raw[GUARD:GUARD + n].view(dtype).view(*shape)

    def check():
        pat = 0x5A5A if raw.dtype == torch.int16 else 0x5A5A5A5A
        assert bool((raw[:GUARD] == pat).all()) and bool((raw[GUARD + n:] == pat).all()), "canary overwritten"
    return view, check


def twice(run, shape, dtype):
    outs = []
    for _ in range(2):
        out, check = guarded(shape, dtype)
        run(out)
        torch.cuda.synchronize()
        check()
        outs.append(out.clone())
    assert torch.equal(outs[0].view(torch.int16 if dtype != torch.float32 else torch.int32),
                       outs[1].view(torch.int16 if dtype != torch.float32 else torch.int32))
    assert ops.device_status() == 0
    return outs[0]


@pytest.mark.parametrize("B,L,K,N,mode", [(64, 128, 256, 768, "rows"), (64, 128, 256, 768, "channels"), (3, 1000, 256, 256, "timein"),
                                          (5, 136, 64, 200, "rows")])
def test_linear_fwd_is_deterministic_and_stays_in_bounds(B, L, K, N, mode):
    g = torch.Generator(device="cpu").manual_seed(1)
    x = torch.randn((B, L, K), generator=g).to(DEV).bfloat16()
    w = (torch.randn((N, K), generator=g) / K ** 0.5).to(DEV).bfloat16()
    b = torch.randn((N,), generator=g).to(DEV)
    with torch.no_grad():
        if mode == "rows":
            twice(lambda out: ops.linear_fwd(x, w, b, out=out), (B, L, N), torch.bfloat16)
        elif mode == "channels":
            twice(lambda out: ops.linear_fwd(x, w, b, out=out.permute(1, 2, 0)), (N, B, L), torch.bfloat16)
        else:
            xt = x.permute(0, 2, 1).contiguous()
            twice(lambda out: ops.linear_fwd(xt.permute(0, 2, 1), w, b, out=out), (B, L, N), torch.bfloat16)


@pytest.mark.parametrize("L,D,B,kind", [(128, 16, 130, 3), (2048, 16, 2, 2), (8192, 8, 2, 2), (32768, 4, 1, 2), (300, 8, 3, 2), (128, 128, 3, 1)])
def test_longconv_is_deterministic_and_stays_in_bounds(L, D, B, kind):
    cfg = dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=B, order=32, residual=True, seed=72)
    m, _ = build_mixer(cfg, DEV)
    g = torch.Generator(device="cpu").manual_seed(L)
    filters = [m.filter_fn, m.filter_fn2]
    with torch.no_grad():
        u = torch.randn((B, L, D), generator=g).to(DEV)
        if kind == 3:
            xin_t = (0.6 * torch.randn((3 * D, B, L), generator=g)).to(DEV).bfloat16()
            u_t = ops.time_major_f16(u)
            specs = [f.spectrum(L, True, 3) for f in filters]
            twice(lambda out: ops.longconv_fwd(xin_t.permute(1, 2, 0), u_t.permute(1, 2, 0), m.short_filter.weight, m.short_filter.bias,
                                               specs, None, kind=3, bf16_rounding=True, out=out.permute(1, 2, 0)), (D, B, L), torch.bfloat16)
        elif kind == 2:
            xin_t = (0.6 * torch.randn((B, 3 * D, L), generator=g)).to(DEV).bfloat16()
            u_t = u.transpose(1, 2).contiguous()
            specs = [f.spectrum(L, True, 2) for f in filters]
            twice(lambda out: ops.longconv_fwd(xin_t.transpose(1, 2), u_t.transpose(1, 2), m.short_filter.weight, m.short_filter.bias,
                                               specs, [f.conv_bias() for f in filters], kind=2, bf16_rounding=True,
                                               out=out.transpose(1, 2)), (B, D, L), torch.bfloat16)
        else:
            xin = (0.6 * torch.randn((B, L, 3 * D), generator=g)).to(DEV).bfloat16()
            specs = [f.spectrum(L, True, 1) for f in filters]
            twice(lambda out: ops.longconv_fwd(xin, u, m.short_filter.weight, m.short_filter.bias, specs,
                                               [f.conv_bias() for f in filters], kind=1, bf16_rounding=True, out=out), (B, L, D), torch.bfloat16)


def test_mlp_kernels_are_deterministic():
    g = torch.Generator(device="cpu").manual_seed(2)
    M, D, I = 1000, 768, 3072
    x = torch.randn((M, D), generator=g).to(DEV).bfloat16()
    wg = (torch.randn((4, 2 * I // 4, D // 4), generator=g) / (D // 4) ** 0.5).to(DEV).bfloat16()
    wo = (torch.randn((4, D // 4, I // 4), generator=g) / (I // 4) ** 0.5).to(DEV).bfloat16()
    bo = torch.randn((D,), generator=g).to(DEV)
    lw, lb = torch.ones(D, device=DEV), torch.zeros(D, device=DEV)
    with torch.no_grad():
        for variant in (0, 1, 3):
            a, b = (ops.blockdiag_glu_fwd(x, wg, I, variant=variant) for _ in range(2))
            assert torch.equal(a, b)
        h = ops.blockdiag_glu_fwd(x, wg, I)
        for variant in (0, 2):
            a, b = (ops.blockdiag_fwd(h, wo, bo, I, D, variant=variant) for _ in range(2))
            assert torch.equal(a, b)
        o = ops.blockdiag_fwd(h, wo, bo, I, D)
        a, b = (ops.add_layernorm_fwd(o, x, lw, lb, 1e-12, torch.float32) for _ in range(2))
        assert torch.equal(a, b)
    assert ops.device_status() == 0


def native(fn, args):
    assert fn(C_.byref(args), torch.cuda.current_stream().cuda_stream) == 0, _lib.lib().m2_last_error()


@pytest.mark.parametrize("L,D,B,kind", [(1, 8, 3, 4), (100, 256, 3, 4), (128, 768, 12, 4), (300, 64, 5, 4), (1024, 64, 9, 4), (100, 128, 70, 3),
                                        (7, 24, 50, 3), (132, 64, 2, 2)])
def test_time_contiguous_families_on_padded_rows(L, D, B, kind):
    """Kinds 2, 3 and 4 on rows of a pitch beyond seq_len: what lies between two rows is in the guarded buffer too."""
    m, _ = build_mixer(dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=B, order=32, residual=True, seed=73), DEV)
    g = torch.Generator(device="cpu").manual_seed(L)
    Lp = (L + 7) // 8 * 8 + 8
    filters = [m.filter_fn, m.filter_fn2]
    xin = torch.full((3 * D, B, Lp), float("nan"), dtype=torch.bfloat16, device=DEV)
    xin[:, :, :L] = (0.6 * torch.randn((3 * D, B, L), generator=g)).to(DEV).bfloat16()
    u = torch.full((D, B, Lp), float("nan"), dtype=torch.float16, device=DEV)
    u[:, :, :L] = torch.randn((D, B, L), generator=g).to(DEV).half()

    def run(out):
        out.fill_(7.0)
        ops.longconv_fwd(xin[:, :, :L].permute(1, 2, 0), u[:, :, :L].permute(1, 2, 0), m.short_filter.weight, m.short_filter.bias,
                         [f.spectrum(L, True, kind) for f in filters], [f.conv_bias() for f in filters] if kind == 2 else None, kind=kind,
                         bf16_rounding=True, out=out[:, :, :L].permute(1, 2, 0))
    with torch.no_grad():
        y = twice(run, (D, B, Lp), torch.bfloat16)
    assert (y[:, :, L:] == 7.0).all() and torch.isfinite(y).all()


@pytest.mark.parametrize("L,D,B", [(65, 256, 3), (128, 768, 1), (127, 256, 50), (128, 768, 64), (260, 256, 5), (2048, 256, 2)])
@pytest.mark.parametrize("packed", [True, False])
def test_mixer_fwd(L, D, B, packed):
    m, _ = build_mixer(dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=B, order=32, residual=True, seed=74), DEV)
    g = torch.Generator(device="cpu").manual_seed(L)
    kind = ops.longconv_pick(B, L, torch.bfloat16, D)
    Lp = (L + 7) // 8 * 8
    x = torch.full((B, Lp, D), float("nan"), dtype=torch.bfloat16, device=DEV)
    x[:, :L] = torch.randn((B, L, D), generator=g).to(DEV).bfloat16()
    u = ops.time_major_f16(x)
    plan = m._make_plan(B, L, kind, torch.device(DEV))

    def run(out):
        a = _lib.MixerArgs.from_buffer_copy(plan.args)
        work, check = guarded((4 * D, a.stride), torch.bfloat16)
        a.x, a.u, a.xin, a.conv, a.out = x.data_ptr(), u.data_ptr(), work.data_ptr(), work[3 * D:].data_ptr(), out.data_ptr()
        a.out_pitch = L if packed else Lp
        native(_lib.lib().m2_mixer_fwd, a)
        torch.cuda.synchronize()
        check()
        if not packed:
            out[:, L:] = 0                       # of padding steps, which hold anything
    with torch.no_grad():
        y = twice(run, (B, L if packed else Lp, D), torch.bfloat16)
    assert torch.isfinite(y).all()


@pytest.mark.parametrize("m,L", [(3, 3), (200, 8), (1000, 40), (4096, 128)])
def test_mlp_fwd(m, L):
    D, I = 768, 3072
    f, _ = build_glu(dict(kind="glu", seed=75, B=1, L=m, D=D, I=I, nb=4), DEV)
    x = torch.randn((m, D), generator=torch.Generator(device="cpu").manual_seed(m)).to(DEV).bfloat16()
    outs = {}

    def run(out):
        a = _lib.MlpArgs.from_buffer_copy(f._plan(torch.device(DEV)).args)
        h, check_h = guarded((m, I), torch.bfloat16)
        o, check_o = guarded((m, D), torch.bfloat16)
        rows, check_rows = guarded((m, D), torch.bfloat16)
        tm, check_tm = guarded((D, m), torch.float16)
        a.m, a.seq_len, a.x, a.h, a.o, a.out, a.out_bf16 = m, L, x.data_ptr(), h.data_ptr(), o.data_ptr(), out.data_ptr(), rows.data_ptr()
        if L % 8 == 0:
            a.out_tm_f16, a.tm_stride = tm.data_ptr(), m
        native(_lib.lib().m2_mlp_fwd, a)
        torch.cuda.synchronize()
        for check in (check_h, check_o, check_rows, check_tm):
            check()
        outs["rows"], outs["tm"] = rows, tm
    with torch.no_grad():
        y = twice(run, (m, D), torch.float32)
        assert torch.equal(outs["rows"], y.bfloat16()) and (L % 8 or torch.equal(outs["tm"], y.half().t()))


@pytest.mark.parametrize("B,L", [(1, 1), (3, 37), (1, 128), (2, 68), (50, 100), (64, 64), (2, 131), (2, 516), (1, 2048)])
def test_encoder_fwd(B, L):
    """The whole encoder in one call, and against the layers one by one: at these sizes the same kernels on the same values."""
    l_max = max(64, 1 << (L - 1).bit_length())
    torch.manual_seed(L)
    model = M2BertModel(M2BertConfig(vocab_size=96, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                                     max_position_embeddings=l_max, long_conv_l_max=l_max, hyena_filter_order=16)).eval().to(DEV)
    ids = torch.randint(0, 96, (B, L), device=DEV)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        plan = model._make_plan(B, L, torch.device(DEV))

        def run(out):
            work, check = guarded((plan.work // 4 + 64,), torch.float32)
            a = _lib.EncoderArgs.from_buffer_copy(plan.args)
            a.workspace, a.out, a.embed.input_ids = (work.data_ptr() + 255) // 256 * 256, out.data_ptr(), ids.data_ptr()
            native(_lib.lib().m2_encoder_fwd, a)
            torch.cuda.synchronize()
            check()
        y = twice(run, (B, L, 256), torch.float32)
        assert torch.equal(y, model(ids)[0])
        handle = model.encoder.register_forward_hook(lambda *a: None)
        single = model(ids)[0]
        handle.remove()
    assert torch.equal(y, single)
