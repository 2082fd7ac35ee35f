"""Float32 layers on the tensor cores (pairs of fp16 values) at the edges of their tiles, against 64-bit arithmetic."""
import pytest
import torch
import torch.nn.functional as F

from m2_b200 import ops
from tests.helpers import Cfg, build_mixer
from tests.golden import cases as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rand(*shape, seed=1, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (scale * torch.randn(shape, generator=g)).to(DEV)


def error(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


@pytest.fixture(autouse=True)
def _status():
    yield
    torch.cuda.synchronize()
    assert ops.device_status() == 0


# A pair is within 2^-23 of a value and the four accumulations of the large terms of 64 products drop up to 2^-23 of their sum
# each, half of it on average and towards zero: 2^-23 (1 + 4 / 2 * the mean size of the partial sums, 0.77) at most, and less as
# pairs err in both directions.  A float32 chain of k products is at 2^-24 sqrt(k / 3).
LIMIT = 2 ** -22


@pytest.mark.parametrize("B,L,K,N", [(1, 1, 128, 1), (1, 127, 132, 8), (1, 129, 128, 65), (3, 43, 188, 130), (1, 64, 768, 2304), (2, 300, 196, 33),
                                     (5, 401, 260, 257), (8, 128, 768, 768), (4, 512, 1536, 768), (1, 20000, 128, 136)])
@pytest.mark.parametrize("bias", [True, False])
def test_linear(B, L, K, N, bias):
    x, w, b = rand(B, L, K), rand(N, K, seed=2), rand(N, seed=3) if bias else None
    ws = ops.split_weights(w)
    ref = F.linear(x.double(), w.double(), b.double() if bias else None)
    y = ops.linear_fwd(x, w, b, w_split=ws)
    assert error(y, ref) < LIMIT
    assert min(B * L, N) < 8 or error(y, ref) < error(ops.linear_fwd(x, w, b), ref)
    for out in (torch.full((B, L, N + 3), float("nan"), device=DEV)[..., :N],
                torch.full((B, N, L + 1), float("nan"), device=DEV)[..., :L].transpose(1, 2)):      # odd strides, time-contiguous
        assert torch.equal(ops.linear_fwd(x, w, b, out=out, w_split=ws), y)
        assert torch.isnan(out._base[..., -1]).all()
    # rows that TMA cannot take, tokens that are not evenly apart: the float32 chain
    odd = torch.empty((B, L, K + 1), device=DEV)[..., :K].copy_(x)
    assert torch.equal(ops.linear_fwd(odd, w, b, w_split=ws), ops.linear_fwd(x, w, b))


@pytest.mark.parametrize("m,nb,p,q", [(1, 2, 128, 4), (65, 2, 132, 66), (200, 3, 164, 130), (2048, 4, 768, 192), (1000, 4, 192, 1536), (129, 2, 384, 200)])
def test_blockdiag_and_glu(m, nb, p, q):
    x, w, b = rand(m, nb * p), rand(nb, q, p, seed=2, scale=p ** -0.5), rand(nb * q, seed=3)
    ws = ops.split_weights(w)
    g = torch.einsum("mkp,kqp->mkq", x.double().view(m, nb, p), w.double()).reshape(m, nb * q)
    assert error(ops.blockdiag_fwd(x, w, b, nb * p, nb * q, w_split=ws), g + b.double()) < LIMIT
    if nb % 2 == 0:
        i = nb * q // 2
        ref = F.gelu(g[:, :i]) * g[:, i:]
        y, chain = ops.blockdiag_glu_fwd(x, w, i, w_split=ws), ops.blockdiag_glu_fwd(x, w, i)
        assert error(y, ref) < 4 * LIMIT               # erff and the products of the GELU add roundings of their own
        assert m < 8 or error(y, ref) < error(chain, ref)


def test_values_of_any_size():
    """Infinities and rows beyond 2^90 give what the float32 chain gives; NaNs stay in their rows and columns; scales do not matter."""
    x, w, b = rand(1, 300, 768), rand(260, 768, seed=2), rand(260, seed=3)
    x[0, 5, 7], x[0, 6, 8], x[0, 7, 9] = float("inf"), float("nan"), 1e30
    x[0, 8] *= 1e-30
    x[0, 9], x[0, 10, 64:128] = 0.0, 0.0
    w[9], w[11, 3], w[12], w[13] = w[9] * 1e30, float("-inf"), w[12] * 1e-20, 0.0
    y, ref = ops.linear_fwd(x, w, b, w_split=ops.split_weights(w)), ops.linear_fwd(x, w, b)
    assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isinf(y), torch.isinf(ref))
    fin = torch.isfinite(ref)
    # both sides within 2^-24 sqrt(768) of the sum of 768 products of the largest row and column values
    size = x.nan_to_num(0, 0, 0).abs().sum(-1, keepdim=True) * w.nan_to_num(0, 0, 0).abs().amax(-1) + b.abs()
    assert ((y - ref).abs()[fin] <= 2 ** -18 * size[fin]).all()


@pytest.mark.parametrize("B,L", [(1, 1), (3, 37), (8, 128), (2, 500)])
def test_modules(B, L):
    """One native call and single launches are the same kernels; the whole model too."""
    from m2_b200 import BertGatedLinearUnitMLP
    from m2_b200.encoder import M2BertConfig, M2BertModel
    torch.manual_seed(L)
    mixer, _ = build_mixer(dict(C.CASES["mixer_small"], L=L, l_max=L, D=256, B=B, order=32, residual=True, seed=7), DEV)
    mlp = BertGatedLinearUnitMLP(Cfg(hidden_size=256, intermediate_size=512, monarch_mlp_nblocks=4, layer_norm_eps=1e-12, hidden_dropout_prob=0.0)).eval().to(DEV)
    model = M2BertModel(M2BertConfig(vocab_size=96, hidden_size=256, intermediate_size=512, num_hidden_layers=2, max_position_embeddings=512,
                                     long_conv_l_max=512, hyena_filter_order=16)).eval().to(DEV)
    u, ids = rand(B, L, 256), torch.randint(0, 96, (B, L), device=DEV)

    def run():
        with torch.no_grad():
            return mixer(u)[0], mlp(u), mlp(u.transpose(0, 1)).transpose(0, 1), model(ids)[0]
    whole = run()
    assert [m._plans.plans for m in (mixer, mlp, model)] and model._plans.plans
    ops.NVTX = True                                  # watched launches are made one by one
    try:
        single = run()
    finally:
        ops.NVTX = False
    assert all(torch.equal(a, b) for a, b in zip(whole, single))
    with torch.no_grad():
        mixer.in_linear.weight.mul_(0.5)             # the split weights are made again
        after = mixer(u)[0]
        assert not torch.equal(after, whole[0])
        mixer.in_linear.weight = torch.nn.Parameter(2 * mixer.in_linear.weight)
        assert torch.equal(mixer(u)[0], whole[0])


@pytest.mark.parametrize("m,nb,p,q", [(2048, 4, 192, 1536), (2048, 4, 768, 192), (2048, 2, 384, 768), (100, 2, 320, 64)])
def test_many_tiles_a_block(m, nb, p, q):
    """Launches right behind one another, several tiles to a thread block, K blocks in odd and even numbers: the same bits every time."""
    x, w = rand(m, nb * p), rand(nb, q, p, seed=2, scale=p ** -0.5)
    ws = ops.split_weights(w)
    for f in (lambda: ops.blockdiag_fwd(x, w, None, nb * p, nb * q, w_split=ws), lambda: ops.blockdiag_glu_fwd(x, w, nb * q // 2, w_split=ws)):
        y = [f() for _ in range(30)]
        assert all(torch.equal(t, y[0]) for t in y)


@pytest.mark.parametrize("T,K,N", [(1, 128, 8), (130, 132, 65), (300, 768, 2304), (2048, 1536, 768)])
def test_values_beside_one_another_of_any_size(T, K, N):
    """Columns of x times a power of two and the same columns of w by its inverse: every product is the same, and so is every bit."""
    x, w = rand(1, T, K), rand(N, K, seed=2)
    y = ops.linear_fwd(x, w, None, w_split=ops.split_weights(w))
    for spread in (12, 24, 40):
        e = torch.randint(-spread, spread + 1, (K,), generator=torch.Generator().manual_seed(spread)).to(DEV)
        xs, ws = torch.ldexp(x, e), torch.ldexp(w, -e)
        assert torch.equal(ops.linear_fwd(xs, ws, None, w_split=ops.split_weights(ws)), y)
    g, h = rand(T, 4 * K), rand(4, 2 * K, K, seed=2, scale=K ** -0.5)
    e = torch.randint(-40, 41, (4, K), generator=torch.Generator().manual_seed(5)).to(DEV)
    gs, hs = torch.ldexp(g.view(T, 4, K), e).view(T, 4 * K), torch.ldexp(h, -e[:, None])
    assert torch.equal(ops.blockdiag_glu_fwd(gs, hs, 4 * K, w_split=ops.split_weights(hs)),
                       ops.blockdiag_glu_fwd(g, h, 4 * K, w_split=ops.split_weights(h)))


# Operands of one sign: every truncation goes the same way, 2^-23 of a quarter, a half, three quarters and all of the sum of 64
# products, what the small terms and the additions in float32 add is below 1.5 * 2^-23 together.
@pytest.mark.parametrize("K", [128, 768, 1536])
def test_one_sign(K):
    x, w = rand(1, 256, K).abs(), rand(256, K, seed=2).abs()
    ref = F.linear(x.double(), w.double())
    assert error(ops.linear_fwd(x, w, None, w_split=ops.split_weights(w)), ref) < 2 ** -21


def test_the_largest_values():
    """Finite values that bf16 rounds to infinity, sums that overflow on the way: the float32 chain's result."""
    x, w = rand(1, 200, 256), rand(136, 256, seed=2)
    x[0, 3, 5], x[0, 150, 70], w[7, 9], w[130, 200] = 3.4028234e38, -3.4e38, 3.4028e38, -3.401e38
    x[0, 9], w[9] = x[0, 9] * 1e19, w[9] * 1e19
    for wz in (w, torch.zeros_like(w)):
        y, ref = ops.linear_fwd(x, wz, None, w_split=ops.split_weights(wz)), ops.linear_fwd(x, wz, None)
        assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isinf(y), torch.isinf(ref))
        for rows in ((3,), (150,)):
            assert torch.equal(y[0, rows], ref[0, rows])
        assert torch.equal(y[..., (7, 130)], ref[..., (7, 130)])


def test_calls_in_one_launch_are_planned():
    """What test_modules compares as one native call did run as one."""
    from m2_b200 import BertGatedLinearUnitMLP
    mlp = BertGatedLinearUnitMLP(Cfg(hidden_size=256, intermediate_size=512, monarch_mlp_nblocks=4, layer_norm_eps=1e-12, hidden_dropout_prob=0.0)).eval().to(DEV)
    mixer, _ = build_mixer(dict(C.CASES["mixer_small"], L=40, l_max=40, D=256, B=2, order=32, residual=True, seed=7), DEV)
    with torch.no_grad():
        mlp(rand(2, 40, 256)), mixer(rand(2, 40, 256))
    assert mlp._plans.plans and mixer._plans.plans


@pytest.mark.parametrize("exponent", [-99, -108, -118, -124])
def test_the_smallest_values(exponent):
    """Parts below the range of bf16: results below 2^-100 are the float32 chain's, those above keep its accuracy; zeros stay zeros."""
    x, w, g = rand(1, 200, 256), rand(136, 256, seed=2), rand(4, 128, 256, seed=3)
    x[0, 40] = 0.0
    xs = x * 2.0 ** exponent
    y, ref = ops.linear_fwd(xs, w, None, w_split=ops.split_weights(w)), ops.linear_fwd(xs, w, None)
    small = y.abs() < 2.0 ** -100
    assert torch.equal(y[small], ref[small]) and small[0, 40].all() and (small.all() or exponent > -108)
    assert error(y * 2.0 ** 90, F.linear(xs.double() * 2.0 ** 90, w.double())) < 2 ** -24 * (256 / 3) ** 0.5     # a chain of 256 products
    if exponent < -110:                              # every result is that small: sums of 256 products below 2^-110
        h = rand(200, 1024, seed=4) * 2.0 ** exponent
        assert torch.equal(ops.blockdiag_fwd(h, g, None, 1024, 512, w_split=ops.split_weights(g)), ops.blockdiag_fwd(h, g, None, 1024, 512))
