"""Float32 modules compute with what their weights hold when the call (or the replay of a captured graph) runs."""
import pytest
import torch

from m2_b200 import BertGatedLinearUnitMLP, BlockdiagLinear, GraphedForward, ops
from m2_b200.encoder import M2BertConfig, M2BertModel
from tests.golden import cases as C
from tests.helpers import Cfg, build_mixer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
D, INTER, L = 512, 1024, 40


@pytest.fixture(autouse=True)
def _status():
    yield
    torch.cuda.synchronize()
    assert ops.device_status() == 0


def make(what):
    torch.manual_seed(3)
    if what == "mixer":
        m = build_mixer(dict(C.CASES["mixer_small"], L=L, l_max=L, D=D, B=2, order=32, residual=True, seed=7), DEV)[0]
        return m, m.in_linear.weight, torch.randn(2, L, D, device=DEV)
    if what == "mlp":
        m = BertGatedLinearUnitMLP(Cfg(hidden_size=D, intermediate_size=INTER, monarch_mlp_nblocks=4, layer_norm_eps=1e-12, hidden_dropout_prob=0.0)).eval().to(DEV)
        return m, m.gated_layers.weight, torch.randn(2, L, D, device=DEV)
    if what == "blockdiag":
        m = BlockdiagLinear(D, INTER, nblocks=4, bias=True).eval().to(DEV)
        return m, m.weight, torch.randn(2, L, D, device=DEV)
    m = M2BertModel(M2BertConfig(vocab_size=96, hidden_size=D, intermediate_size=INTER, num_hidden_layers=2, max_position_embeddings=64,
                                 long_conv_l_max=64, hyena_filter_order=16)).eval().to(DEV)
    return m, m.encoder.layer[1].mlp.wo.weight, torch.randint(0, 96, (2, L), device=DEV)


def call(m, x):
    with torch.no_grad():
        y = m(x)
    return y[0] if isinstance(y, tuple) else y


@pytest.mark.parametrize("what", ["mixer", "mlp", "blockdiag", "model"])
def test_writes_through_data(what):
    """A write that moves no version counter."""
    m, w, x = make(what)
    first = call(m, x).clone()
    w.data.mul_(3.0)
    fresh, w2, _ = make(what)
    with torch.no_grad():
        w2.mul_(3.0)
    y = call(m, x)
    assert not torch.equal(y, first) and torch.equal(y, call(fresh, x))


@pytest.mark.parametrize("what", ["mixer", "mlp", "blockdiag", "model"])
def test_graphs_read_the_weights(what):
    """A captured forward follows a weight that is changed in place, and holds all that it reads: calls in between free nothing of it."""
    m, w, x = make(what)
    g = GraphedForward(m, x, autocast=False, warmup=1)
    out = lambda: (lambda y: y[0] if isinstance(y, tuple) else y)(g(x)).clone()
    assert torch.equal(out(), call(m, x))
    with torch.no_grad():
        w.mul_(3.0)
    after = call(m, x)
    junk = [torch.full((n,), float("nan"), device=DEV) for n in (1 << 12, 1 << 16, 1 << 18, 1 << 20) for _ in range(8)]
    assert torch.equal(out(), after) and len(junk)


def test_parametrized_weights_do_not_stop_the_host(monkeypatch):
    from torch.nn.utils import parametrize

    class Twice(torch.nn.Module):
        def forward(self, w):
            return 2 * w
    m, w, x = make("mlp")
    with torch.no_grad():
        w.mul_(2.0)
    want = call(m, x)
    m, _, _ = make("mlp")
    parametrize.register_parametrization(m.gated_layers, "weight", Twice())

    def stop(self):
        raise AssertionError("the host waits for the stream")
    monkeypatch.setattr(torch.cuda.Stream, "synchronize", stop)
    assert torch.equal(call(m, x), want) and torch.equal(call(m, x), want)


def test_layers_keep_no_copies():
    m, _, x = make("mlp")
    before = torch.cuda.memory_allocated()
    call(m, x)
    assert torch.cuda.memory_allocated() - before < sum(4 * p.numel() for p in m.parameters()) // 2
