"""The plans that modules keep per shape: when one may be used again (CPU), and that a forward through them sees every
change that the layer-by-layer path sees (GPU)."""
import copy
import pickle

import pytest
import torch
import torch.nn as nn

from m2_b200._plan import PlanCache, Watch, any_dropping, any_hooks
from m2_b200.encoder import M2BertConfig, M2BertModel


def net():
    return nn.Sequential(nn.Linear(4, 4), nn.LayerNorm(4))


def edit_in_place(m):
    with torch.no_grad():
        m[0].weight.mul_(2)


def new_parameter(m):
    m[0].weight = nn.Parameter(m[0].weight.detach().clone())


def new_storage(m):
    m[0].weight.data = m[0].weight.detach().clone()


def no_parameter(m):
    del m[0].bias


def new_module(m):
    m[0] = nn.Linear(4, 4)


def new_eps(m):
    m[1].eps = 1e-3


@pytest.mark.parametrize("change", [edit_in_place, new_parameter, new_storage, no_parameter, new_module, new_eps])
def test_watch_sees_changes(change):
    m = net()
    w = Watch(m)
    assert w.same()
    change(m)
    assert not w.same()


def test_plan_cache_is_bounded_and_drops_stale_plans():
    m, cache, made = net(), PlanCache(most=2), []

    def make():
        made.append(0)
        return len(made)
    assert [cache.get(m, k, make) for k in "aab"] == [1, 1, 2]
    assert cache.get(m, "c", make) == 3 and cache.get(m, "a", make) == 4       # "a" was dropped for "c"
    edit_in_place(m)
    assert cache.get(m, "c", make) == 5
    assert not copy.deepcopy(cache).plans and not pickle.loads(pickle.dumps(cache)).plans


def test_tensors_without_versions_get_no_plan():
    with torch.inference_mode():
        m = net()
    assert PlanCache().get(m, 0, dict) is None


def test_hooks_and_dropout_are_noticed():
    m = net()
    assert not any_hooks([m])
    h = m.register_forward_pre_hook(lambda *a: None)
    assert any_hooks([m])
    h.remove()
    m.forward = lambda x: x
    assert any_hooks([m])
    m.dropout = nn.Dropout(0.0)
    assert not any_dropping([m])
    m.dropout.p = 0.1
    assert any_dropping([m]) and not any_dropping([m.eval()])


@pytest.mark.gpu
def test_encoder_plan_follows_the_modules():
    torch.manual_seed(0)
    conf = M2BertConfig(vocab_size=96, hidden_size=256, intermediate_size=512, num_hidden_layers=2, max_position_embeddings=64,
                        long_conv_l_max=64)
    model = M2BertModel(conf).eval().cuda()
    ids = torch.randint(0, 96, (3, 37), device="cuda")

    def out():
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return model(ids)[0]

    def layer_by_layer():
        handle = model.encoder.register_forward_hook(lambda *a: None)
        y = out()
        handle.remove()
        return y
    first = out()
    assert torch.equal(first, out())
    del model._plans                              # as in a model pickled whole before there were plans
    assert torch.equal(first, out())
    layer = model.encoder.layer[1]
    for change in (lambda: layer.mlp.wo.bias.add_(1.0), lambda: layer.attention.filter_fn.bias.add_(1.0),
                   lambda: layer.attention.in_linear.weight.mul_(1.5), lambda: model.embeddings.word_embeddings.weight.mul_(-1.0)):
        before = out()
        with torch.no_grad():
            change()
        after, ref = out(), layer_by_layer()
        assert not torch.equal(before, after)
        # same kernels and rounding points; the padded rows only change which of two convolution families runs
        assert ((after - ref).norm() / ref.norm()).item() < 2e-2
    original = layer.forward
    layer.forward = lambda h, **kw: 2 * original(h)
    doubled = out()
    del layer.forward
    assert ((doubled - 2 * out()).norm() / doubled.norm()).item() < 2e-2
    with pytest.raises(RuntimeError), torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        model(torch.zeros((1, 65), dtype=torch.long, device="cuda"))
