"""What the modules hand to the one-call entry points (m2_mixer_fwd, m2_mlp_fwd, m2_encoder_fwd), which see pointers and sizes
and no tensors.  On the CPU with the launch replaced by a recorder: nothing here reaches a GPU."""
import copy
import ctypes
import dataclasses
import gc
import re
import weakref
from pathlib import Path

import pytest
import torch
import torch.nn as nn
from torch.nn.utils import parametrize

from m2_b200 import BertGatedLinearUnitMLP, MonarchMixerSequenceMixing, _lib, glu_mlp, ops, sequence_mixer
from m2_b200._plan import PlanCache, Watch, plans_of
from m2_b200.encoder import M2BertConfig, M2BertModel
from tests.helpers import Cfg

D, INTER = 256, 512


class CudaLike(torch.Tensor):
    """A CPU tensor that says it is on a GPU."""

    def __new__(cls, t):
        return t.as_subclass(cls)

    is_cuda = True


@pytest.fixture
def calls(monkeypatch):
    """Names of the launches that would have been made."""
    names = []
    monkeypatch.setattr(ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "_launch", lambda name, *a, **k: names.append(name))
    return names


def mixer(d=D):
    return MonarchMixerSequenceMixing(d, l_max=128, bidirectional=True, hyena_emb_dim=5, hyena_filter_order=16,
                                      residual_long_conv=True, hyena_kernel_lr=1e-3).eval()


def mlp(d=D, inter=INTER, nblocks=4):
    return BertGatedLinearUnitMLP(Cfg(hidden_size=d, intermediate_size=inter, monarch_mlp_nblocks=nblocks, layer_norm_eps=1e-12,
                                      hidden_dropout_prob=0.0)).eval()


def mix(m, u, kind=4):
    with torch.no_grad():
        return m._forward_bf16(u, u, kind)


def feed(m, x):
    with torch.no_grad():
        x2 = x.reshape(-1, x.shape[-1]).to(torch.bfloat16)
        return m._forward_bf16(x, x2, m._plan(x.device), False)


def test_right_widths_are_launched(calls):
    assert mix(mixer(), torch.zeros(2, 128, D)).shape == (2, 128, D) and calls[-1] == "m2_mixer_fwd"
    assert feed(mlp(), torch.zeros(2, 128, D)).shape == (2, 128, D) and calls[-1] == "m2_mlp_fwd"


@pytest.mark.parametrize("width", [D - 8, D + 8, 2 * D])
def test_another_width_is_refused(calls, width):
    with pytest.raises(AssertionError):
        mix(mixer(), torch.zeros(2, 128, width))
    with pytest.raises(AssertionError):
        feed(mlp(), torch.zeros(2, 128, width))
    assert not calls


@pytest.mark.parametrize("run,module,edit", [
    (mix, mixer, lambda m: setattr(m, "in_linear", nn.Linear(D, 3 * D - 3))),
    (mix, mixer, lambda m: setattr(m, "out_linear", nn.Linear(D - 1, D))),
    (mix, mixer, lambda m: setattr(m, "short_filter", nn.Conv1d(3 * D, 3 * D, 5, groups=3 * D))),
    (mix, mixer, lambda m: setattr(m, "filter_fn2", mixer(D // 2).filter_fn)),
    (feed, mlp, lambda m: setattr(m, "layernorm", nn.LayerNorm(D // 2)))])
def test_weights_of_another_shape_are_refused(calls, run, module, edit):
    m = module()
    edit(m)
    with pytest.raises(AssertionError):
        run(m, torch.zeros(2, 128, D))
    assert not {"m2_mixer_fwd", "m2_mlp_fwd"} & set(calls)


def test_the_weights_decide_the_width(calls):
    m = mixer()
    m.d_model = D // 2                               # nothing but the choice of a kernel family reads it
    assert mix(m, torch.zeros(2, 128, D)).shape == (2, 128, D)
    assert m._plans.plans.popitem()[1].args.d_model == D


@pytest.mark.parametrize("run,module", [(mix, mixer), (feed, mlp)])
def test_weights_on_another_device_are_refused(calls, run, module):
    with pytest.raises(RuntimeError, match="device"):
        run(module().to("meta"), torch.zeros(2, 128, D))
    assert not {"m2_mixer_fwd", "m2_mlp_fwd"} & set(calls)


def test_linear_layers_without_bias(calls):
    m, f = mixer(), mlp()
    m.in_linear, m.out_linear = nn.Linear(D, 3 * D, bias=False), nn.Linear(D, D, bias=False)
    f.wo.bias = None
    mix(m, torch.zeros(2, 128, D))
    feed(f, torch.zeros(2, 128, D))
    assert calls[-1] == "m2_mlp_fwd" and "m2_mixer_fwd" in calls
    a, b = m._make_plan(2, 128, 4, torch.device("cpu")).args, f._plan(torch.device("cpu")).args
    assert a.b_in is None and a.b_out is None and b.wo_bias is None and a.w_in and b.ln_b


@pytest.mark.parametrize("f", [lambda: mlp(inter=INTER + 2),      # wo.weight (4, 64, 129): 516 columns for 514 features
                               lambda: other_blocks(mlp(), "gated_layers"), lambda: other_blocks(mlp(), "wo")])
def test_weights_of_other_blocks_take_single_launches(calls, monkeypatch, f):
    monkeypatch.setattr(glu_mlp, "_compute_dtype", lambda x: torch.bfloat16)
    f, model = f(), small_model()
    with torch.no_grad():
        assert f(torch.zeros(2, 128, D)).shape == (2, 128, D)
    assert calls == ["m2_blockdiag_glu_fwd", "m2_blockdiag_fwd", "m2_add_layernorm_fwd"]
    model.encoder.layer[1].mlp = f
    assert model._make_plan(2, 128, torch.device("cpu")) is None


def other_blocks(f, name):
    setattr(f, name, getattr(mlp(nblocks=2), name))
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("f", [lambda: mlp(inter=INTER + 2), lambda: other_blocks(mlp(), "gated_layers"), lambda: other_blocks(mlp(), "wo")])
def test_mlp_with_other_blocks(f):
    torch.manual_seed(4)
    f, x = f().cuda(), torch.randn(3, 24, D, device="cuda")
    with torch.no_grad():
        want = f(x)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            got = f(x)
    # four bf16 roundings (input, weights, h, wo's output) of 2^-9 each on values that LayerNorm brings to 1
    assert (got - want).norm() / want.norm() < 4 * 2 ** -8


@pytest.mark.parametrize("L", [132, 256, 1024])
@pytest.mark.parametrize("d", [256, 768, 1536])
def test_family_4_is_not_picked_for_tensors_it_refuses(L, d):
    limit = 2 ** 33 // (3 * d * L)                   # sequences whose in_linear output the kernel's offsets can reach

    def pick(b):
        return ops.longconv_pick(b, L, torch.bfloat16, d)
    assert 4 in map(pick, range(1, 65)) and pick(limit + 1) == pick(2 * limit) == 2


def test_the_longest_unused_plan_is_dropped():
    m, cache, made = nn.Linear(2, 2), PlanCache(most=2), []
    for key in "hot", "x", "hot", "y", "hot":
        cache.get(m, key, lambda: made.append(key) or key)
    assert made == ["hot", "x", "y"]


def test_a_refusal_is_remembered_until_something_changes():
    m, cache, made = nn.Linear(2, 2), PlanCache(), []
    assert [cache.get(m, 0, lambda: made.append(0)) for _ in range(3)] == [None] * 3 and len(made) == 1
    m.weight = nn.Parameter(torch.zeros(2, 2))
    assert cache.get(m, 0, lambda: made.append(0)) is None and len(made) == 2


def test_other_tensors_on_a_module_do_not_matter():
    m = small_model()
    m.temperature = torch.ones(())
    assert Watch(m).same()
    m.encoder.layer[0].attention.in_linear._parameters.pop("bias")
    m.encoder.layer[0].attention.in_linear.bias = torch.zeros(3 * D)
    with pytest.raises(RuntimeError):
        Watch(m)


class Doubled(nn.Module):
    def forward(self, t):
        return 2 * t


def test_computed_parameters_are_held_for_the_call(calls):
    """A parametrized bias is another tensor on every access: its pointer is good while somebody holds that one."""
    m, f = mixer(), mlp()
    parametrize.register_parametrization(m.out_linear, "bias", Doubled())
    parametrize.register_parametrization(f.layernorm, "weight", Doubled())
    for plan, pointer in ((m._make_plan(2, 128, 4, torch.device("cpu")), "b_out"), (f._plan(torch.device("cpu")), "ln_w")):
        assert getattr(plan.args, pointer) in [t.data_ptr() for t in plan.held] and not plan.lasting
    mix(m, torch.zeros(2, 128, D))
    assert not plans(m) and not plans(f)


def test_replicas_have_plans_of_their_own(calls):
    m, u = mixer(), torch.zeros(2, 128, D)
    mix(m, u)
    replica = m._replicate_for_data_parallel()       # shares __dict__, its parameters become plain attributes
    for child in ("in_linear", "out_linear", "short_filter", "filter_fn", "filter_fn2"):
        replica._modules[child] = m._modules[child]._replicate_for_data_parallel()
        for k, t in m._modules[child]._parameters.items():
            setattr(replica._modules[child], k, t.detach().clone())
    for f in ("filter_fn", "filter_fn2"):
        replica._modules[f]._modules.update(m._modules[f]._modules)
    mix(replica, u)
    assert replica._plans is not m._plans and not plans(replica) and plans(m)
    assert "m2_linear_fwd" in calls[-3:]             # tensors that cannot be watched: single launches
    twin = copy.copy(m)
    mix(twin, u)
    assert twin._plans is not m._plans and m._plans.owner() is m and plans(m)


def small_model():
    return M2BertModel(M2BertConfig(vocab_size=8, hidden_size=D, intermediate_size=INTER, num_hidden_layers=2, hyena_filter_order=16)).eval()


SETTINGS = [(lambda m: setattr(m.encoder.layer[1].attention.filter_fn, "use_bias", False)),
            (lambda m: setattr(m.encoder.layer[0].attention, "residual_long_conv", False)),
            (lambda m: setattr(m.encoder.layer[0].attention, "hyena_training_additions", True)),
            (lambda m: setattr(m.encoder.layer[0].attention, "d_model", D // 2)),
            (lambda m: setattr(m.embeddings, "use_positional_encodings", False)),
            (lambda m: setattr(m.embeddings.LayerNorm, "eps", 0.5)),
            (lambda m: setattr(m.encoder.layer[1].mlp.layernorm, "eps", 0.5)),
            (lambda m: setattr(m.encoder.layer[0].mlp.config, "intermediate_size", INTER // 2)),
            (lambda m: setattr(m.encoder.layer[0].mlp, "config", dataclasses.replace(m.config, monarch_mlp_nblocks=2)))]


@pytest.mark.parametrize("change", SETTINGS)
def test_settings_that_plans_are_made_from_are_watched(change):
    m = small_model()
    w = Watch(m)
    assert w.same()
    change(m)
    assert not w.same()


def test_a_tensor_that_was_not_there_is_watched():
    m = nn.Linear(2, 2, bias=False)
    w = Watch(m)
    assert w.same()
    m.bias = nn.Parameter(torch.zeros(2))
    assert not w.same()


@pytest.mark.gpu
@pytest.mark.parametrize("L", [37, 72, 256])
@pytest.mark.parametrize("change", [SETTINGS[0], SETTINGS[4], SETTINGS[6],
                                    lambda m: [setattr(y.attention, "residual_long_conv", False) for y in m.encoder.layer]])
def test_planned_and_single_launches_agree_after_a_setting_changed(change, L):
    torch.manual_seed(6)
    m = M2BertModel(M2BertConfig(vocab_size=8, hidden_size=D, intermediate_size=INTER, num_hidden_layers=2, hyena_filter_order=16,
                                 max_position_embeddings=256, long_conv_l_max=256)).eval().cuda()
    ids = torch.randint(0, 8, (3, L), device="cuda")

    def out():
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return m(ids)[0]
    before = out()
    change(m)
    after = out()
    handle = m.encoder.register_forward_hook(lambda *a: None)
    single = out()
    handle.remove()
    assert not torch.equal(before, after) and torch.equal(after, single)


def test_the_next_kernel_is_let_in_after_tensor_memory_is_allocated():
    """Kernels that are launched while the one before them runs wait for it; one that holds tensor memory while the kernel
    before it still waits for some would never end.  Source order of allocation, block barrier and trigger."""
    seen = 0
    for path in sorted((Path(ops.__file__).parent / "csrc").glob("*.cu")):
        code = "\n".join(line.split("//")[0] for line in path.read_text().splitlines())
        for kernel in code.split("__global__")[1:]:
            alloc, trigger = re.search(r"tmem_alloc2?\(", kernel), re.search(r"pdl_(wait|trigger)\(\)", kernel)
            if alloc and trigger:
                seen += 1
                assert alloc.start() < trigger.start() and "__syncthreads()" in kernel[alloc.end():trigger.start()], path.name
    assert seen >= 6


@pytest.mark.gpu
def test_families_one_after_the_other_on_one_stream():
    """Short launches that overlap: kinds 4 and 2 and a GEMM in turn, each with tensor memory of its own."""
    from tests.test_gpu_precision import mixer as built, run as conv
    m, xin, u = built(132, 64, 2)
    w = torch.randn(192, 64, device="cuda").bfloat16()
    first = None
    for _ in range(20):
        y = [conv(m, 4, xin, u), conv(m, 2, xin, u), conv(m, 4, xin, u), ops.linear_fwd(u.bfloat16(), w, None), conv(m, 2, xin, u)]
        first = first or y
        assert all(torch.equal(a, b) for a, b in zip(first, y))
    assert ops.device_status() == 0


def test_shapes_of_token_type_ids():
    t = torch.arange(6, dtype=torch.int32)
    cpu = torch.device("cpu")
    assert ops.token_ids(None, 2, 3, cpu) is None
    for same in (t, t.view(2, 3), t.view(6, 1), t.view(2, 3).t().contiguous().t()):
        assert ops.token_ids(same, 2, 3, cpu).view(2, 3).tolist() == [[0, 1, 2], [3, 4, 5]]
    assert ops.token_ids(t[:3].view(1, 3), 2, 3, cpu).view(2, 3).tolist() == [[0, 1, 2]] * 2
    for wrong in (t[:4], t[:2].view(1, 2), t[:4].view(2, 2)):
        with pytest.raises(RuntimeError):
            ops.token_ids(wrong, 2, 3, cpu)
    with pytest.raises(RuntimeError, match="one device"):      # a host pointer in a kernel's arguments otherwise
        ops.token_ids(t, 2, 3, torch.device("meta"))


@pytest.mark.gpu
@pytest.mark.parametrize("hooked", [False, True])
def test_token_type_ids_of_any_accepted_shape(hooked):
    model = small_model().cuda()
    if hooked:                                       # layer by layer
        model.encoder.register_forward_hook(lambda *a: None)
    ids, types = torch.randint(0, 8, (3, 40), device="cuda"), torch.randint(0, 2, (1, 40), device="cuda")

    def out(t):
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return model(ids, token_type_ids=t)[0]
    want = out(types.expand(3, 40))
    assert torch.equal(out(types), want) and torch.equal(out(types.repeat(3, 1).view(-1)), want)


@pytest.mark.parametrize("dtype", [torch.float64, torch.int64])
@pytest.mark.parametrize("L", [16, 128])
def test_residual_inputs_of_other_types_are_refused(calls, monkeypatch, dtype, L):
    monkeypatch.setattr(sequence_mixer, "_autocast_bf16", lambda: True)
    m, u = mixer(), CudaLike(torch.zeros((2, L, D), dtype=dtype))
    with torch.no_grad(), pytest.raises(TypeError):
        m(u)
    assert "m2_mixer_fwd" not in calls
    m.residual_long_conv = False                     # nothing but its bf16 copy is read then
    with torch.no_grad():
        m(u)


@pytest.mark.parametrize("kind,act,u", [(0, _lib.M2_BF16, _lib.M2_F16), (0, _lib.M2_F32, _lib.M2_F16), (1, _lib.M2_BF16, _lib.M2_F16),
                                        (0, _lib.M2_F16, _lib.M2_F32)])
def test_half_operands_are_refused_where_no_kernel_reads_them(kind, act, u):
    """Sizes of another type would have the kernels read past the end; the check comes before any launch."""
    a = _lib.LongconvArgs()
    a.batch, a.seq_len, a.d_model, a.n_filters, a.kind, a.act_dtype, a.u_dtype = 1, 128, 128, 2, kind, act, u
    host = ctypes.create_string_buffer(64)
    at = (ctypes.addressof(host) + 15) // 16 * 16
    a.xin = a.u = a.out = a.short_w = a.short_b = at
    a.xin_sc = a.u_sc = a.out_sc = 1
    for i in range(2):
        a.spec[i] = a.bias[i] = at
    assert _lib.lib().m2_longconv_fwd(ctypes.byref(a), None) == 2 and b"float32 or bf16" in _lib.lib().m2_last_error()


def test_modules_with_plans_are_freed_without_the_collector(calls):
    """A module that its own plans keep alive would keep its GPU memory until the next garbage collection."""
    gc.collect()
    gc.disable()
    try:
        m, f, model = mixer(), mlp(), small_model()
        mix(m, torch.zeros(2, 128, D))
        feed(f, torch.zeros(2, 128, D))
        plans_of(model).get(model, 0, lambda: model._make_plan(2, 128, torch.device("cpu")))
        assert plans(m) and plans(f) and plans(model)
        dead = [weakref.ref(x) for x in (m, f, model)]
        del m, f, model
        assert [x() for x in dead] == [None] * 3
    finally:
        gc.enable()


def plans(m):
    return list(m._plans.plans.values())


def test_plans_keep_no_copies_and_no_parameters(calls):
    """A CUDA graph bakes the addresses of a plan in and outlives it, another stream may use them, and model.cpu() is to free
    the GPU's memory: so a plan that is kept points to registered tensors and to the module's caches, and holds only the latter."""
    m, f = mixer(), mlp()
    mix(m, torch.zeros(2, 128, D))
    feed(f, torch.zeros(2, 128, D))
    for module in (m, f):
        own = {t.data_ptr() for t in module.parameters()}
        assert len(plans(module)) == 1 and not own & {t.data_ptr() for t in plans(module)[0].held}
    for module, run in ((m, mix), (f, feed)):
        module.bfloat16()                            # float32 copies of biases, taps and LayerNorm belong to each call
        run(module, torch.zeros(2, 128, D))
        run(module, torch.zeros(2, 128, D))
        assert not plans(module)
    m = mixer()
    m.filter_fn.use_bias = False                     # kind 2 takes a vector of zeros for it
    mix(m, torch.zeros(2, 256, D)[:, :128], kind=2)
    assert not plans(m)


@pytest.mark.gpu
def test_a_graph_outlives_the_plans_it_was_captured_with():
    from m2_b200 import GraphedForward
    torch.manual_seed(3)
    m, f = mixer().cuda().bfloat16(), mlp().cuda().bfloat16()

    def layer(u):
        return f(m(u)[0])
    u = torch.randn(4, 128, D, device="cuda")
    graphed = GraphedForward(layer, u)
    want = graphed(u).clone()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        for n in range(1, 20):
            layer(u[:, :4 * n])
    junk = [torch.full((n,), 1e30, device="cuda") for n in (D, 3 * D, 9 * D, D, 3 * D) for _ in range(50)]
    assert torch.equal(graphed(u), want) and len(junk) == 250
