"""The GLU feed-forward block of an M2-BERT layer on BlockdiagLinear weights, with the
reference's constructor, forward signature and state_dict keys (reference:
bert/src/bert_layers.py:457-508): gated_layers, wo, layernorm.
"""
from __future__ import annotations

import ctypes as C

import torch
import torch.nn as nn

from . import _lib, ops
from ._plan import Plan, expect, plans_of
from ._tags import attach, forward_only
from .blockdiag_linear import BlockdiagLinear, _compute_dtype


class BertGatedLinearUnitMLP(nn.Module):
    """LayerNorm(wo(gelu(G[..., :I]) * G[..., I:]) + x),  G = gated_layers(x).

    `config` needs hidden_size, intermediate_size, monarch_mlp_nblocks, layer_norm_eps,
    hidden_dropout_prob (and use_monarch_mlp=True: dense nn.Linear layers are the
    reference's other option and are not what this package accelerates).  G is never
    materialised: the gated GEMM applies GELU and the product in its epilogue.
    """

    plan_attrs = ("config", "config.hidden_size", "config.intermediate_size", "config.monarch_mlp_nblocks", "layernorm.eps")

    def __init__(self, config):
        super().__init__()
        self.config = config
        if not getattr(config, "use_monarch_mlp", True):
            raise NotImplementedError("m2_b200.BertGatedLinearUnitMLP needs use_monarch_mlp=True")
        self.is_padded = getattr(config, "monarch_mixer_sequence_mixing", True)
        nb = config.monarch_mlp_nblocks
        self.gated_layers = BlockdiagLinear(config.hidden_size, config.intermediate_size * 2,
                                            bias=False, nblocks=nb)
        self.act = nn.GELU(approximate="none")
        self.wo = BlockdiagLinear(config.intermediate_size, config.hidden_size, nblocks=nb)
        self.dropout = nn.Dropout(config.hidden_dropout_prob)
        self.layernorm = nn.LayerNorm(config.hidden_size, eps=config.layer_norm_eps)

    def fill_args(self, plan, a, dev, f32=False):
        """Writes the pointers of this module's weights into `a` (a _lib.MlpArgs or _lib.EncoderLayer) of `plan`; False where
        the native call, which knows one block count and whole blocks only, does not compute what the weights say.  It sees
        pointers and no tensors, so what they point to is checked here against the config and the device it runs on."""
        D, inter, nb = self.config.hidden_size, self.config.intermediate_size, self.config.monarch_mlp_nblocks
        if self.gated_layers.weight.shape != (nb, 2 * inter // nb, D // nb) or self.wo.weight.shape != (nb, D // nb, inter // nb):
            return False
        expect(dev, (self.gated_layers.weight, (nb, 2 * inter // nb, D // nb)), (self.wo.weight, (nb, D // nb, inter // nb)),
               (self.wo.bias, (D,)), (self.layernorm.weight, (D,)), (self.layernorm.bias, (D,)))
        for name, lin in (("wg", self.gated_layers), ("wo", self.wo)):
            if f32:
                setattr(a, name, plan.f32(lin.weight))
                continue
            w = lin._weight_as(torch.bfloat16)
            setattr(a, name, plan.registered(w, lin.weight) if lin.weight.dtype == torch.bfloat16 else plan.cached(w))
        if self.wo.bias is not None:
            a.wo_bias = plan.f32(self.wo.bias)
        a.ln_w, a.ln_b, a.eps = plan.f32(self.layernorm.weight), plan.f32(self.layernorm.bias), float(self.layernorm.eps)
        return True

    def _plan(self, dev, f32=False):
        def make():
            a = _lib.MlpArgs()
            a.f32 = f32
            a.d_model, a.inter, a.nblocks = self.config.hidden_size, self.config.intermediate_size, self.config.monarch_mlp_nblocks
            split = _lib.lib().m2_mlp_split_bytes(a.d_model, a.inter, a.nblocks) if f32 else 0
            plan = Plan(a, split=split, launches=3 + (f32 and ops.split_used(a.d_model // a.nblocks, a.inter // a.nblocks)))
            return plan if self.fill_args(plan, a, dev, f32) else None
        return plans_of(self).get(self, (dev.index, f32), make)

    def _forward_bf16(self, x, x2, plan, copies_only):
        """The three launches as one call; outputs as in forward()."""
        B, L, D = x.shape
        if D != self.config.hidden_size:
            raise AssertionError(f"input has {D} features, the MLP {self.config.hidden_size}")
        m = B * L
        dev = x.device
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        work = torch.empty((m, self.config.intermediate_size + D), dtype=torch.bfloat16, device=dev)
        aug = torch.empty((m, D), dtype=torch.bfloat16, device=dev)
        tm = torch.empty((D, B, L), dtype=torch.float16, device=dev) if ops.reads_time_major(B, L, D) else None
        y = aug.view(B, L, D) if copies_only and tm is not None else torch.empty((B, L, D), dtype=torch.float32, device=dev)
        a = _lib.MlpArgs.from_buffer_copy(plan.args)
        a.m, a.seq_len = m, L
        a.x, a.h = x2.data_ptr(), work.data_ptr()
        a.o = a.h + 2 * m * self.config.intermediate_size
        a.out_bf16 = aug.data_ptr()
        if y.dtype == torch.float32:
            a.out = y.data_ptr()
        if tm is not None:
            a.out_tm_f16, a.tm_stride = tm.data_ptr(), m
        ops._launch("m2_mlp_fwd", aug, _lib.lib().m2_mlp_fwd, C.byref(a), launches=3)
        return attach(y, bf16=aug, tm=tm, src_dtype=torch.float32)

    def _forward_f32(self, x, x2, plan):
        """The launches on float32 activations (the split of the weights, two GEMMs, LayerNorm) as one call."""
        D, inter = self.config.hidden_size, self.config.intermediate_size
        if x2.shape[-1] != D:
            raise AssertionError(f"input has {x2.shape[-1]} features, the MLP {D}")
        x2 = x2.contiguous()
        m = x2.shape[0]
        work = torch.empty((m, inter + D), dtype=torch.float32, device=x2.device)
        split = torch.empty(plan.split, dtype=torch.uint8, device=x2.device)
        y = torch.empty(x.shape, dtype=torch.float32, device=x2.device)
        a = _lib.MlpArgs.from_buffer_copy(plan.args)
        a.m = m
        a.x, a.h, a.out = x2.data_ptr(), work.data_ptr(), y.data_ptr()
        a.o, a.split = a.h + 4 * m * inter, split.data_ptr()
        ops._launch("m2_mlp_fwd", y, _lib.lib().m2_mlp_fwd, C.byref(a), launches=plan.launches)
        return y

    @forward_only
    def forward(self, hidden_states: torch.Tensor, copies_only: bool = False) -> torch.Tensor:
        """copies_only (used by M2BertEncoder between layers): when the next mixer of this shape
        reads nothing but the bf16 and time-major fp16 copies of the output, skip the float32
        tensor and return the bf16 copy as the hidden state (tagged with the dtype the
        reference's tensor would have, which decides one rounding point in the mixer)."""
        if self.training and self.dropout.p > 0:
            raise RuntimeError("m2_b200: dropout inside the fused MLP is not implemented; use eval()")
        cfg = self.config
        x = hidden_states
        dt = _compute_dtype(x)
        x2 = x.reshape(-1, x.shape[-1])
        if x2.dtype != dt:
            x2 = x2.to(dt)
        if dt == torch.bfloat16 and x.dim() == 3 and x2.shape[0] and x.shape[-1] % 256 == 0 and x.shape[-1] <= 2048 and not ops.observed():
            plan = self._plan(x.device)
            if plan is not None:
                return self._forward_bf16(x, x2, plan, copies_only)
        if dt == torch.float32 and x.is_cuda and x2.shape[0] and not ops.observed():
            plan = self._plan(x.device, f32=True)
            if plan is not None:
                return self._forward_f32(x, x2, plan)
        wg, wo = self.gated_layers._weight_as(dt), self.wo._weight_as(dt)
        h = ops.blockdiag_glu_fwd(x2, wg, cfg.intermediate_size, w_split=ops.split_of(wg))
        o = ops.blockdiag_fwd(h, wo, self.wo.bias, cfg.intermediate_size, cfg.hidden_size, w_split=ops.split_of(wo))
        # under autocast LayerNorm runs in float32 and returns float32
        out_dtype = torch.float32 if dt == torch.bfloat16 else dt
        aug = None
        if dt == torch.bfloat16 and x.dim() == 3 and x.shape[-1] % 256 == 0 and x.shape[-1] <= 2048:
            # the next layer's in_linear reads this output cast to bf16: write that copy here
            # instead of leaving it to a separate cast pass
            aug = torch.empty((x2.shape[0], x.shape[-1]), dtype=torch.bfloat16, device=x.device)
        tm = None
        if aug is not None and ops.reads_time_major(*x.shape):
            # a following mixer of this shape runs a time-contiguous convolution kernel, which reads the
            # layer input as a time-major fp16 tensor: written here too
            tm = torch.empty((x.shape[2], x.shape[0], x.shape[1]), dtype=torch.float16, device=x.device)
        skip = copies_only and tm is not None
        y = ops.add_layernorm_fwd(o, x2, self.layernorm.weight, self.layernorm.bias,
                                  self.layernorm.eps, None if skip else out_dtype, bf16_copy=aug, tm_copy=tm,
                                  fill_pad=False)
        if skip:
            y = aug[:, :x.shape[-1]].view(x.shape[0], x.shape[1], x.shape[2])
        else:
            y = y.reshape(x.shape)
        if aug is not None or tm is not None:
            attach(y, bf16=aug, tm=tm, src_dtype=out_dtype)
        return y
