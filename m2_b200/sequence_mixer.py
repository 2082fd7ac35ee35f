"""MonarchMixerSequenceMixing with the reference's constructor, forward signature and
state_dict layout (reference: bert/src/mm/monarch_mixer_sequence_mixer.py:12-154); the part
between in_linear and out_linear is one fused CUDA kernel.
"""
from __future__ import annotations

import ctypes as C

import torch
import torch.nn as nn

from . import _lib, ops
from ._plan import Plan, expect, plans_of
from ._tags import copies_of, forward_only, src_dtype_of
from .hyena_filter import HyenaFilter, _autocast_bf16


class _Bf16Linear:
    """bf16 copy of a Linear's weight (what autocast would cast per call), refreshed when the parameter changes;
    the bias stays float32 -- the GEMM kernel rounds it to bf16 itself, as autocast's cast does."""

    def __init__(self):
        self.key, self.w = None, None

    def get(self, lin):
        key = (lin.weight.data_ptr(), lin.weight._version, lin.weight.device)
        if key != self.key:
            self.key, self.w = key, lin.weight.detach().to(torch.bfloat16).contiguous()
        return self.w


def bf16_input(u):
    """(B, L, D) bf16 tensor in_linear reads: the copy a preceding m2_b200 LayerNorm wrote (if u has not
    been edited since), else u cast to bf16."""
    B, L, D = u.shape
    rec = copies_of(u)
    c = rec.bf16 if rec is not None else None
    if c is not None and c.shape == (B * L, D) and c.device == u.device:
        return c.view(B, L, D)
    if u.dtype == torch.bfloat16 and u.stride(-1) == 1:
        return u
    return u.to(torch.bfloat16)


def _round_up(n, m):
    return (n + m - 1) // m * m


class MonarchMixerSequenceMixing(nn.Module):
    """Gated bidirectional long-convolution sequence mixer.

    forward(u): u (B, L, d_model) -> (y (B, L, d_model), None) where, per channel,
    x1, x2, v = split(short_conv(in_linear(u)));  y = out_linear(long_conv(v * x1) * x2
    [+ long_conv2(u)]).  Under torch.autocast(bfloat16) the kernels round to bf16 exactly
    where the reference's PyTorch ops would.
    """

    plan_attrs = ("d_model", "residual_long_conv", "hyena_training_additions")

    def __init__(self, d_model, l_max=128, dropout=0.0, hyena_kernel_lr=None, bidirectional=False,
                 hyena_lr_pos_emb=1e-5, hyena_w=10, hyena_w_mod=1, hyena_wd=0.1, hyena_emb_dim=3,
                 hyena_filter_dropout=0.0, hyena_filter_order=16, residual_long_conv=False,
                 hyena_training_additions=False, verbose=False):
        super().__init__()
        self.d_model = d_model
        self.l_max = l_max
        self.kernel_lr = hyena_kernel_lr
        self.channels = 1
        self.bidirectional = bidirectional
        self.residual_long_conv = residual_long_conv
        self.NUM_PROJECTIONS = 3
        if verbose:
            print(f"-- Bidirectional: {bidirectional}  residual long conv: {residual_long_conv}  "
                  f"w: {hyena_w}  w_mod: {hyena_w_mod}  order: {hyena_filter_order}  emb: {hyena_emb_dim}")

        def make_filter():
            return HyenaFilter(d_model, order=hyena_filter_order, seq_len=l_max,
                               dropout=hyena_filter_dropout, bidirectional=bidirectional,
                               lr=hyena_kernel_lr, lr_pos_emb=hyena_lr_pos_emb, w=hyena_w,
                               w_mod=hyena_w_mod, wd=hyena_wd, emb_dim=hyena_emb_dim)

        self.filter_fn = make_filter()
        if residual_long_conv:
            self.filter_fn2 = make_filter()
        self.in_linear = nn.Linear(d_model, 3 * d_model)
        self.out_linear = nn.Linear(d_model, d_model)
        self.hyena_training_additions = hyena_training_additions
        if hyena_training_additions:
            self.act = nn.Identity()
            self.drop = nn.Dropout(dropout)
            self.layernorm = nn.LayerNorm(d_model)
        width = d_model * self.NUM_PROJECTIONS
        self.short_filter = nn.Conv1d(width, width, kernel_size=3, groups=width, padding=2)

    def _weights(self):
        """bf16 copies of in_linear's and out_linear's weights."""
        if not hasattr(self, "_w_in"):
            self._w_in, self._w_out = _Bf16Linear(), _Bf16Linear()
        return self._w_in.get(self.in_linear), self._w_out.get(self.out_linear)

    def filters(self):
        return [self.filter_fn, self.filter_fn2] if self.residual_long_conv else [self.filter_fn]

    def fill_args(self, plan, a, L, kind, dev, f32=False):
        """Writes the pointers of this module's weights and filter tables into `a` (a _lib.MixerArgs or _lib.EncoderLayer)
        of `plan`.  The native call sees pointers only, so what they point to is checked here against in_linear's width and
        the device it runs on."""
        D = self.in_linear.weight.shape[-1]
        expect(dev, (self.in_linear.weight, (3 * D, D)), (self.in_linear.bias, (3 * D,)), (self.out_linear.weight, (D, D)),
               (self.out_linear.bias, (D,)), (self.short_filter.weight, (3 * D, 1, 3)), (self.short_filter.bias, (3 * D,)),
               *((f.bias, (D,)) for f in self.filters()), *((f.implicit_filter[6].weight, (D, None)) for f in self.filters()))
        if f32:
            for lin in (self.in_linear, self.out_linear):
                if lin.weight.dtype != torch.float32 or not lin.weight.is_contiguous():
                    raise AssertionError("float32 inputs need contiguous float32 weights")
            a.w_in, a.w_out = plan.f32(self.in_linear.weight), plan.f32(self.out_linear.weight)
        else:
            a.w_in, a.w_out = (plan.cached(w) for w in self._weights())
        a.short_w, a.short_b = plan.f32(self.short_filter.weight), plan.f32(self.short_filter.bias)
        if self.in_linear.bias is not None:
            a.b_in = plan.f32(self.in_linear.bias)
        if self.out_linear.bias is not None:
            a.b_out = plan.f32(self.out_linear.bias)
        for i, f in enumerate(self.filters()):
            a.spec[i] = plan.cached(f.spectrum(L, not f32, kind))
            if kind in (0, 2):                       # kinds 3 and 4 have it inside their tables
                a.bias[i] = plan.f32(f.bias) if f.use_bias else plan.passing(ops._f32c(f.conv_bias()))

    def _make_plan(self, B, L, kind, dev, f32=False):
        a = _lib.MixerArgs()
        Lp = L if f32 else _round_up(L, 8)
        a.f32 = f32
        a.batch, a.seq_len, a.pitch, a.out_pitch, a.d_model = B, L, Lp, L, self.in_linear.weight.shape[-1]
        a.kind, a.n_filters = kind, 2 if self.residual_long_conv else 1
        a.stride, a.u_stride = _round_up(B * Lp, 16), B * Lp
        plan = Plan(a, split=_lib.lib().m2_mixer_split_bytes(a.d_model) if f32 else 0, launches=3 + (f32 and ops.split_used(a.d_model)))
        self.fill_args(plan, a, L, kind, dev, f32)
        return plan

    def _forward_bf16(self, u, ures, kind):
        """bf16 path: the convolution kernels work on channel-major, time-contiguous rows -- in_linear writes (3D, B, L)
        and out_linear reads (D, B, L) through the operand arrangements of m2_linear_fwd, no transposed copy of an
        activation.  Rows are padded to a multiple of 8 steps so that every one starts on a 16-byte boundary."""
        B, L, D = u.shape
        if D != self.in_linear.weight.shape[-1]:
            raise AssertionError(f"input has {D} channels, the mixer {self.in_linear.weight.shape[-1]}")
        Lp = _round_up(L, 8)
        dev = u.device
        rec = copies_of(u)
        x = rec.bf16 if rec is not None else None                                # (B*L, D) from the LayerNorm
        rows = None                              # bf16 rows to be written together with the time-major copy below
        if x is None or L != Lp or x.shape != (B * L, D) or x.device != dev or not x.is_contiguous():
            if ures is u and u.dtype == torch.float32 and (rec is None or rec.tm is None or L != Lp):
                x = torch.empty((B, Lp, D), dtype=torch.bfloat16, device=dev)
                rows = x[:, :L]
            elif L == Lp:
                x = u.to(torch.bfloat16).contiguous()
            else:
                x = torch.empty((B, Lp, D), dtype=torch.bfloat16, device=dev)
                x[:, :L].copy_(u)
        u_t = None
        if ures is not None:
            rec = copies_of(ures)
            u_t = rec.tm if rec is not None else None                            # (D, B, L) fp16 from the LayerNorm
            if rows is not None or u_t is None or u_t.shape != (D, B, Lp) or L != Lp or u_t.device != dev or not u_t.is_contiguous():
                u_t = torch.empty((D, B, Lp), dtype=torch.float16, device=dev)
                ops.time_major_f16(ures if ures.dtype in (torch.float32, torch.bfloat16) else ures.float(), out=u_t[:, :, :L], rows=rows)
        yu_bf16 = ures is not None and src_dtype_of(ures) == torch.bfloat16
        plan = plans_of(self).get(self, (B, L, kind, dev.index), lambda: self._make_plan(B, L, kind, dev))
        stride = _round_up(B * Lp, 16)
        # allocated per call: inside a CUDA-graph capture the buffers then belong to the graph's own pool
        work = torch.empty((4 * D, stride), dtype=torch.bfloat16, device=dev)
        y = torch.empty((B, L, D), dtype=torch.bfloat16, device=dev)
        if plan is None or ops.observed():
            return self._launch_singly(x, u_t, work, y, kind, yu_bf16)
        a = _lib.MixerArgs.from_buffer_copy(plan.args)
        a.x, a.u = x.data_ptr(), u_t.data_ptr() if u_t is not None else None
        a.yu_bf16 = yu_bf16
        a.xin = work.data_ptr()
        a.conv, a.out = a.xin + 2 * 3 * D * stride, y.data_ptr()
        ops._launch("m2_mixer_fwd", y, _lib.lib().m2_mixer_fwd, C.byref(a), launches=3)
        return y

    def _forward_f32(self, u):
        """The float32 mixer on contiguous token rows as one native call; None where single launches have to do it."""
        B, L, D = u.shape
        if D != self.in_linear.weight.shape[-1] or not u.is_contiguous() or ops.observed():
            return None
        dev = u.device
        plan = plans_of(self).get(self, (B, L, "f32", dev.index), lambda: self._make_plan(B, L, 0, dev, f32=True))
        if plan is None:
            return None
        work = torch.empty((B * L, 4 * D), dtype=torch.float32, device=dev)
        split = torch.empty(plan.split, dtype=torch.uint8, device=dev)
        y = torch.empty((B, L, D), dtype=torch.float32, device=dev)
        a = _lib.MixerArgs.from_buffer_copy(plan.args)
        a.x, a.out, a.xin, a.split = u.data_ptr(), y.data_ptr(), work.data_ptr(), split.data_ptr()
        a.conv = a.xin + 4 * 3 * D * B * L
        ops._launch("m2_mixer_fwd", y, _lib.lib().m2_mixer_fwd, C.byref(a), launches=plan.launches)
        return y

    def _launch_singly(self, x, u_t, work, y, kind, yu_bf16):
        """The three launches of m2_mixer_fwd one by one."""
        B, L, D = y.shape
        Lp = _round_up(L, 8)
        n = B * Lp
        w_in, w_out = self._weights()
        ops.linear_fwd(x.view(1, n, D), w_in, self.in_linear.bias, out=work[:3 * D, :n].t().unsqueeze(0))

        def rows(t):                                                             # (B, L, C) view of channel-major rows
            return t[:, :n].unflatten(1, (B, Lp))[:, :, :L].permute(1, 2, 0)
        fs = self.filters()
        ops.longconv_fwd(rows(work[:3 * D]), u_t[:, :, :L].permute(1, 2, 0) if u_t is not None else None,
                         self.short_filter.weight, self.short_filter.bias, [f.spectrum(L, True, kind) for f in fs],
                         [f.conv_bias() for f in fs] if kind == 2 else None, kind=kind, bf16_rounding=True,
                         out=rows(work[3 * D:]), yu_bf16=yu_bf16)
        if L == Lp:
            return ops.linear_fwd(work[3 * D:, :n].t().unsqueeze(0), w_out, self.out_linear.bias, out=y.view(1, n, D)).view(B, L, D)
        return ops.linear_fwd(rows(work[3 * D:]), w_out, self.out_linear.bias, out=y)

    @forward_only
    def forward_channels(self, u, lo, hi):
        """Channels [lo, hi) of the tensor out_linear consumes, (B, L, hi - lo) bf16, computed from the full
        input u (B, L, d_model) under bf16 autocast -- the unit of work when the mixer is sharded by d_model
        channel over several GPUs: short convolution, gates and long convolutions are independent per
        channel, in_linear contributes its rows c, D + c, 2D + c, and only out_linear mixes channels (it is
        not part of a shard).  Shards computed on different GPUs and concatenated along the last axis equal
        forward_channels(u, 0, d_model) bit for bit (forward() itself may run another convolution family, whose results agree
        within the mode's tolerance).  The reference has no counterpart (its parallelism is
        data parallel only); this follows bert/src/mm/monarch_mixer_sequence_mixer.py:108-149 per channel."""
        if not (u.is_cuda and _autocast_bf16()):
            raise RuntimeError("forward_channels runs on CUDA tensors under torch.autocast('cuda', dtype=torch.bfloat16)")
        B, L, D = u.shape
        if not (0 <= lo < hi <= D):
            raise ValueError(f"channel range [{lo}, {hi}) outside d_model {D}")
        C = hi - lo
        filters = [self.filter_fn] + ([self.filter_fn2] if self.residual_long_conv else [])
        kind = ops.longconv_kind(L, torch.bfloat16, C)
        if kind == 1:
            kind = 0                         # the small-batch FFT family wants 128-channel tiles; a shard need not have them
        key = (lo, hi, L, kind, tuple(f._version_key() for f in filters),
               self.in_linear.weight._version, self.in_linear.bias._version,
               self.short_filter.weight._version, self.short_filter.bias._version,
               tuple(f.bias._version for f in filters))
        cache = getattr(self, "_shard_cache", None)
        if cache is None or cache[0] != key:
            rows = torch.cat([torch.arange(g * D + lo, g * D + hi, device=u.device) for g in range(3)])
            w_in, _ = self._weights()
            shard = dict(
                w=w_in[rows].contiguous(), b=self.in_linear.bias.detach()[rows].contiguous(),
                sw=self.short_filter.weight.detach()[rows].contiguous(), sb=self.short_filter.bias.detach()[rows].contiguous(),
                specs=[ops.filter_spectrum(f.time_filter(L, True)[lo:hi].contiguous(), L, kind) for f in filters],
                biases=[f.conv_bias().detach()[lo:hi].contiguous() for f in filters])
            self._shard_cache = cache = (key, shard)
        sh = cache[1]
        ures = u if self.residual_long_conv else None
        if kind == 2:
            Lp = _round_up(L, 16)
            xin_t = torch.empty((B, 3 * C, Lp), dtype=torch.bfloat16, device=u.device)[:, :, :L]
            ops.linear_fwd(bf16_input(u), sh["w"], sh["b"], out=xin_t.permute(0, 2, 1))
            u_view, yu_bf16 = None, False
            if ures is not None:
                rec = copies_of(ures)
                tm = rec.tm if rec is not None else None
                if tm is not None and tm.shape == (D, B, L):
                    u_view, yu_bf16 = tm[lo:hi].permute(1, 2, 0), src_dtype_of(ures) == torch.bfloat16
                else:
                    u_view = ures[..., lo:hi].transpose(1, 2).contiguous().transpose(1, 2)
            y_t = torch.empty((B, C, Lp), dtype=torch.bfloat16, device=u.device)[:, :, :L]
            ops.longconv_fwd(xin_t.permute(0, 2, 1), u_view, sh["sw"], sh["sb"], sh["specs"], sh["biases"],
                             kind=2, bf16_rounding=True, out=y_t.permute(0, 2, 1), yu_bf16=yu_bf16)
            return y_t.permute(0, 2, 1)
        xin = ops.linear_fwd(bf16_input(u), sh["w"], sh["b"])
        return ops.longconv_fwd(xin, ures[..., lo:hi] if ures is not None else None, sh["sw"], sh["sb"], sh["specs"],
                                sh["biases"], kind=kind, bf16_rounding=True)

    @forward_only
    def forward(self, u, **kwargs):
        if not u.is_cuda:
            raise RuntimeError("m2_b200.MonarchMixerSequenceMixing needs CUDA tensors; there is no CPU fallback")
        if self.hyena_training_additions:
            if self.training and self.drop.p > 0:
                raise RuntimeError("m2_b200: dropout inside the fused mixer is not implemented; use eval()")
            u = self.layernorm(u)
        L = u.size(-2)
        bf16 = _autocast_bf16()
        if not bf16 and u.dtype != torch.float32:
            raise RuntimeError("m2_b200 mixer runs float32 inputs, or any input under "
                               "torch.autocast('cuda', dtype=torch.bfloat16); got "
                               f"{u.dtype} without autocast")
        if u.dim() == 2:
            u = u.unsqueeze(0)
        u_orig = u
        ures = u_orig if self.residual_long_conv else None
        if ures is not None:
            ops._dt(ures)                       # the residual filter reads the input itself: TypeError for float64 or integers
        if bf16:
            kind = ops.longconv_pick(u.size(0), L, torch.bfloat16, self.d_model)
            if kind and u.size(0):
                return self._forward_bf16(u, ures, kind), None
        elif u.size(0):
            y = self._forward_f32(u)
            if y is not None:
                return y, None
        kind = 0                                # float32 convolution on token rows
        if ures is not None and ures.dtype == torch.float16:
            ures = ures.float()
        filters = self.filters()
        biases = [f.conv_bias() for f in filters]
        specs = [f.spectrum(L, bf16, kind) for f in filters]
        if bf16:
            w_in, w_out = self._weights()
            xin = ops.linear_fwd(bf16_input(u), w_in, self.in_linear.bias)
        else:
            w_in, w_out = self.in_linear.weight.detach(), self.out_linear.weight.detach()
            xin = ops.linear_fwd(u, w_in, self.in_linear.bias, w_split=ops.split_of(w_in))
        y = ops.longconv_fwd(xin, ures, self.short_filter.weight, self.short_filter.bias, specs, biases,
                             kind=kind, bf16_rounding=bf16)
        return ops.linear_fwd(y, w_out, self.out_linear.bias, w_split=ops.split_of(w_out)), None
