"""What the modules lay out once per shape and keep for the next call: kernel arguments with the pointers of weights and
filter tables filled in.  A plan is used again only while every parameter, buffer and submodule it was made from is the
same object with the same storage and version counter; activations, workspaces, outputs and copies of parameters are never
kept.
"""
from __future__ import annotations

import weakref
from collections import OrderedDict
from operator import attrgetter, is_

import torch

from . import ops

_version = attrgetter("_version")
_ptr = torch.Tensor.data_ptr


WEIGHTS = ("weight", "bias", "freq", "z", "t", "deltas")       # names of the tensors that plans and filter tables are made from


class Watch:
    """The parameters, buffers, submodules and settings below `root` as they are now; `same()` says whether they still are."""

    def __init__(self, root):
        mods = list(root.modules())
        if any(isinstance(vars(m).get(name), torch.Tensor) for m in mods for name in WEIGHTS):
            # weights that are plain attributes (replicas, pruned or functionalised modules) are in no table to be watched
            raise RuntimeError("weights outside the modules' parameters and buffers")
        slots = [(d, k, t) for m in mods for d in (m._parameters, m._buffers) for k, t in d.items()]   # None: no such tensor
        kids = [(m._modules, k, c) for m in mods for k, c in m._modules.items()]
        self.dicts, self.keys, self.values = zip(*(slots + kids))
        self.tensors = [t for _, _, t in slots if t is not None]
        self.versions = list(map(_version, self.tensors))      # RuntimeError for tensors made under inference_mode
        self.ptrs = list(map(_ptr, self.tensors))
        # plain attributes that plans are made from: those a module's class names in `plan_attrs`, and eps
        names = [(m, type(m).plan_attrs if hasattr(type(m), "plan_attrs") else ("eps",) if isinstance(m, torch.nn.LayerNorm) else ())
                 for m in mods]
        self.attrs = [(weakref.ref(m), attrgetter(*n)) for m, n in names if n]     # weak: root holds this, and would hold itself
        self.attr_values = [get(m()) for m, get in self.attrs]

    def same(self):
        try:
            return (all(map(is_, map(dict.__getitem__, self.dicts, self.keys), self.values))
                    and list(map(_version, self.tensors)) == self.versions and list(map(_ptr, self.tensors)) == self.ptrs
                    and [get(m()) for m, get in self.attrs] == self.attr_values)
        except (KeyError, AttributeError):
            return False


class Plan:
    """Arguments of a native call with the pointers of weights and filter tables filled in.

    `held` keeps alive what the module's own caches made (bf16 weights, filter tables); registered tensors are not held, as
    Watch sees when they go.  Where a tensor had to be copied (a parameter that is not contiguous float32) the plan is not
    `lasting`: the copy then belongs to one call, to its stream and, inside a CUDA-graph capture, to the graph's own pool,
    and a captured graph never points to what only a plan keeps."""

    def __init__(self, args, **more):
        self.args, self.held, self.lasting = args, [], True
        self.__dict__.update(more)

    def cached(self, t):
        """Pointer of a tensor that a cache of the module holds as long as its source does not change."""
        self.held.append(t)
        return t.data_ptr()

    def registered(self, t, source):
        """Pointer of `t`, the parameter `source` itself or a copy of it.  A source that is no parameter (a parametrized module
        computes it on every access) is held like a copy."""
        if t.data_ptr() == source.data_ptr() and isinstance(source, torch.nn.Parameter):
            return t.data_ptr()
        return self.passing(t)

    def f32(self, source):
        """Pointer of a parameter as contiguous float32."""
        return self.registered(ops._f32c(source), source)

    def passing(self, t):
        """Pointer of a tensor made for this call."""
        self.held.append(t)
        self.lasting = False
        return t.data_ptr()


class SplitWeight:
    """Modules saved with pickle may hold one from when they kept split weights; nothing reads it."""


REFUSED = object()       # kept in the place of a plan that make() did not give


class PlanCache:
    """At most `most` plans of one module, the longest unused dropped first."""

    def __init__(self, most=16, owner=None):
        self.most, self.watch, self.plans = most, None, OrderedDict()
        self.owner = owner and weakref.ref(owner)

    def get(self, root, key, make):
        """The plan of `key`, made by make() when there is none; None when make() returns that (remembered like a plan) or
        the module's tensors cannot be watched."""
        if self.watch is None or not self.watch.same():
            self.plans = OrderedDict()
            try:
                self.watch = Watch(root)
            except RuntimeError:
                self.watch = None
                return None
        plans = self.plans
        plan = plans.get(key)
        if plan is None:
            plan = make()
            if not getattr(plan, "lasting", True):
                return plan
            plans[key] = plan = REFUSED if plan is None else plan
        try:
            plans.move_to_end(key)
            while len(plans) > self.most:
                plans.popitem(last=False)
        except KeyError:                     # another thread took it out
            pass
        return None if plan is REFUSED else plan

    def __deepcopy__(self, memo):
        return PlanCache(self.most)          # a copied module has other tensors

    def __reduce__(self):
        return PlanCache, (self.most,)


def plans_of(module):
    """The module's own PlanCache.  One that came with a copied __dict__ (a data-parallel replica, copy.copy) belongs to the
    module it was made for: plans and Watch of one would answer for the other's tensors."""
    cache = vars(module).get("_plans")
    if cache is None or cache.owner is None or cache.owner() is not module:
        cache = module._plans = PlanCache(owner=module)
    return cache


def expect(dev, *tensors):
    """Raises unless every (tensor, shape) has that shape (None: any size) and lies on `dev`; a missing tensor is not looked at."""
    for t, shape in tensors:
        if t is None:
            continue
        if len(t.shape) != len(shape) or any(n is not None and n != m for m, n in zip(t.shape, shape)):
            raise AssertionError(f"weight of shape {tuple(t.shape)} where {shape} is expected")
        if t.device != dev:
            raise RuntimeError(f"m2_b200 kernels need weights on the input's device: {t.device} and {dev}")


def any_hooks(modules):
    """Whether a hook, or a forward() set on an instance, would see (or change) what goes through one of `modules`."""
    g = torch.nn.modules.module
    if g._global_forward_hooks or g._global_forward_pre_hooks:
        return True
    return any(m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__ for m in modules)


def any_dropping(modules):
    """Whether a dropout of one of `modules` is on."""
    return any(m.training and m.dropout.p > 0 for m in modules)
