"""Sparse token <-> expert-slot movement: scatter ("encode"), gather ("decode"), gate-grad.

Three interchangeable backends implement the same three primitives

    scatter(x[S,M], gates[K,S]|None)   -> disp[E*C, M]   disp[idx*C+loc] = g * x      (K1)
    gather (disp[E*C,M], gates|None)   -> out[S, M]      out = sum_k g_k * disp[slot_k] (K2)
    gate_grad(disp[E*C,M], dy[S,M])    -> dg[K, S]       dg_k = <disp[slot_k], dy>      (K3)

* ``cuda``  : hand-written sm_100a kernels (slot-major, atomics-free, bit-reproducible),
* ``cpu``   : the C++ reference loops of the native extension (fp32 / fp64),
* ``torch`` : a composite of differentiable ATen ops (any dtype / device; also the oracle).

They replace the reference's three JIT kernels (``PlanMoE/jit_kernels/sparse.py:17-134``) and
its CPU loops (``PlanMoE/custom/custom_kernel.cpp:57-112``).  A token whose location is
``>= capacity`` (or whose expert id is negative) is dropped: it writes nothing and reads zeros.
"""

import torch

from . import native


class SlotPlan:
    """Stacked routing tensors shared by the three primitives.

    idx, loc : int32 [K, S]   expert id and slot-in-expert of the k-th choice of each token
    E, C     : number of global experts and capacity (slots per expert)
    slot_map : int32 [E*C], value ``t*K+k`` of the (token, choice) that owns the slot, or -1.
               Built lazily; slot ownership is unique, which is what makes the scatter a
               plain store instead of an atomic add.
    """

    def __init__(self, idx, loc, num_experts, capacity, slot_map=None):
        self.idx = idx.contiguous()
        self.loc = loc.contiguous()
        self.K, self.S = int(idx.size(0)), int(idx.size(1))
        self.E, self.C = int(num_experts), int(capacity)
        self._slot_map = slot_map

    @property
    def slot_map(self):
        if self._slot_map is None:
            self._slot_map = build_slot_map(self.idx, self.loc, self.E, self.C)
        return self._slot_map


def build_slot_map(idx, loc, E, C):
    K, S = idx.shape
    if idx.is_cuda:
        return native.lib().build_slot_map(idx, loc, E, C)
    smap = torch.full((E * C,), -1, dtype=torch.int32, device=idx.device)
    tk = (torch.arange(S, device=idx.device, dtype=torch.int32).view(1, S) * K +
          torch.arange(K, device=idx.device, dtype=torch.int32).view(K, 1))
    valid = (loc < C) & (idx >= 0) & (loc >= 0)
    smap[(idx.long() * C + loc.long())[valid]] = tk[valid]
    return smap


# ---------------------------------------------------------------------------------------
# torch composite backend (differentiable by construction)
# ---------------------------------------------------------------------------------------

def scatter_torch(x, plan, gates=None):
    out = x.new_zeros((plan.E * plan.C, x.size(-1)))
    for k in range(plan.K):
        valid = (plan.loc[k] < plan.C) & (plan.idx[k] >= 0)
        slot = (plan.idx[k].long() * plan.C + plan.loc[k].long())[valid]
        src = x[valid]
        if gates is not None:
            src = src * gates[k][valid].unsqueeze(-1).to(x.dtype)
        out = out.index_add(0, slot, src)
    return out


def gather_torch(disp, plan, gates=None):
    out = None
    for k in range(plan.K):
        valid = (plan.loc[k] < plan.C) & (plan.idx[k] >= 0)
        slot = (plan.idx[k].long() * plan.C + plan.loc[k].long()).clamp_(0, plan.E * plan.C - 1)
        rows = disp[slot] * valid.unsqueeze(-1).to(disp.dtype)
        if gates is not None:
            rows = rows * gates[k].unsqueeze(-1).to(disp.dtype)
        out = rows if out is None else out + rows
    return out


def gate_grad_torch(disp, dy, plan):
    res, acc = [], torch.promote_types(disp.dtype, torch.float32)
    for k in range(plan.K):
        valid = (plan.loc[k] < plan.C) & (plan.idx[k] >= 0)
        slot = (plan.idx[k].long() * plan.C + plan.loc[k].long()).clamp_(0, plan.E * plan.C - 1)
        res.append((disp[slot].to(acc) * dy.to(acc)).sum(-1) * valid)
    return torch.stack(res)


# ---------------------------------------------------------------------------------------
# native backends
# ---------------------------------------------------------------------------------------

def _native_ok(x):
    if x.is_cuda:
        return x.dtype in (torch.bfloat16, torch.float16, torch.float32)
    return (x.dtype in (torch.float32, torch.float64) and native.available()
            and not native.force_python_fallback())


def _rows(x):
    return native.aligned(x) if x.is_cuda else x.contiguous()


def _vector_rows(x):
    """Whether rows are whole 16-byte vectors, which is what the CUDA kernels move; others take the composite."""
    return x.size(-1) * x.element_size() % 16 == 0


def _scatter(x, plan, gates):
    x = _rows(x)
    if x.is_cuda and not _vector_rows(x):
        return scatter_torch(x, plan, gates)
    if x.is_cuda:
        return native.lib().dispatch_scatter(x, plan.slot_map, gates, plan.K, plan.E * plan.C)
    return native.lib().cpu_scatter(x, plan.idx, plan.loc, gates, plan.E, plan.C)


def _gather(disp, plan, gates):
    disp = _rows(disp)
    if disp.is_cuda and not _vector_rows(disp):
        return gather_torch(disp.float(), plan, gates).to(disp.dtype)     # added up in fp32, as the kernel does
    if disp.is_cuda:
        return native.lib().dispatch_gather(disp, plan.idx, plan.loc, gates, plan.C)
    return native.lib().cpu_gather(disp, plan.idx, plan.loc, gates, plan.C)


def _gate_grad(disp, dy, plan):
    disp, dy = _rows(disp), _rows(dy)
    if disp.is_cuda and not _vector_rows(disp):
        return gate_grad_torch(disp, dy, plan)
    if disp.is_cuda:
        return native.lib().dispatch_gate_grad(disp, dy, plan.idx, plan.loc, plan.C)
    return native.lib().cpu_gate_grad(disp, dy, plan.idx, plan.loc, plan.C)


def _gates_for(x, gates):
    """Kernels take gates as fp32 [K,S] on CUDA and in the data dtype on CPU."""
    if gates is None:
        return None
    return gates.detach().to(torch.float32 if x.is_cuda else x.dtype).contiguous()


class _Live:
    """Gates that a node was given, for a gradient of its gradient: they go into that as they are, with their history, where the
    gradient itself uses a copy of their values."""

    def __init__(self, gates):
        self.made = [(g, None if g.is_inference() else g._version) for g in gates]

    def get(self):
        if any(v is not None and g._version != v for g, v in self.made):
            raise RuntimeError("gates needed for the gradient of a gradient have been modified by an inplace operation")
        return [g for g, _ in self.made]


# Under create_graph the functions below answer with differentiable operations: encode and decode are each other's adjoint.

class _Scatter(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gates, plan):
        ctx.plan = plan
        g = _gates_for(x, gates)
        ctx.save_for_backward(x if gates is not None else None, g)
        ctx.gdtype = gates.dtype if gates is not None else None
        ctx.live = _Live([gates]) if gates is not None else None
        return _scatter(x, plan, g)

    @staticmethod
    def backward(ctx, ddisp):
        x, g = ctx.saved_tensors
        plan = ctx.plan
        want_gates = g is not None and ctx.needs_input_grad[1]
        if torch.is_grad_enabled():
            return (gather(ddisp, plan, ctx.live.get()[0] if g is not None else None),
                    gate_grad_torch(ddisp, x, plan).to(ctx.gdtype) if want_gates else None, None)
        ddisp = _rows(ddisp)
        dx = _gather(ddisp, plan, g)
        dg = _gate_grad(ddisp, x, plan).to(ctx.gdtype) if want_gates else None
        return dx, dg, None


class _Gather(torch.autograd.Function):
    @staticmethod
    def forward(ctx, disp, gates, plan):
        ctx.plan = plan
        g = _gates_for(disp, gates)
        ctx.save_for_backward(disp if gates is not None else None, g)
        ctx.gdtype = gates.dtype if gates is not None else None
        ctx.live = _Live([gates]) if gates is not None else None
        return _gather(disp, plan, g)

    @staticmethod
    def backward(ctx, dy):
        disp, g = ctx.saved_tensors
        plan = ctx.plan
        want_gates = g is not None and ctx.needs_input_grad[1]
        if torch.is_grad_enabled():
            return (scatter(dy, plan, ctx.live.get()[0] if g is not None else None),
                    gate_grad_torch(disp, dy, plan).to(ctx.gdtype) if want_gates else None, None)
        dy = _rows(dy)
        ddisp = _scatter(dy, plan, g)
        dg = _gate_grad(disp, dy, plan).to(ctx.gdtype) if want_gates else None
        return ddisp, dg, None


class _ScatterPicks(torch.autograd.Function):
    """``_Scatter`` with the gates as fp32 ``rows [K, S]``, rounded to the data's type by the kernels; their gradient goes to
    the picks' own tensors."""

    @staticmethod
    def forward(ctx, x, plan, rows, *gates):
        ctx.plan, ctx.round = plan, x.dtype != torch.float32
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(x, rows)
        ctx.live = _Live(gates)
        return native.lib().dispatch_scatter(_rows(x), plan.slot_map, rows, plan.K, plan.E * plan.C, ctx.round)

    @staticmethod
    def backward(ctx, ddisp):
        x, rows = ctx.saved_tensors
        plan = ctx.plan
        if ddisp is None:
            return (None,) * (3 + plan.K)
        want_gates = any(ctx.needs_input_grad[3:])
        if torch.is_grad_enabled():
            dg = gate_grad_torch(ddisp, x, plan).unbind(0) if want_gates else [None] * plan.K
            return (gather(ddisp, plan, torch.stack(ctx.live.get()).to(x.dtype)), None, None, *dg)
        ddisp = _rows(ddisp)
        dx = native.lib().dispatch_gather(ddisp, plan.idx, plan.loc, rows, plan.C, ctx.round)
        dg = _gate_grad(ddisp, x, plan).unbind(0) if want_gates else [None] * plan.K
        return (dx, None, None, *dg)


class _GatherPicks(torch.autograd.Function):
    """``_Gather`` with the gates as fp32 ``rows [K, S]``."""

    @staticmethod
    def forward(ctx, disp, plan, rows, *gates):
        ctx.plan, ctx.round = plan, disp.dtype != torch.float32
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(disp, rows)
        ctx.live = _Live(gates)
        return native.lib().dispatch_gather(_rows(disp), plan.idx, plan.loc, rows, plan.C, ctx.round)

    @staticmethod
    def backward(ctx, dy):
        disp, rows = ctx.saved_tensors
        plan = ctx.plan
        if dy is None:
            return (None,) * (3 + plan.K)
        want_gates = any(ctx.needs_input_grad[3:])
        if torch.is_grad_enabled():
            dg = gate_grad_torch(disp, dy, plan).unbind(0) if want_gates else [None] * plan.K
            return (scatter(dy, plan, torch.stack(ctx.live.get()).to(disp.dtype)), None, None, *dg)
        dy = _rows(dy)
        ddisp = native.lib().dispatch_scatter(dy, plan.slot_map, rows, plan.K, plan.E * plan.C, ctx.round)
        dg = _gate_grad(disp, dy, plan).unbind(0) if want_gates else [None] * plan.K
        return (ddisp, None, None, *dg)


def plain_autograd(*tensors):
    """Whether a call's gradients, if any, are those of ordinary reverse-mode autograd, which the C++ nodes know: no function
    transform (vmap, functional gradients), no forward-mode, no tracing, no dispatch mode, no tensor subclass."""
    return (not torch._C._are_functorch_transforms_active() and torch.autograd.forward_ad._current_level < 0
            and not torch.compiler.is_compiling() and not torch.jit.is_tracing()
            and torch.utils._python_dispatch._get_current_dispatch_mode() is None
            and all(type(t) in (torch.Tensor, torch.nn.Parameter) for t in tensors))


def picks_ok(x, plan, gates):
    """Whether gates go to the kernels pick by pick: fp32 gates of every token for data of the CUDA kernels."""
    return (x.is_cuda and _native_ok(x) and _vector_rows(x) and len(gates) == plan.K
            and all(g.dtype == torch.float32 and g.device == x.device and g.shape == (plan.S,) for g in gates))


def scatter_picks(x, plan, rows, gates):
    return _ScatterPicks.apply(x, plan, rows, *gates)


def gather_picks(disp, plan, rows, gates):
    if len(gates) <= 4 and plain_autograd(disp, *gates):
        return native.lib().gather_picks_node(disp, plan.idx, plan.loc, rows, list(gates), plan._slot_map, plan.E, plan.C)
    return _GatherPicks.apply(disp, plan, rows, *gates)


def scatter(x, plan, gates=None):
    """Differentiable encode: ``[S, M] -> [E*C, M]`` (w.r.t. ``x`` and ``gates``)."""
    if gates is None and x.is_cuda and _native_ok(x) and x.dim() == 2 and _vector_rows(x) and plain_autograd(x):
        return native.lib().scatter_node(x, plan.idx, plan.loc, plan.slot_map, plan.E, plan.C)
    if _native_ok(x):
        return _Scatter.apply(x, gates, plan)
    return scatter_torch(x, plan, gates)


def gather(disp, plan, gates=None):
    """Differentiable decode: ``[E*C, M] -> [S, M]`` (w.r.t. ``disp`` and ``gates``)."""
    if _native_ok(disp):
        return _Gather.apply(disp, gates, plan)
    return gather_torch(disp, plan, gates)
