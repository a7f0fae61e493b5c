"""Top-k routing (``extract_critical``) and the encode / decode dispatcher.

API parity with the reference's ``PlanMoE/impls/fast_dispatch.py``: ``extract_critical``
(:140-195) returns ``((E, indices_s, locations_s, gates_s, capacity), l_loss)``;
``fast_encode`` (:197-201) gives ``[E, C, M]``; ``fast_decode`` (:203-207) gives ``[S, M]``;
``TutelMoeFastDispatcher`` (:82-131) keeps its ``update / encode / decode`` methods.

Routing rules kept bit-for-bit (they fix which token lands in which slot):
  * top-k on softmax scores; gate_k = score of the k-th pick,
  * slot location = running count of earlier tokens that picked the same expert, where every
    k-th pick ranks after all (k-1)-th picks of that expert,
  * ``normalize_gate`` divides by the clamped sum over k (only when k > 1),
  * capacity = k * int(cf * ceil(S/E)); cf == 0 -> dynamic (max location + 1, MAX-reduced);
    cf < 0 -> min(dynamic, bound from |cf|); then rounded up to ``alignment``,
  * a pick whose location >= capacity is dropped.

Unlike the reference, bf16 data is moved by a native bf16 kernel (no fp32 round trip) and the
scatter is a unique-slot store instead of an atomic add.
"""

import torch

from . import losses
from .communicate import simple_all_reduce
from ..jit_kernels import gating
from ..jit_kernels.gating import fast_cumsum_sub_one
from ..ops import dispatch as D
from ..ops import native


def _versions(tensors):
    """What ``_unchanged`` compares with, None where versions are not counted (inference tensors)."""
    return None if any(t.is_inference() for t in tensors) else [(t, t._version) for t in tensors]


def _unchanged(tensors, made):
    return made is not None and len(tensors) == len(made) and all(t is m and t._version == v for t, (m, v) in zip(tensors, made))


class RoutingPlan(tuple):
    """The 5-tuple ``(E, indices_s, locations_s, gates_s, capacity)`` plus cached stacked
    tensors for the kernels (``.slots`` is an ``ops.dispatch.SlotPlan``).  ``slots`` and ``rows`` (fp32 gates ``[K, S]``) are
    what the lists say in memory of their own; each is used as long as its lists are what they were."""

    def __new__(cls, num_experts, indices_s, locations_s, gates_s, capacity, slots=None, rows=None):
        self = super().__new__(cls, (num_experts, indices_s, locations_s, gates_s, capacity))
        self._slots = None
        self._made = slots, _versions((*indices_s, *locations_s)) if slots is not None else None
        self._rows = rows, _versions(gates_s) if rows is not None else None
        return self

    @property
    def slots(self):
        if self._slots is None:
            slots, made = self._made
            if _unchanged((*self[1], *self[2]), made):
                self._slots = slots
                return slots
            idx = torch.stack([x.to(torch.int32).view(-1) for x in self[1]])
            loc = torch.stack([x.to(torch.int32).view(-1) for x in self[2]])
            self._slots = D.SlotPlan(idx, loc, self[0], self[4])
        return self._slots

    def stacked_gates(self):
        return torch.stack(list(self[3]))

    def gate_rows(self):
        """The gates as they are now, detached, in memory that the lists' owner does not write to."""
        rows, made = self._rows
        return rows if _unchanged(self[3], made) else torch.stack([g.detach() for g in self[3]])


def _as_plan(crit):
    if isinstance(crit, RoutingPlan):
        return crit
    return RoutingPlan(*crit)


def compute_sorted_location(x, importance_scores):
    """Batch-prioritised routing: locations are assigned in order of token importance
    (lowest ``importance_scores`` first) instead of token order."""
    order = importance_scores.argsort(dim=0)
    sorted_x = x[order]
    sorted_loc = fast_cumsum_sub_one(sorted_x) * sorted_x
    out = torch.empty_like(sorted_loc)
    out[order] = sorted_loc
    return out


def _gates_of(gates_all, normalize_gate):
    """Per-pick gate lists from the picked scores ``[S, k]``."""
    gates_s = [gates_all[:, k] for k in range(gates_all.size(1))]
    if gates_all.size(1) > 1 and normalize_gate:
        denom = torch.clamp(gates_all.sum(dim=1), min=torch.finfo(gates_all.dtype).eps)
        gates_s = [g / denom for g in gates_s]
    return gates_s


def _route_on_kernels(scores, top_k, loss_fn):
    """Whether the routing kernels take this call.  They pick from fp32 scores (a tie goes to the lower expert id) and
    know the GShard loss; other losses and types, batch-prioritised order, function transforms (vmap, forward-mode),
    tracing and tensor subclasses take the ATen composition."""
    return (scores.is_cuda and scores.dtype == torch.float32 and scores.dim() == 2 and scores.size(0) > 0
            and 1 <= scores.size(1) <= 64 and 1 <= top_k <= 4 and scores.size(0) * top_k < 2 ** 31
            and (loss_fn is None or loss_fn is losses.gshard_loss)
            and gating.use_fast_cumsum and D.plain_autograd(scores))


def _align(capacity, alignment):
    return capacity + -capacity % alignment


def extract_critical(scores, top_k, loss_fn=losses.gshard_loss, capacity_factor=1.0,
                     batch_prioritized_routing=False, normalize_gate=True, group=None, alignment=1):
    S, E = int(scores.size(0)), int(scores.size(1))
    top_k = min(int(top_k), E)
    per_expert = (S + E - 1) // E
    if not batch_prioritized_routing and _route_on_kernels(scores, top_k, loss_fn):
        capacity = _align(top_k * int(capacity_factor * per_expert), alignment) if capacity_factor > 0 else 0
        scores = scores.contiguous()
        # top-k, gates, locations, slot map and loss in two launches; gradients and slots use ``own``, a second copy of picks,
        # locations and gates: the caller may change the lists of a plan in place
        idx, loc, slot_map, _top1, _value, own, *gates_s = native.lib().route_scores_node(scores, top_k, capacity, bool(normalize_gate),
                                                                                         loss_fn is not None)
        l_loss = gates_s.pop() if loss_fn is not None else None
        if capacity_factor <= 0:
            peak = simple_all_reduce(loc.max(), group=group, op=torch.distributed.ReduceOp.MAX)
            capacity = int(peak) + 1
            if capacity_factor < 0:
                capacity = min(capacity, top_k * int(-capacity_factor * per_expert))
            capacity, slot_map = _align(capacity, alignment), None
        plan = RoutingPlan(E, list(idx.unbind(0)), list(loc.unbind(0)), gates_s, capacity,
                           D.SlotPlan(own[0], own[1], E, capacity, slot_map), own[2].view(torch.float32))
        return plan, l_loss
    topk_indices = torch.topk(scores, top_k, dim=1).indices
    gates_all = scores.gather(1, topk_indices)                      # [S, k], differentiable

    l_loss = loss_fn(scores, topk_indices) if loss_fn is not None else None

    if batch_prioritized_routing:
        importance = -scores.max(dim=1)[0]
        locate = lambda m: compute_sorted_location(m, importance)   # noqa: E731
    else:
        locate = fast_cumsum_sub_one

    indices_s, locations_s = [], []
    base = None
    for k in range(top_k):
        ids = topk_indices[:, k]
        mask = losses._one_hot_with_dtype(ids, E, dtype=torch.int32)
        pos = locate(mask)
        if base is not None:
            pos = pos + base
        locations_s.append(pos.gather(1, ids.view(-1, 1)).view(-1).to(torch.int32))
        indices_s.append(ids.to(torch.int32))
        counts = mask.sum(dim=0, keepdim=True)
        base = counts if base is None else base + counts

    gates_s = _gates_of(gates_all, normalize_gate)
    if capacity_factor > 0:
        capacity = top_k * int(capacity_factor * per_expert)
    else:
        peak = torch.max(torch.cat(locations_s, dim=0))
        capacity = int(simple_all_reduce(peak, group=group, op=torch.distributed.ReduceOp.MAX)) + 1
        if capacity_factor < 0:
            capacity = min(capacity, top_k * int(-capacity_factor * per_expert))
    capacity = _align(capacity, alignment)
    return RoutingPlan(E, indices_s, locations_s, gates_s, capacity), l_loss


class TutelMoeFastDispatcher:
    """Stateful encode/decode helper (reference: fast_dispatch.py:82-131)."""

    def __init__(self, num_global_experts, capacity, model_dim, dispatch_dtype):
        self.num_global_experts = int(num_global_experts)
        self.capacity = int(capacity)
        self.model_dim = int(model_dim)
        self.dtype = dispatch_dtype
        self.original_dtype = dispatch_dtype
        self.is_postscore = True
        self._plan = None

    def update(self, indices_, locations_, gates_, capacity=None, is_postscore=True):
        self.capacity = int(capacity) or self.capacity
        self.indices_ = [x.to(torch.int32).view(-1) for x in indices_]
        self.locations_ = [x.to(torch.int32) for x in locations_]
        self.gates_ = list(gates_)
        self.is_postscore = is_postscore
        self.sample_size = int(self.indices_[0].size(0))
        self._plan = RoutingPlan(self.num_global_experts, self.indices_, self.locations_,
                                 self.gates_, self.capacity)

    def _gates(self, like):
        return torch.stack([g.to(like.dtype) for g in self.gates_])

    def encode(self, data):
        gates = None if self.is_postscore else self._gates(data)
        return D.scatter(data, self._plan.slots, gates)

    def decode(self, data):
        gates = self._gates(data) if self.is_postscore else None
        return D.gather(data.reshape(-1, data.size(-1)), self._plan.slots, gates)


fast_dispatcher = TutelMoeFastDispatcher


def fast_encode(data, critial_data, is_postscore=True):
    """[S, M] tokens -> [E, C, M] expert slots (gate-weighted iff ``not is_postscore``)."""
    plan = _as_plan(critial_data)
    if not is_postscore and D.picks_ok(data, plan.slots, plan[3]):
        return D.scatter_picks(data, plan.slots, plan.gate_rows(), plan[3]).view(plan[0], -1, data.size(-1))
    gates = None if is_postscore else plan.stacked_gates().to(data.dtype)
    return D.scatter(data, plan.slots, gates).view(plan[0], -1, data.size(-1))


def fast_decode(data, critial_data, is_postscore=True):
    """[E, C, M] expert slots -> [S, M] tokens (gate-weighted iff ``is_postscore``)."""
    plan = _as_plan(critial_data)
    if is_postscore and D.picks_ok(data, plan.slots, plan[3]):
        return D.gather_picks(data.reshape(-1, data.size(-1)), plan.slots, plan.gate_rows(), plan[3])
    gates = plan.stacked_gates().to(data.dtype) if is_postscore else None
    return D.gather(data.reshape(-1, data.size(-1)), plan.slots, gates)
