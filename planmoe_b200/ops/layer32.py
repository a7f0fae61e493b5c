"""The fp32 layer of one rank as one autograd node.

Same operations as the generic path (``impls/moe_layer.py::_generic_forward``): linear gate, softmax, routing kernels, encode, library
fp32 products around bias and activation, decode.  There a pass is some thirty launches under as many autograd nodes and
Python calls, and for the sizes that fp32 is used at the host is what it takes; here forward and backward are one native call
each (``csrc/layer32.h``).
"""

import torch
import torch.nn.functional as F

from . import native
from .dispatch import plain_autograd
from .gemm import ACT_CODES
from ..utils import stage_timer

_EXPERT_PARAMS = ('batched_fc1_w', 'batched_fc1_bias', 'batched_fc2_w', 'batched_fc2_bias')


class _Layer32(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, wg, w1, b1, w2, b2, again, K, capacity, normalize, act):
        ctx.set_materialize_grads(False)
        y, loss, *saved = native.lib().layer32_forward(x, wg, w1, b1, w2, b2, K, capacity, normalize, act)
        ctx.save_for_backward(x, wg, w1, b1, w2, b2, *saved)
        ctx.again, ctx.args = again, (normalize, act)
        return y, loss

    @staticmethod
    def backward(ctx, dy, dloss):
        if dy is None and dloss is None:
            return (None,) * 11
        x, wg, w1, b1, w2, b2, *saved = ctx.saved_tensors
        need = ctx.needs_input_grad[:6]
        if torch.is_grad_enabled():                 # create_graph: through the operations of the generic path
            inputs = [t for t, n in zip((x, wg, w1, b1, w2, b2), need) if n]
            pairs = [(o, g) for o, g in zip(ctx.again(x, wg, w1, b1, w2, b2), (dy, dloss)) if g is not None and o.requires_grad]
            found = iter(torch.autograd.grad([o for o, _ in pairs], inputs, [g for _, g in pairs], create_graph=True,
                                             allow_unused=True))
            return (*(next(found) if n else None for n in need), *(None,) * 5)
        return (*native.lib().layer32_backward(dy, dloss, x, wg, w1, w2, saved, *ctx.args, list(need)), *(None,) * 5)


def _no_hooks(fn):
    return not isinstance(fn, torch.nn.Module) or not (fn._forward_hooks or fn._forward_pre_hooks or fn._backward_hooks or fn._backward_pre_hooks)


def takes(layer, gctx, x, top_k, cf, degree, comm_name, reserve_shape):
    """Whether a call of the generic path is one that the node knows: one rank, fp32 throughout, a plain linear gate, FFN
    experts with a known activation, no hooks on any of them, no more chunks than there are transfers for, the
    built-in transfers (which move nothing here) and methods, GShard loss, token order, gates applied after the experts, a
    positive capacity factor; products in full fp32 and outside autocast; ordinary reverse-mode autograd."""
    from ..experts.ffn import FusedExpertsNetwork
    from ..gates.top import LinearTopKGate
    from ..impls.communicate import AllToAllStatus
    from ..impls.moe_layer import MOELayer
    from ..parallel import codecs, comms
    from . import fused_moe
    from torch.nn.modules import module as nnm
    if not (x.is_cuda and x.dtype == torch.float32 and x.dim() == 2 and x.size(0) > 0 and x.size(1) % 4 == 0 and cf > 0
            and 1 <= degree <= AllToAllStatus.max_num_split):
        return False
    ex = layer.experts
    if (layer.world_size != 1 or layer.sharded_count != 1 or layer.experts_type != 'ffn' or layer.compress_name != 'no'
            or codecs.factory('no') is not codecs.NoCompressor or comm_name not in ('naive', 'pipe', 'hetu', 'dd')
            or comms.factory(comm_name) not in comms.BUILTIN or not layer.is_gshard_loss or not layer.is_postscore
            or layer.batch_prioritized_routing or layer.collect_stats or len(reserve_shape) != 1 or stage_timer.enabled()):
        return False
    if (not fused_moe._unhooked(ex, FusedExpertsNetwork) or not fused_moe._unhooked(gctx, LinearTopKGate)
            or not fused_moe._unhooked(gctx.wg, torch.nn.Linear) or ex.skip_expert or ex.fused_act is None
            or not _no_hooks(ex.activation_fn)
            or any(n in layer.__dict__ or getattr(type(layer), n) is not getattr(MOELayer, n) for n in ('expert_local', '_route'))
            or nnm._global_forward_hooks or nnm._global_forward_pre_hooks
            or nnm._global_backward_hooks or nnm._global_backward_pre_hooks):
        return False
    wg = gctx.wg.weight
    ps = [getattr(ex, n) for n in _EXPERT_PARAMS]
    E = layer.num_global_experts
    capacity = min(int(top_k), E) * int(cf * ((x.size(0) + E - 1) // E))
    return (capacity > 0 and gctx.wg.bias is None and not (layer.training and gctx.gate_noise > 0) and E <= 64
            and 1 <= min(int(top_k), E) <= 4 and x.size(0) * top_k < 2 ** 31 and ps[2].size(2) % 4 == 0
            and ps[3].size(1) == ps[2].size(2) and wg.size(1) == x.size(1) == ps[0].size(1)
            and all(p.dtype == torch.float32 and p.device == x.device for p in (wg, *ps))
            # the legacy flag, allow_tf32, cannot be read once TF32 was chosen by this switch, which follows the legacy ones
            and not torch.is_autocast_enabled('cuda') and torch.backends.cuda.matmul.fp32_precision in ('none', 'ieee')
            and plain_autograd(x, wg, *ps))


def _as_operations(act, top_k, cf, degree, normalize):
    """The same pass as differentiable operations."""
    from ..impls.fast_dispatch import extract_critical, fast_decode, fast_encode

    def run(x, wg, w1, b1, w2, b2):
        crit, loss = extract_critical(F.softmax(F.linear(x, wg), dim=1), top_k=top_k, capacity_factor=cf, normalize_gate=normalize,
                                      alignment=4 * degree)
        h = act(torch.matmul(fast_encode(x, crit), w1) + b1.unsqueeze(1))
        return fast_decode(torch.matmul(h, w2) + b2.unsqueeze(1), crit), loss
    return run


def forward(layer, x, gctx, top_k, cf, degree):
    """``(y, l_aux, capacity)``"""
    from ..impls.communicate import AllToAllStatus
    AllToAllStatus.init(layer.group, degree, 1)          # what the chunked transfers of later calls read
    E, S = layer.num_global_experts, x.size(0)
    top_k = min(int(top_k), E)
    capacity = top_k * int(cf * ((S + E - 1) // E))
    capacity += -capacity % (4 * degree)
    ex, normalize = layer.experts, bool(layer.normalize_gate)
    args = (native.aligned(x), gctx.wg.weight, *(getattr(ex, n) for n in _EXPERT_PARAMS))
    more = (top_k, capacity, normalize, ACT_CODES[ex.fused_act])
    if torch.is_grad_enabled() and any(t.requires_grad for t in args):
        y, loss = _Layer32.apply(*args, _as_operations(ex.activation_fn, top_k, cf, degree, normalize), *more)
    else:
        y, loss = native.lib().layer32_forward(*args, *more)[:2]
    layer.protected_shape = torch.Size((E, capacity // degree, args[4].size(2)))
    return y, loss, capacity
