"""Kernels stand in for the experts' activation only as long as it is one that they know: not for another function put in its
place, a subclass with its own forward, or (where the generic path would run it) a module with hooks."""

import pytest
import torch
import torch.nn.functional as F

from planmoe_b200 import moe
from planmoe_b200.experts.ffn import FusedExpertsNetwork


class Shifted(torch.nn.ReLU):
    def forward(self, x):
        return super().forward(x - 0.5)


class Renamed(torch.nn.GELU):
    pass


def _patched():
    m = torch.nn.SiLU()
    m.forward = lambda x: F.silu(x) * 2
    return m


@pytest.mark.parametrize('fn,name', [('gelu', 'gelu'), (None, 'relu'), ('identity', 'identity'), (torch.nn.ReLU(inplace=True), 'relu'), (F.silu, 'silu'),
                                     (torch.nn.Identity(), 'identity'), (Renamed(), 'gelu'), (Shifted(), None), (_patched(), None),
                                     (torch.nn.GELU('tanh'), None), (torch.tanh, None), (lambda x: F.relu(x), None)])
def test_name_of_what_is_computed(fn, name):
    net = FusedExpertsNetwork(8, activation_fn=fn)
    assert net.fused_act == name
    module = isinstance(fn, torch.nn.Module)             # a registered module is replaced by a module
    net.activation_fn = torch.nn.Tanh() if module else torch.tanh
    assert net.fused_act is None
    net.activation_fn = torch.nn.ReLU() if module else F.relu
    assert net.fused_act == ('relu' if name else None)   # a network that began with an unknown one stays where it is


def test_activation_with_self_is_never_a_known_one():
    net = FusedExpertsNetwork(8, activation_fn_with_self=lambda x, me: F.relu(x))
    assert net.fused_act is None


def _layer(act, dtype):
    torch.manual_seed(1)
    with torch.device('cuda'):
        layer = moe.moe_layer(gate_type={'type': 'top', 'k': 2}, model_dim=64,
                              experts={'type': 'ffn', 'count_per_node': 4, 'hidden_size_per_expert': 64, 'activation_fn': act})
    return layer.cuda().to(dtype)


def _pass(layer, x):
    layer.zero_grad(set_to_none=True)
    xin = x.clone().requires_grad_()
    y = layer(xin)
    (y.float().square().sum() + y.l_aux).backward()
    return [y.detach(), xin.grad] + [p.grad for p in layer.parameters()]


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('what', ['replaced', 'subclass', 'patched'])
def test_layer_computes_the_present_activation(what, dtype):
    layer = _layer({'replaced': 'relu', 'subclass': Shifted(), 'patched': _patched()}[what], dtype)
    f = {'replaced': torch.tanh, 'subclass': lambda t: F.relu(t - 0.5), 'patched': lambda t: F.silu(t) * 2}[what]
    if what == 'replaced':
        layer.experts.activation_fn = f
    plain = _layer(lambda t: f(t), dtype)                # nothing that a kernel could know
    x = torch.randn(40, 64, device='cuda', dtype=dtype)
    # the same operations: products and activation of the library, routing and row moves of the same kernels
    for a, b in zip(_pass(layer, x), _pass(plain, x)):
        torch.testing.assert_close(a, b, rtol=0, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['forward', 'pre', 'backward', 'pre_backward'])
def test_hooks_of_the_activation_fire(kind):
    act, seen = torch.nn.ReLU(), []
    layer = _layer(act, torch.float32)
    register = {'forward': act.register_forward_hook, 'pre': act.register_forward_pre_hook, 'backward': act.register_full_backward_hook,
                'pre_backward': act.register_full_backward_pre_hook}[kind]
    register(lambda *a: seen.append(kind))
    _pass(layer, torch.randn(40, 64, device='cuda'))
    assert seen == [kind]
