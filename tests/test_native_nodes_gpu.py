"""The C++ autograd nodes of routing, encode, decode and the layer of one rank against the Python functions that they stand in for."""

import pytest
import torch
import torch.nn.functional as F

from planmoe_b200 import moe
from planmoe_b200.impls.fast_dispatch import extract_critical, fast_decode, fast_encode
from planmoe_b200.ops import dispatch, fused_moe

pytestmark = pytest.mark.gpu


def _python_only(monkeypatch):
    monkeypatch.setattr(dispatch, 'plain_autograd', lambda *t: False)
    monkeypatch.setattr(fused_moe, 'plain_autograd', lambda *t: False)


def _tokens(form, dtype):
    gen = torch.Generator(device='cuda').manual_seed(3)
    base = torch.randn(97, 64, generator=gen, device='cuda').to(dtype)
    if form == 'transposed':
        return base.t().contiguous().t()
    if form == 'off_vector':                             # contiguous, but not on a 16-byte boundary
        store = torch.empty(97 * 64 + 1, dtype=dtype, device='cuda')
        store[1:].copy_(base.view(-1))
        return store[1:].view(97, 64)
    return base


@pytest.mark.parametrize('dtype', [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize('form', ['plain', 'transposed', 'off_vector'])
@pytest.mark.parametrize('wants', ['both', 'tokens', 'gates', 'late_map', 'top1', 'top4'])
def test_encode_decode(monkeypatch, dtype, form, wants):
    def run():
        x = _tokens(form, dtype).detach().requires_grad_(wants != 'gates')
        logits = torch.randn(97, 5, generator=torch.Generator(device='cuda').manual_seed(4), device='cuda')
        logits.requires_grad_(wants != 'tokens')
        top_k = {'top1': 1, 'top4': 4}.get(wants, 2)
        crit, l_aux = extract_critical(F.softmax(logits, dim=1), top_k, capacity_factor=0.0 if wants == 'late_map' else 0.75)
        slots = fast_encode(x, crit)
        y = fast_decode(slots, crit)
        dy = _tokens(form, dtype).flip(0)
        outs, grads = [y], [dy]
        if l_aux.requires_grad:
            outs, grads = outs + [l_aux], grads + [torch.ones_like(l_aux)]
        torch.autograd.backward(outs, grads)
        return slots, y, l_aux, x.grad, logits.grad
    got = run()
    _python_only(monkeypatch)
    # routing itself has no Python node: without plain autograd it is the composition of library operations, which agrees
    # in slots, and in sums up to rounding (of the gates to the data's type: 2^-8 of a value, and of their gradients' terms)
    for a, b in zip(got, run()):
        assert (a is None) == (b is None)
        if a is not None:
            tol = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=1e-2, atol=2e-2)
            torch.testing.assert_close(a.float(), b.float(), **tol)


def test_decode_alone_is_the_python_function(monkeypatch):
    scores = F.softmax(torch.randn(200, 6, device='cuda'), dim=1).requires_grad_()
    crit, _ = extract_critical(scores, 2, loss_fn=None)
    disp = torch.randn(6 * crit[4], 40, device='cuda', dtype=torch.float16, requires_grad=True)
    dy = torch.randn(200, 40, device='cuda', dtype=torch.float16)

    def run():
        return torch.autograd.grad(fast_decode(disp, crit), [disp, *crit[3]], dy, retain_graph=True)
    got = run()
    _python_only(monkeypatch)
    assert all(torch.equal(a, b) for a, b in zip(got, run()))


def test_saved_tensor_hooks_and_a_second_backward():
    seen = []
    x = torch.randn(64, 32, device='cuda', requires_grad=True)
    scores = F.softmax(torch.randn(64, 4, device='cuda'), dim=1).requires_grad_()

    def pack(t):
        seen.append(t.shape)
        return t
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        crit, l_aux = extract_critical(scores, 2)
        y = fast_decode(fast_encode(x, crit), crit)
    assert len(seen) >= 6
    y.sum().backward(retain_graph=True)
    first = x.grad.clone()
    y.sum().backward()
    assert torch.equal(x.grad, 2 * first)
    with pytest.raises(RuntimeError):
        y.sum().backward()


@pytest.mark.parametrize('K,cf,postscore,int8,prio', [(2, 1.25, True, False, False), (1, 0.0, True, False, False), (2, 1.0, False, False, True),
                                                      (2, 1.0, True, True, False)])
def test_layer_is_the_python_function(monkeypatch, K, cf, postscore, int8, prio):
    torch.manual_seed(0)
    with torch.device('cuda'):
        layer = moe.moe_layer(gate_type={'type': 'top', 'k': K, 'capacity_factor': cf, 'fp32_gate': True}, model_dim=128,
                              experts={'type': 'ffn', 'count_per_node': 4, 'hidden_size_per_expert': 192, 'activation_fn': 'gelu'},
                              is_postscore=postscore, compress_name='int8' if int8 else 'no', batch_prioritized_routing=prio)
    layer = layer.cuda().bfloat16()
    layer.gates.float()
    x = torch.randn(333, 128, device='cuda', dtype=torch.bfloat16)
    dy = torch.randn(333, 128, device='cuda', dtype=torch.bfloat16)

    def run(outs, frozen):
        for p in layer.parameters():
            p.requires_grad_(True)
        layer.experts.batched_fc1_bias.requires_grad_(not frozen)
        xin = x.clone().requires_grad_(not frozen)
        layer.zero_grad(set_to_none=True)
        y = layer(xin)
        pairs = {'both': [(y, dy), (y.l_aux, None)], 'y': [(y, dy)], 'loss': [(y.l_aux, None)]}[outs]
        torch.autograd.backward([o for o, _ in pairs], [g for _, g in pairs])
        return [y.detach(), y.l_aux.detach(), xin.grad] + [p.grad for p in layer.parameters()] + [layer.last_stats['capacity']]
    forms = [('both', False), ('y', False), ('loss', False), ('both', True)]
    got = [run(*f) for f in forms]
    _python_only(monkeypatch)
    for a, b in zip(got, [run(*f) for f in forms]):
        assert all((p is None and q is None) or (torch.equal(p, q) if torch.is_tensor(p) else p == q) for p, q in zip(a, b))
