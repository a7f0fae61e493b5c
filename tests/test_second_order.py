"""Gradients of gradients through encode, decode and the layer, against plain differentiable operations in 64 bits; what has no
second derivative says so instead of leaving a term out."""

import pytest
import torch
import torch.nn.functional as F

from planmoe_b200 import moe
from planmoe_b200.impls.fast_dispatch import extract_critical, fast_decode, fast_encode
from planmoe_b200.ops import dispatch as D
from planmoe_b200.ops import gemm

S, M, E, C = 9, 4, 3, 4


def _slots(device='cpu', dtype=torch.float64):
    """A plan with dropped picks and empty slots, tokens, slots and gates."""
    gen = torch.Generator().manual_seed(0)
    idx = torch.stack([torch.randperm(E, generator=gen)[:2] for _ in range(S)]).t().contiguous()
    hot = F.one_hot(idx.reshape(-1), E)
    loc = (hot.cumsum(0) * hot).sum(1).view(2, S) - 1
    make = lambda *shape: torch.randn(*shape, generator=gen, dtype=torch.float64).to(device, dtype).requires_grad_()   # noqa: E731
    plan = D.SlotPlan(idx.int().to(device), loc.int().to(device), E, C)
    return plan, make(S, M), make(E * C, M), make(2, S)


@pytest.mark.parametrize('gated', [False, True])
def test_encode_and_decode_twice_on_the_cpu(gated):
    plan, x, disp, gates = _slots()
    more = (gates,) if gated else ()
    assert torch.autograd.gradgradcheck(lambda t, *g: D.scatter(t, plan, *g), (x, *more))
    assert torch.autograd.gradgradcheck(lambda t, *g: D.gather(t, plan, *g), (disp, *more))


def _one_hot64(crit, S_):
    """[S, E * C] per pick: one where the pick owns the slot."""
    idx, loc = torch.stack(list(crit[1])).long(), torch.stack(list(crit[2])).long()
    kept = (loc < crit[4]).unsqueeze(2)
    return (F.one_hot((idx * crit[4] + loc).clamp_max(crit[0] * crit[4] - 1), crit[0] * crit[4]) * kept).double()


def _close(got, want, rel):
    for a, b in zip(got, want):
        assert float((a.double() - b).norm()) <= rel * float(b.norm()), (float((a.double() - b).norm()), float(b.norm()))


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize('postscore', [True, False])
@pytest.mark.parametrize('nodes', ['native', 'python'])
def test_routing_encode_decode_twice(monkeypatch, dtype, postscore, nodes):
    """d/d(tokens, scores) of |dL/dtokens|^2 + |dL/dscores|^2 with an L that is not linear in anything."""
    gen = torch.Generator(device='cuda').manual_seed(5)
    # of a quarter: the results are of fifth degree in the tokens and come to 8e5 for unit ones, more than fp16 holds
    x0 = (torch.randn(61, 32, generator=gen, device='cuda') * 0.25).to(dtype)
    s0 = F.softmax(torch.randn(61, 5, generator=gen, device='cuda'), dim=1)
    crit0, _ = extract_critical(s0, 2, capacity_factor=0.75)
    hot = _one_hot64(crit0, 61)
    if nodes == 'python':
        monkeypatch.setattr(D, 'plain_autograd', lambda *t: False)

    def twice(f, x, s):
        y = f(x, s)
        gx, gs = torch.autograd.grad(y.to(torch.float64).square().sum(), [x, s], create_graph=True)
        return (gx, gs) + torch.autograd.grad(gx.double().square().sum() + gs.double().square().sum(), [x, s])

    def ours(x, s):
        crit, _ = extract_critical(s, 2, capacity_factor=0.75)
        slots = fast_encode(x, crit, postscore)
        return fast_decode(slots * slots, crit, postscore)

    def plain(x, s):
        g = s.gather(1, torch.stack(list(crit0[1])).long().t())
        g = (g / g.sum(1, keepdim=True)).t().unsqueeze(2)
        weighted = (hot * g).sum(0)
        slots = (weighted if not postscore else hot.sum(0)).t() @ x
        return (weighted if postscore else hot.sum(0)) @ (slots * slots)
    got = twice(ours, x0.clone().requires_grad_(), s0.clone().requires_grad_())
    want = twice(plain, x0.double().requires_grad_(), s0.double().requires_grad_())
    # a chain of some twenty roundings to the data's type, in terms that hardly cancel
    _close(got, want, 20 * {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype])


@pytest.mark.gpu
@pytest.mark.parametrize('nodes', ['native', 'python'])
def test_gates_changed_since(monkeypatch, nodes):
    """A gradient uses the gates that decode was given; its own gradient, which runs through their history, refuses others."""
    if nodes == 'python':
        monkeypatch.setattr(D, 'plain_autograd', lambda *t: False)
    scores = F.softmax(torch.randn(40, 4, device='cuda'), dim=1)
    crit, _ = extract_critical(scores, 2)
    disp = torch.randn(4 * crit[4], 32, device='cuda', requires_grad=True)
    gates = [g.clone() for g in crit[3]]
    crit = (*crit[:3], gates, crit[4])
    y = fast_decode(disp, crit)
    before, = torch.autograd.grad(y.square().sum(), disp, retain_graph=True)
    gates[0].mul_(2)
    after, = torch.autograd.grad(y.square().sum(), disp, retain_graph=True)
    assert torch.equal(before, after)
    with pytest.raises(RuntimeError, match='inplace'):
        torch.autograd.grad(y.square().sum(), disp, create_graph=True)


def _layer(dtype, **more):
    torch.manual_seed(1)
    with torch.device('cuda'):
        layer = moe.moe_layer(gate_type={'type': 'top', 'k': 2, 'capacity_factor': 1.0}, model_dim=64,
                              experts={'type': 'ffn', 'count_per_node': 4, 'hidden_size_per_expert': 64, 'activation_fn': 'gelu'}, **more)
    return layer.cuda().to(dtype)


@pytest.mark.gpu
@pytest.mark.parametrize('fused', ['1', '0'])
def test_fp32_layer_twice(monkeypatch, fused):
    """The node of the fp32 layer and the generic path, each against 64 bits."""
    from planmoe_b200.ops import layer32
    if fused == '0':
        monkeypatch.setattr(layer32, 'takes', lambda *a: False)
    layer = _layer(torch.float32)
    ex, wg = layer.experts, layer.gates[0].wg.weight
    params = [wg, ex.batched_fc1_w, ex.batched_fc1_bias, ex.batched_fc2_w, ex.batched_fc2_bias]
    x = torch.randn(40, 64, device='cuda')
    crit, _ = extract_critical(F.softmax(F.linear(x, wg.detach()), dim=1), 2, alignment=4)
    hot, C_ = _one_hot64(crit, 40), crit[4]

    def twice(f, inputs):
        y, l_aux = f(*inputs)
        found = torch.autograd.grad(y.square().sum() + l_aux, inputs, create_graph=True)
        return found + torch.autograd.grad(sum(g.square().sum() for g in found), inputs)

    def plain(x, wg, w1, b1, w2, b2):
        s = F.softmax(x @ wg.t(), dim=1)
        g = s.gather(1, torch.stack(list(crit[1])).long().t())
        weighted = (hot * (g / g.sum(1, keepdim=True)).t().unsqueeze(2)).sum(0)
        slots = (hot.sum(0).t() @ x).view(4, C_, -1)
        out = F.gelu(slots @ w1 + b1.unsqueeze(1)) @ w2 + b2.unsqueeze(1)
        top1 = F.one_hot(crit[1][0].long(), 4).sum(0)
        return weighted @ out.view(4 * C_, -1), (s.sum(0) * top1).sum() * 4 / 40 ** 2

    def ours(xin, *_):
        y = layer(xin)
        return y, y.l_aux
    got = twice(ours, [x.clone().requires_grad_()] + params)
    want = twice(plain, [t.detach().double().requires_grad_() for t in [x] + params])
    _close(got, want, 1e-5)                              # some twenty fp32 roundings of sums of up to 64 terms


@pytest.mark.gpu
@pytest.mark.parametrize('path', ['layer', 'timers', 'experts', 'exchange', 'ffn', 'gate'])
def test_no_second_derivative_is_an_error(monkeypatch, path):
    """First derivatives under create_graph are the ordinary ones; using their graph raises."""
    from planmoe_b200.utils import stage_timer
    if path == 'exchange':
        monkeypatch.setenv('PLANMOE_LOCAL', '0')
    layer = _layer(torch.bfloat16, **({'is_gshard_loss': False} if path == 'experts' else {}))
    if path == 'timers':
        stage_timer.enable()
    x = torch.randn(40, 64, device='cuda', dtype=torch.bfloat16)
    ex = layer.experts

    def run(create):
        xin = x.clone().requires_grad_()
        if path == 'ffn':
            y = gemm.expert_ffn(xin.view(4, 10, 64), ex.batched_fc1_w, ex.batched_fc1_bias, ex.batched_fc2_w, ex.batched_fc2_bias, 'gelu')
        elif path == 'gate':
            from planmoe_b200.ops.fused_moe import fused_gate
            y = fused_gate(xin, 2, 8, True)[0]
        else:
            y = layer(xin)
        w = xin if path == 'gate' else ex.batched_fc1_w
        return torch.autograd.grad(y.float().square().sum(), [xin, w], create_graph=create), xin
    try:
        (want, _), (got, xin) = run(False), run(True)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        # by anything that the gradients depend on, also beside terms that are sound
        more = {'gate': [], 'ffn': [ex.batched_fc1_bias, ex.batched_fc2_w]}.get(path, [ex.batched_fc2_bias, layer.gates[0].wg.weight])
        for by in [xin] + more:
            with pytest.raises(RuntimeError, match='differentiated twice'):
                torch.autograd.grad(got[0].float().square().sum() + by.float().square().sum(), by, retain_graph=True)
    finally:
        stage_timer.enable(False)
