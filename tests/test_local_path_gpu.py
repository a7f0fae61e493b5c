"""One rank without the exchange against the exchange of one rank (PLANMOE_LOCAL=0), over the forms both take: capacities
that are no multiple of a row block, experts without a token, dropped tokens, every number of picks."""

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 2.0 ** -7          # one bf16 rounding of an intermediate, on either side


def _layer(E, M, H, k, cf, act='gelu', **kw):
    from planmoe_b200 import moe
    layer = moe.moe_layer(gate_type={'type': 'top', 'k': k, 'capacity_factor': cf, 'fp32_gate': True}, model_dim=M,
                          experts={'type': 'ffn', 'count_per_node': E, 'hidden_size_per_expert': H, 'activation_fn': act},
                          seeds=(1, 2, 3), **kw)
    layer = layer.cuda().to(torch.bfloat16)
    layer.gates.float()
    return layer


def _pass(layer, x0, dy, degree=None):
    from planmoe_b200.parallel import transport
    x = x0.clone().requires_grad_()
    layer.zero_grad(set_to_none=True)
    y = layer(x, a2a_ffn_overlap_degree=degree)
    torch.autograd.backward([y, y.l_aux], [dy, torch.full_like(y.l_aux, 0.1)])
    transport.get_transport(layer.group).check()
    out = [y.detach(), x.grad] + [p.grad for p in layer.parameters()]
    layer.l_aux = None
    return out


def _close(a, b):
    assert len(a) == len(b)
    for u, v in zip(a, b):
        if v is None:
            assert u is None
            continue
        assert u.dtype == v.dtype and torch.isfinite(u).all()
        top = float(v.float().abs().max())
        assert float((u.float() - v.float()).abs().max()) <= TOL * top, (u.shape, top)


@pytest.mark.parametrize('S,E,k,cf', [(1, 1, 1, 1.0), (16, 8, 2, 2.0), (130, 3, 3, 1.0), (700, 5, 1, 0.0), (1000, 2, 2, 1.0),
                                      (2048, 4, 4, 0.3), (3001, 6, 2, 1.25), (600, 64, 2, 1.0)])
@pytest.mark.parametrize('postscore', [True, False])
def test_matches_the_exchange(S, E, k, cf, postscore, monkeypatch):
    layer = _layer(E, 192, 320, k, cf, is_postscore=postscore)
    torch.manual_seed(5)
    x = torch.randn(S, 192, device='cuda').bfloat16()
    dy = torch.randn(S, 192, device='cuda').bfloat16()
    here = _pass(layer, x, dy)
    with torch.no_grad():
        assert torch.equal(layer(x), here[0])             # no derivative saved: the same forward
    monkeypatch.setenv('PLANMOE_LOCAL', '0')
    _close(here, _pass(layer, x, dy))


@pytest.mark.parametrize('act', ['relu', 'silu', 'identity'])
def test_experts_without_tokens_and_frozen_weights(act, monkeypatch):
    layer = _layer(6, 128, 256, 2, 1.0, act=act, batch_prioritized_routing=True)
    with torch.no_grad():
        layer.gates[0].wg.weight[2:].mul_(0).sub_(0.05)   # tokens with a positive sum never reach experts 2 .. 5
    layer.experts.batched_fc1_w.requires_grad_(False)
    layer.experts.batched_fc2_bias.requires_grad_(False)
    torch.manual_seed(1)
    x = torch.rand(900, 128, device='cuda').bfloat16()
    dy = torch.randn(128, 900, device='cuda').bfloat16().t()          # a strided gradient
    here = _pass(layer, x, dy, degree=2)
    monkeypatch.setenv('PLANMOE_LOCAL', '0')
    _close(here, _pass(layer, x, dy, degree=2))


def test_rows_off_the_vector_boundary():
    layer = _layer(2, 128, 256, 2, 1.0)
    x = torch.randn(300 * 128 + 1, device='cuda').bfloat16()
    off = x[1:].view(300, 128)
    assert off.data_ptr() % 16
    with torch.no_grad():
        assert torch.equal(layer(off), layer(off.clone()))


def test_unused_rows_are_never_read():
    """Memory that an earlier tensor left behind as NaN shows up nowhere, whatever the blocks behind the used rows hold."""
    layer = _layer(4, 128, 256, 2, 4.0)
    x = torch.randn(500, 128, device='cuda').bfloat16()
    dy = torch.randn(500, 128, device='cuda').bfloat16()
    first = _pass(layer, x, dy)
    torch.full((64 << 20,), float('nan'), device='cuda')              # freed at once: the next pass may be given it
    again = _pass(layer, x, dy)
    for u, v in zip(first, again):
        assert torch.equal(u, v) and torch.isfinite(u).all()
