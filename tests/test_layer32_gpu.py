"""The fp32 layer of one rank as one node against the generic path."""

import pytest
import torch

from planmoe_b200 import moe
from planmoe_b200.ops import layer32

pytestmark = pytest.mark.gpu


def _layer(E, K, cf, act, M, H, **more):
    torch.manual_seed(1)
    with torch.device('cuda'):
        layer = moe.moe_layer(gate_type={'type': 'top', 'k': K, 'capacity_factor': cf}, model_dim=M,
                              experts={'type': 'ffn', 'count_per_node': E, 'hidden_size_per_expert': H, 'activation_fn': act}, **more)
    return layer.cuda()


def _watch(monkeypatch):
    took, takes = [], layer32.takes

    def watched(*a):
        took.append(takes(*a))
        return took[-1]
    monkeypatch.setattr(layer32, 'takes', watched)
    return took


def _both(monkeypatch, run):
    took = _watch(monkeypatch)
    got = run()
    assert took and took[0]
    monkeypatch.setattr(layer32, 'takes', lambda *a: False)
    return got, run()


def _same(got, want):
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        if a is not None:                                # the same products; sums of up to 1000 terms in another order
            torch.testing.assert_close(a, b, rtol=1e-5, atol=2e-5)


@pytest.mark.parametrize('E,K,cf,act,S,M,H', [(8, 2, 1.0, 'relu', 512, 256, 512), (2, 1, 1.25, 'gelu', 65, 66 * 2, 77), (7, 2, 0.5, 'silu', 300, 64, 65),
                                              (4, 4, 2.0, 'relu', 33, 128, 129), (1, 1, 1.0, 'gelu', 64, 64, 64)])
@pytest.mark.parametrize('outs', ['both', 'y', 'loss', 'frozen_experts', 'frozen_tokens', 'none'])
def test_passes(monkeypatch, E, K, cf, act, S, M, H, outs):
    layer = _layer(E, K, cf, act, M, H)
    x, dy = torch.randn(S, M, device='cuda'), torch.randn(S, M, device='cuda')

    def run():
        for n, p in layer.named_parameters():
            p.requires_grad_(outs != 'none' and not (outs == 'frozen_experts' and 'fc' in n))
        xin = x.clone().requires_grad_(outs not in ('none', 'frozen_tokens'))
        layer.zero_grad(set_to_none=True)
        y = layer(xin)
        pairs = {'loss': [(y.l_aux, None)], 'y': [(y, dy)], 'none': []}.get(outs, [(y, dy), (y.l_aux, None)])
        if pairs:
            torch.autograd.backward([o for o, _ in pairs], [g for _, g in pairs])
        assert layer.last_stats['path'] == 'generic'
        return [y.detach(), y.l_aux.detach(), xin.grad] + [p.grad for p in layer.parameters()]
    _same(*_both(monkeypatch, run))


def test_gradient_of_a_gradient(monkeypatch):
    layer = _layer(4, 2, 1.0, 'gelu', 64, 32)
    x = torch.randn(40, 64, device='cuda', requires_grad=True)

    def run():
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        w = layer.experts.batched_fc1_w
        g, = torch.autograd.grad(y.square().sum() + y.l_aux, w, create_graph=True)
        g.square().sum().backward()
        return [g.detach(), w.grad, layer.experts.batched_fc2_w.grad]
    got, want = _both(monkeypatch, run)
    for a, b in zip(got, want):                          # sums of squares: relative to their size
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))


@pytest.mark.parametrize('what', ['hook', 'autocast', 'tf32', 'noise', 'prio', 'dynamic', 'bf16', 'dual_level', 'stats'])
def test_other_calls_stay_where_they_were(monkeypatch, what):
    layer = _layer(4, 2, 0.0 if what == 'dynamic' else 1.0, 'relu', 64, 32, batch_prioritized_routing=what == 'prio')
    x = torch.randn(40, 64, device='cuda')
    took = _watch(monkeypatch)
    if what == 'hook':
        layer.experts.register_forward_hook(lambda m, i, o: None)
    elif what == 'noise':
        layer.gates[0].gate_noise = 1.0
    elif what == 'tf32':
        monkeypatch.setattr(torch.backends.cuda.matmul, 'allow_tf32', True)
    elif what == 'stats':
        layer.collect_stats = True
    elif what == 'bf16':
        layer.bfloat16()
        x = x.bfloat16()
    if what == 'dual_level':
        with torch.no_grad(), torch.autograd.forward_ad.dual_level():
            layer(x)
    else:
        with torch.autocast('cuda', enabled=what == 'autocast'):
            layer(x)
    assert took and not any(took)


@pytest.mark.parametrize('where', ['matmul', 'all'])
@pytest.mark.parametrize('precision', ['tf32', 'ieee'])
def test_fp32_precision_switches(monkeypatch, where, precision):
    """The present switches (the legacy flag cannot be read once one of them is set to TF32): full precision takes the node."""
    holder = torch.backends.cuda.matmul if where == 'matmul' else torch.backends
    layer = _layer(4, 2, 1.0, 'gelu', 64, 32)
    x = torch.randn(40, 64, device='cuda')
    took, before = _watch(monkeypatch), [(h, h.fp32_precision) for h in (torch.backends, torch.backends.cuda.matmul)]

    def run():
        layer.zero_grad(set_to_none=True)
        xin = x.clone().requires_grad_()
        y = layer(xin)
        (y.square().sum() + y.l_aux).backward()
        return [y.detach(), y.l_aux.detach(), xin.grad] + [p.grad for p in layer.parameters()]
    try:
        torch.backends.cuda.matmul.fp32_precision = 'none'       # products follow the switch for all operations
        holder.fp32_precision = precision
        got = run()
        assert took == [precision == 'ieee']
        monkeypatch.setattr(layer32, 'takes', lambda *a: False)
        want = run()
    finally:
        for h, value in before:
            h.fp32_precision = value
    for a, b in zip(got, want):                          # sums of up to 64 terms in another order; TF32: the same operations
        torch.testing.assert_close(a, b, rtol=1e-5, atol=2e-5)


def test_more_chunks_than_transfers_are_refused():
    layer = _layer(4, 2, 1.0, 'relu', 64, 32)
    x = torch.randn(600, 64, device='cuda')
    from planmoe_b200.impls.communicate import AllToAllStatus
    layer(x, a2a_ffn_overlap_degree=AllToAllStatus.max_num_split)
    assert (AllToAllStatus.num_split, AllToAllStatus.split_dim) == (AllToAllStatus.max_num_split, 1)
    with pytest.raises(AssertionError):
        layer(x, a2a_ffn_overlap_degree=2 * AllToAllStatus.max_num_split)


@pytest.mark.parametrize('what', ['expert_local', 'route', 'comm', 'codec'])
def test_parts_of_the_generic_path_put_in_place(monkeypatch, what):
    """A subclass's methods and algorithms registered under a built-in name are the ones that run."""
    from planmoe_b200.impls.moe_layer import MOELayer
    from planmoe_b200.parallel import codecs, comms
    seen = []

    class Local(MOELayer):
        def expert_local(self, x, reserve_shape):
            seen.append('expert_local')
            return super().expert_local(x, reserve_shape)

    class Route(MOELayer):
        def _route(self, *a):
            seen.append('route')
            return super()._route(*a)

    class Comm(comms.NaiveComm):
        def all_to_all(self, t):
            seen.append('comm')
            return super().all_to_all(t)

    class Codec(codecs.NoCompressor):
        def compress(self, *a, **k):
            seen.append('codec')
            return super().compress(*a, **k)
    layer = _layer(4, 2, 1.0, 'relu', 64, 32)
    if what in ('expert_local', 'route'):
        layer.__class__ = {'expert_local': Local, 'route': Route}[what]
    elif what == 'comm':
        monkeypatch.setitem(comms._REGISTRY, 'naive', Comm)
    else:
        monkeypatch.setitem(codecs._REGISTRY, 'no', Codec)
    layer(torch.randn(40, 64, device='cuda'))
    assert what in seen
