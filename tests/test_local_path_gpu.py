"""One rank without the exchange against the exchange of one rank (PLANMOE_LOCAL=0), over the forms both take: capacities
that are no multiple of a row block, experts without a token, dropped tokens, every number of picks."""

import contextlib
import os
import subprocess
import sys
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 2.0 ** -7          # one bf16 rounding of an intermediate, on either side


def _layer(E, M, H, k, cf, act='gelu', fp32_gate=True, **kw):
    from planmoe_b200 import moe
    layer = moe.moe_layer(gate_type={'type': 'top', 'k': k, 'capacity_factor': cf, 'fp32_gate': fp32_gate}, model_dim=M,
                          experts={'type': 'ffn', 'count_per_node': E, 'hidden_size_per_expert': H, 'activation_fn': act},
                          seeds=(1, 2, 3), **kw)
    layer = layer.cuda()
    gate = layer.gates[0].wg.weight.detach().clone()
    layer = layer.to(torch.bfloat16)
    if fp32_gate:
        layer.gates.float()
        layer.gates[0].wg.weight.data.copy_(gate)         # all 24 bits of it
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
                                      (2048, 4, 4, 0.3), (3001, 6, 2, 1.25), (600, 64, 2, 1.0), (4100, 16, 2, 1.0), (5000, 9, 2, 0.0)])
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


@pytest.mark.parametrize('local', ['1', '0'])
@pytest.mark.parametrize('wire', ['no', 'int8'])
def test_rows_off_the_vector_boundary(local, wire, monkeypatch):
    monkeypatch.setenv('PLANMOE_LOCAL', local)
    layer = _layer(2, 128, 256, 2, 1.0, compress_name=wire)
    off = [torch.randn(320 * 128 + 1, device='cuda').bfloat16()[1:].view(320, 128) for _ in range(2)]
    assert all(t.data_ptr() % 16 for t in off)
    with torch.no_grad():
        assert torch.equal(layer(off[0]), layer(off[0].clone()))
    from planmoe_b200.parallel import transport
    got = []
    for place in (lambda t: t, torch.clone):
        x = place(off[0].detach()).requires_grad_()
        layer.zero_grad(set_to_none=True)
        layer(x).backward(place(off[1]))
        got.append([x.grad] + [p.grad for p in layer.parameters()])
    transport.get_transport(layer.group).check()
    for u, v in zip(*got):
        assert torch.equal(u, v)


@contextlib.contextmanager
def _poisoned():
    """New floating-point tensors start as NaN."""
    before = torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled()
    fill = torch.utils.deterministic.fill_uninitialized_memory
    torch.use_deterministic_algorithms(True, warn_only=True)
    torch.utils.deterministic.fill_uninitialized_memory = True
    try:
        yield
    finally:
        torch.use_deterministic_algorithms(before[0], warn_only=before[1])
        torch.utils.deterministic.fill_uninitialized_memory = fill


@pytest.mark.parametrize('wire', ['no', 'int8'])
def test_unused_rows_are_never_read(wire):
    """Rows behind an expert's last used block are not written (they keep the NaN that every tensor starts with here), and
    show up in no result; two experts have no token at all."""
    from planmoe_b200.ops import native
    from planmoe_b200.parallel import transport
    layer = _layer(4, 128, 256, 2, 4.0, compress_name=wire)
    with torch.no_grad():
        layer.gates[0].wg.weight[2:].mul_(0).sub_(0.05)   # tokens with a positive sum never reach experts 2 and 3
    torch.manual_seed(6)
    x = torch.rand(500, 128, device='cuda').bfloat16()
    dy = torch.randn(500, 128, device='cuda').bfloat16()
    first = _pass(layer, x, dy)
    ex, tr = layer.experts, transport.get_transport(layer.group)
    with _poisoned():
        again = _pass(layer, x, dy)
        out, capacity = native.lib().local_moe_forward(
            x, layer.gates[0].wg.weight, ex.batched_fc1_w, ex.batched_fc1_bias, ex.batched_fc2_w, ex.batched_fc2_bias, 2, 1000,
            None, True, False, False, 1, True, wire == 'int8', tr.budget_ms, tr.status.device_ptr(), True, None)
    for u, v in zip(first, again):
        assert torch.equal(u, v) and torch.isfinite(u).all()
    used, rows, h = out[5].tolist(), out[9], out[11]
    assert used == [500, 500, 0, 0] and rows.size(1) >= capacity
    for slots in (rows, h):
        assert slots[:2, 512:].isnan().all() and slots[2:, 256:].isnan().all()
        assert torch.isfinite(slots[:2, :512]).all() and torch.isfinite(slots[2:, :256]).all()


@pytest.mark.parametrize('fp32_gate,S', [(False, 33), (False, 4097), (True, 515)])
def test_gate_forms(fp32_gate, S, monkeypatch):
    """A bf16 gate (logits and balance loss in bf16), a bf16 weight under an fp32 gate, and a gate that somebody listens to."""
    layer = _layer(2, 320, 128, 2, 1.0, fp32_gate=fp32_gate)
    layer.gates[0].to(torch.bfloat16)
    torch.manual_seed(2)
    x = torch.randn(S, 320, device='cuda').bfloat16()
    dy = torch.randn(S, 320, device='cuda').bfloat16()
    here = _pass(layer, x, dy)
    with torch.no_grad():
        layer(x)
    assert layer.l_aux.dtype == (torch.float32 if fp32_gate else torch.bfloat16)
    seen = []
    handle = layer.gates[0].wg.register_forward_hook(lambda mod, args, out: seen.append(out.shape))
    if not fp32_gate:                                     # an fp32 gate uses the weight without calling the linear module
        hooked = _pass(layer, x, dy)
        assert seen == [(S, 2)]
        _close(here, hooked)
    handle.remove()
    monkeypatch.setenv('PLANMOE_LOCAL', '0')
    _close(here, _pass(layer, x, dy))


@pytest.mark.parametrize('S,E,M', [(1, 1, 64), (37, 3, 96), (4096, 8, 2048), (4113, 16, 1056)])
def test_projection_is_at_fp32_precision(S, E, M):
    """Logits and the weight's gradient against 64 bits, no further off than an fp32 GEMM is."""
    from planmoe_b200.ops import native
    torch.manual_seed(0)
    layer = _layer(E, M, 64, 1, 1.0)
    x = torch.randn(S, M, device='cuda').bfloat16()
    w = layer.gates[0].wg.weight
    ex = layer.experts
    from planmoe_b200.parallel import transport
    tr = transport.get_transport(layer.group)
    out, _cap = native.lib().local_moe_forward(x, w, ex.batched_fc1_w, ex.batched_fc1_bias, ex.batched_fc2_w, ex.batched_fc2_bias,
                                               1, 4 * S, None, True, False, False, 1, True, False, tr.budget_ms,
                                               tr.status.device_ptr(), True, None)
    logits = out[2].double()
    ref = x.double() @ w.detach().double().t()
    lib = (x.float() @ w.detach().float().t()).double()
    # 2^-22 of the largest sum of magnitudes: two roundings, whatever order the library added in
    slack = 2.0 ** -22 * float((x.double().abs() @ w.detach().double().abs().t()).max())
    assert float((logits - ref).abs().max()) <= max(float((lib - ref).abs().max()), slack)


def test_priority_order_is_a_permutation_whatever_the_scores():
    """Ties, NaN rows, more than one key tile, a token count that no tile divides: ranks and order stay inverse to each other."""
    from planmoe_b200.ops import native
    torch.manual_seed(0)
    for S in (1, 63, 4097, 9473, 20000):
        logits = torch.randn(S, 8, device='cuda')
        logits[S // 2] = float('nan')
        logits[: S // 3] = logits[0]
        rank, perm = native.lib().importance_order(logits)
        assert torch.equal(rank[perm.long()], torch.arange(S, device='cuda', dtype=torch.int32))
        key = torch.softmax(logits, 1).max(1).values.nan_to_num(0.0)
        ordered = key[perm.long()]
        assert bool((ordered[:-1] >= ordered[1:] - 2e-7).all())
        tied = rank[: S // 3]
        assert bool((tied[1:] > tied[:-1]).all())          # equal keys: token order


@pytest.mark.parametrize('S,E,k,cf', [(32, 1, 1, 1.0), (768, 3, 2, 1.0), (1000, 5, 2, 0.0), (2048, 32, 2, 1.0)])
def test_int8_rows_match_the_exchange(S, E, k, cf, monkeypatch):
    """Rows quantised and expanded where the slots are filled against wire rows, landing buffer and de-quantiser role."""
    layer = _layer(E, 256, 384, k, cf, compress_name='int8')
    torch.manual_seed(9)
    x = torch.randn(S, 256, device='cuda').bfloat16()
    x[S // 3] = 0.5                                       # a constant row has no range
    dy = torch.randn(S, 256, device='cuda').bfloat16()
    here = _pass(layer, x, dy)
    assert layer.last_stats['wire'] == 'int8' and layer.last_stats['capacity'] % 32 == 0      # the exchange takes no other
    monkeypatch.setenv('PLANMOE_LOCAL', '0')
    _close(here, _pass(layer, x, dy))


def _int8_close(a, b):
    """Rows of normal values have a range of at most 6.5 standard deviations, a step of a 255th of that and so a relative
    error of 0.0074 (2-norm); a result has met at most two or three such roundings, independent of one another."""
    for u, v in zip(a, b):
        assert u.dtype == v.dtype and torch.isfinite(u).all()
        assert float((u.float() - v.float()).norm()) <= 3e-2 * float(v.float().norm()), u.shape


@pytest.mark.parametrize('plain_gate', [True, False])
@pytest.mark.parametrize('S,E,k,cf,capacity,ample', [(30, 8, 1, 1.0, 4, (5.0, 8.0)), (390, 8, 2, 1.0, 100, (2.7, 2.6)),
                                                     (1000, 8, 2, 1.01, 252, (2.0, 2.05)), (4805, 8, 2, 1.0, 1204, (2.0, 2.05))])
def test_int8_capacities_of_every_remainder(S, E, k, cf, capacity, ample, plain_gate):
    """Capacities that are no whole slices of 32 rows: the same tokens are dropped as without int8, and where none is, the
    layout makes no difference to any bit."""
    layers = [_layer(E, 256, 384, k, 1.0, compress_name=name) for name in ('int8', 'no')]
    torch.manual_seed(11)
    x = torch.randn(S, 256, device='cuda').bfloat16()
    dy = torch.randn(S, 256, device='cuda').bfloat16()
    for layer in layers:
        layer.collect_stats = True
        if not plain_gate:                                # somebody listens to the gate: its own node, the experts another
            layer.gates[0].register_forward_hook(lambda mod, args, out: None)

    def run(layer, factor):
        layer.gates[0].capacity_factor = factor
        return _pass(layer, x, dy), layer.last_stats

    (got, stats), (plain, _) = (run(layer, cf) for layer in layers)
    assert stats['capacity'] == capacity and stats['path'] == 'fused' and int(stats['tokens_dropped']) > 0
    assert torch.equal((got[0] == 0).all(1), (plain[0] == 0).all(1))
    _int8_close(got, plain)
    (odd, odd_stats), (whole, whole_stats) = (run(layers[0], factor) for factor in ample)
    assert int(odd_stats['tokens_dropped']) == int(whole_stats['tokens_dropped']) == 0
    assert odd_stats['capacity'] % 32 and whole_stats['capacity'] % 32 == 0
    for u, v in zip(odd, whole):
        assert torch.equal(u, v)


def test_int8_dynamic_capacity_of_a_deep_pipeline():
    """The ladder of dynamic capacities has steps of 4 * degree: 80 slots here."""
    layer = _layer(5, 256, 384, 2, 0.0, compress_name='int8')
    torch.manual_seed(12)
    x = torch.randn(120, 256, device='cuda').bfloat16()
    dy = torch.randn(120, 256, device='cuda').bfloat16()
    got = _pass(layer, x, dy, degree=20)
    assert layer.last_stats['capacity'] % 32
    for u, v in zip(got, _pass(layer, x, dy, degree=1)):
        assert torch.equal(u, v)


@pytest.mark.parametrize('S,cf,degree,path', [(1000, 1.01, 1, 'generic'), (1024, 1.0, 1, 'fused'), (1024, 1.0, 3, 'generic'),
                                              (1000, 0.0, 1, 'fused'), (1000, 0.0, 3, 'fused'), (1000, 0.0, 20, 'fused')])
def test_int8_exchange_takes_whole_slices_only(S, cf, degree, path, monkeypatch):
    """Static capacities that are no whole slices per chunk take the generic path, dynamic ones are sized to fit."""
    layer = _layer(8, 256, 384, 2, cf, compress_name='int8')
    torch.manual_seed(13)
    x = torch.randn(S, 256, device='cuda').bfloat16()
    dy = torch.randn(S, 256, device='cuda').bfloat16()
    here = _pass(layer, x, dy, degree=degree)
    assert layer.last_stats['path'] == 'fused'
    monkeypatch.setenv('PLANMOE_LOCAL', '0')
    there = _pass(layer, x, dy, degree=degree)
    assert layer.last_stats['path'] == path
    if cf == 0:
        assert layer.last_stats['capacity'] % (32 * degree) == 0
    _int8_close(here, there)


@pytest.mark.parametrize('fp32_gate', [True, False])
@pytest.mark.parametrize('S,M,E,k', [(500, 128, 4, 2), (33, 320, 9, 1)])
def test_backward_of_the_balance_loss_alone(S, M, E, k, fp32_gate, monkeypatch):
    """The experts take no part in it: no gradient, rather than one of zeros that an optimizer would act on."""
    layer = _layer(E, M, 256, k, 1.0, fp32_gate=fp32_gate)
    torch.manual_seed(14)
    x0 = torch.randn(S, M, device='cuda').bfloat16()
    out = []
    for local in ('1', '0'):
        monkeypatch.setenv('PLANMOE_LOCAL', local)
        x = x0.clone().requires_grad_()
        layer.zero_grad(set_to_none=True)
        layer(x).l_aux.backward()
        out.append([x.grad] + [p.grad for p in layer.parameters()])
        layer.l_aux = None
    assert sum(g is not None for g in out[0]) == 2
    _close(*out)


@pytest.mark.parametrize('local', ['0', '1'])
@pytest.mark.parametrize('plain_gate', [True, False])
def test_forward_mode_is_refused_without_gradients_too(local, plain_gate, monkeypatch):
    """No tangent is dropped: the kernels have no forward-mode rule, with or without the exchange."""
    import torch.autograd.forward_ad as fwAD
    monkeypatch.setenv('PLANMOE_LOCAL', local)
    layer = _layer(4, 128, 256, 2, 1.0)
    if not plain_gate:
        layer.gates[0].register_forward_hook(lambda mod, args, out: out.detach())
    x = torch.randn(64, 128, device='cuda').bfloat16()
    with torch.no_grad():
        with fwAD.dual_level():
            with pytest.raises(NotImplementedError, match='jvp'):
                layer(fwAD.make_dual(x, torch.ones_like(x)))
        with pytest.raises(Exception):
            torch.func.vmap(layer)(x.view(2, 32, 128))
        assert torch.isfinite(layer(x)).all()


def test_other_threads_run_while_the_capacity_is_awaited():
    layer = _layer(4, 128, 256, 2, 0.0)
    x = torch.randn(512, 128, device='cuda').bfloat16()
    beats, done = [], threading.Event()

    def beat():
        while not done.wait(0.005):
            beats.append(time.perf_counter())

    with torch.no_grad():
        layer(x)
        torch.cuda.synchronize()
        other = threading.Thread(target=beat)
        other.start()
        try:
            torch.cuda._sleep(900_000_000)                # about half a second of device time in front of the layer
            start = time.perf_counter()
            layer(x)
            end = time.perf_counter()
        finally:
            done.set()
            other.join()
    assert end - start > 0.1
    assert sum(start < t < end for t in beats) > 5


@pytest.mark.parametrize('degree', [1, 3, 20])
def test_stats_say_what_ran(degree, monkeypatch):
    """A dynamic capacity is a multiple of 4 * degree whichever way the layer runs, and no exchange is called none."""
    layer = _layer(4, 128, 256, 2, 0.0)
    torch.manual_seed(15)
    x = torch.randn(300, 128, device='cuda').bfloat16()
    seen = []
    for local in ('1', '0'):
        monkeypatch.setenv('PLANMOE_LOCAL', local)
        with torch.no_grad():
            layer(x, a2a_ffn_overlap_degree=degree)
        seen.append(layer.last_stats)
    assert seen[0]['capacity'] == seen[1]['capacity'] and seen[0]['capacity'] % (4 * degree) == 0
    assert [s['comm'] for s in seen] == ['none', 'flat-push']


_VARIANT_CHILD = """
import os, torch
from tests.test_local_path_gpu import _close, _layer, _pass
torch.use_deterministic_algorithms(True, warn_only=True)
torch.utils.deterministic.fill_uninitialized_memory = True    # new tensors start as NaN
layer = _layer(4, 128, 256, 2, 2.0)
x = torch.randn(700, 128, device='cuda').bfloat16()
dy = torch.randn_like(x)
here = _pass(layer, x, dy)
os.environ['PLANMOE_LOCAL'] = '0'
_close(here, _pass(layer, x, dy))
print('same')
"""


def test_measuring_switch_of_the_send_variant_changes_no_result():
    """PLANMOE_GEMM_COPY_VARIANT=1 selects a kernel without column sums and used-row counts: launches that need them keep
    theirs.  The switch is read once per process."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    child = subprocess.run([sys.executable, '-c', _VARIANT_CHILD], cwd=root, capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, PLANMOE_GEMM_COPY_VARIANT='1', PYTHONPATH=root))
    assert child.returncode == 0 and 'same' in child.stdout, child.stderr[-2000:]
