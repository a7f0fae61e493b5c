"""``extract_critical`` on the routing kernels against its ATen composition: every form that the kernels accept."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(scores, monkeypatch, **kw):
    """(kernel result, composition result), each with its own leaf."""
    from planmoe_b200.impls import fast_dispatch as FD
    from planmoe_b200.jit_kernels import gating
    out = []
    for fast in (True, False):
        monkeypatch.setattr(gating, 'use_fast_cumsum', fast)
        leaf = scores.detach().clone().requires_grad_()
        view = leaf.t() if kw.get('transposed') else leaf
        args = {k: v for k, v in kw.items() if k != 'transposed'}
        out.append((leaf, *FD.extract_critical(view, **args)))
    return out


@pytest.mark.parametrize('S,E,k', [(1, 1, 1), (5, 3, 2), (127, 8, 2), (128, 9, 1), (129, 16, 4), (1000, 33, 3), (4097, 64, 2)])
@pytest.mark.parametrize('cf', [1.0, 0.4, 0.0, -0.5])
@pytest.mark.parametrize('normalize', [True, False])
def test_matches_composition(S, E, k, cf, normalize, monkeypatch):
    torch.manual_seed(S + E)
    scores = torch.softmax(torch.randn(S, E, device='cuda'), dim=1)
    transposed = S == 129
    if transposed:
        scores = scores.t().contiguous()
    (a, pa, la), (b, pb, lb) = _both(scores, monkeypatch, top_k=k, capacity_factor=cf, normalize_gate=normalize, alignment=4,
                                     transposed=transposed)
    assert pa[0] == pb[0] and pa[4] == pb[4]
    for i in (1, 2):
        assert len(pa[i]) == len(pb[i]) == k
        for u, v in zip(pa[i], pb[i]):
            assert u.dtype == v.dtype and torch.equal(u, v)
    for u, v in zip(pa[3], pb[3]):
        torch.testing.assert_close(u, v, rtol=4e-7, atol=0)          # a division of sums of at most four scores
    torch.testing.assert_close(la, lb, rtol=2e-6, atol=0)            # S * E positive terms, another order
    assert torch.equal(pa.slots.slot_map, pb.slots.slot_map)
    weights = [torch.randn(S, device='cuda') for _ in range(k)]
    for leaf, p, l in ((a, pa, la), (b, pb, lb)):
        (sum((g * w).sum() for g, w in zip(p[3], weights)) + 0.3 * l).backward()
    torch.testing.assert_close(a.grad, b.grad, rtol=1e-5, atol=1e-5 * float(b.grad.abs().max()))


def test_partial_and_second_gradients(monkeypatch):
    torch.manual_seed(0)
    scores = torch.softmax(torch.randn(300, 8, device='cuda'), dim=1)
    got = []
    for leaf, p, l in _both(scores, monkeypatch, top_k=2):
        first, = torch.autograd.grad(p[3][1].square().sum(), leaf, create_graph=True)     # pick 0 and the loss get none
        second, = torch.autograd.grad(first.square().sum(), leaf)
        only_loss, = torch.autograd.grad(l, leaf)              # the gates' graph is gone, the loss has its own
        got.append((first.detach(), second, only_loss))
    for u, v in zip(*got):
        torch.testing.assert_close(u, v, rtol=1e-4, atol=1e-5 * float(v.abs().max()))


def test_unusual_scores(monkeypatch):
    """Scores that are no probabilities, NaN rows and infinities stay inside the experts' range."""
    from planmoe_b200.impls import fast_dispatch as FD
    scores = torch.randn(400, 6, device='cuda')
    scores[3] = float('nan')
    scores[4, 2] = float('nan')
    scores[5] = -float('inf')
    scores[6, 1] = float('inf')
    plan, _ = FD.extract_critical(scores, 3)
    idx = torch.stack(plan[1]).long()
    assert int(idx.min()) >= 0 and int(idx.max()) < 6
    assert all(len(set(r)) == 3 for r in idx.t().tolist())
    assert idx[0, 4] == 2 and idx[0, 6] == 1
    loc = torch.stack(plan[2])
    for e in range(6):
        assert sorted(loc[idx == e].tolist()) == list(range(int((idx == e).sum())))


def test_gates_of_unusual_scores(monkeypatch):
    """A NaN pick makes all gates of its token NaN, as the clamp of the composition does; infinities, negative and vanishing
    sums likewise agree, with their gradients."""
    scores = torch.rand(200, 6, generator=torch.Generator().manual_seed(4)).cuda()
    scores[1, 3] = float('nan')
    scores[2, 0], scores[2, 5] = float('nan'), float('inf')
    scores[3, 1] = float('inf')
    scores[4] = -scores[4]                                # sums below the clamp's bound
    scores[5] *= 1e-9
    scores[6, 2], scores[6, 4] = 3.0, -float('inf')
    weights = torch.rand(2, 200, device='cuda')
    got = []
    for leaf, p, _ in _both(scores, monkeypatch, top_k=2):
        grad, = torch.autograd.grad([p[3][0], p[3][1]], leaf, list(weights))
        got.append((torch.stack(p[1]), torch.stack([g.detach() for g in p[3]]), grad))
    (ia, ga, da), (ib, gb, db) = got
    assert torch.equal(ia, ib) and bool(ga[:, 1].isnan().all())
    torch.testing.assert_close(ga, gb, rtol=4e-7, atol=0, equal_nan=True)       # a sum of two scores and a division
    torch.testing.assert_close(da, db, rtol=1e-5, atol=1e-5, equal_nan=True)


def test_what_may_change_in_place_before_the_backward(monkeypatch):
    """As with the composition: the plan's lists may, the scores may for the loss, but not for the gates."""
    from planmoe_b200.impls import fast_dispatch as FD
    from planmoe_b200.jit_kernels import gating
    scores = torch.softmax(torch.randn(300, 8, device='cuda'), dim=1)
    weight = torch.rand(300, device='cuda')
    got = []
    for fast in (True, False):
        monkeypatch.setattr(gating, 'use_fast_cumsum', fast)
        leaf = scores.clone().requires_grad_()
        plan, loss = FD.extract_critical(leaf, 2)
        plan[1][0][::3] = -1                              # the caller drops some picks
        plan[2][1].add_(5)
        both, = torch.autograd.grad((plan[3][0] * weight).sum() + loss, leaf)
        held = leaf * 1
        plan, loss = FD.extract_critical(held, 2)
        held.mul_(3)
        alone, = torch.autograd.grad(loss, leaf, retain_graph=True)
        with pytest.raises(RuntimeError, match='inplace'):
            torch.autograd.grad(plan[3][0].sum(), leaf)
        got.append((both, alone))
    for u, v in zip(*got):
        torch.testing.assert_close(u, v, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize('cf', [1.0, 0.0])
def test_lists_changed_after_the_first_use_of_a_plan(cf, monkeypatch):
    """The slots of a plan are laid down by its first use: neither decode nor the gradients see later changes of the lists."""
    from planmoe_b200.impls import fast_dispatch as FD
    from planmoe_b200.jit_kernels import gating
    scores = torch.softmax(torch.randn(300, 8, device='cuda'), dim=1)
    x = torch.randn(300, 64, device='cuda')
    dy = torch.randn(300, 64, device='cuda')
    got = []
    for fast in (True, False):
        monkeypatch.setattr(gating, 'use_fast_cumsum', fast)
        leaf, xl = scores.clone().requires_grad_(), x.clone().requires_grad_()
        plan, _ = FD.extract_critical(leaf, 2, capacity_factor=cf)
        slots = FD.fast_encode(xl, plan)
        plan[1][0].add_(1).remainder_(8)
        plan[2][1].add_(3)
        y = FD.fast_decode(slots, plan)
        plan[2][0].add_(3)
        y.backward(dy)
        got.append((slots.detach(), y.detach(), xl.grad, leaf.grad))
    for u, v in zip(*got):
        torch.testing.assert_close(u, v, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float16])
@pytest.mark.parametrize('postscore', [True, False])
@pytest.mark.parametrize('before', [True, False])
def test_gates_changed_around_the_uses_of_a_plan(dtype, postscore, before, monkeypatch):
    """Encode and decode each take the gates as they are at the call, and keep them for their gradients."""
    from planmoe_b200.impls import fast_dispatch as FD
    from planmoe_b200.jit_kernels import gating
    scores = torch.softmax(torch.randn(300, 8, device='cuda'), dim=1)
    x = torch.randn(300, 64, device='cuda').to(dtype)
    dy = torch.randn(300, 64, device='cuda').to(dtype)
    got = []
    for fast in (True, False):
        monkeypatch.setattr(gating, 'use_fast_cumsum', fast)
        leaf, xl = scores.clone().requires_grad_(), x.clone().requires_grad_()
        plan, _ = FD.extract_critical(leaf, 2)
        if before:
            plan[3][1].mul_(0.5)
        slots = FD.fast_encode(xl, plan, postscore)
        y = FD.fast_decode(slots, plan, postscore)
        with torch.no_grad():
            plan[3][0].mul_(7.0)                          # the caller's own use of the list, afterwards
        y.backward(dy)
        got.append((slots.detach(), y.detach(), xl.grad, leaf.grad))
    eps = torch.finfo(dtype).eps
    for u, v in zip(*got):                                # the composition rounds the gates' gradient to the data's type
        assert float((u.float() - v.float()).abs().max()) <= 4 * eps * float(v.float().abs().max()) + 1e-6


def test_changed_lists_and_other_forms_take_the_composition(monkeypatch):
    from planmoe_b200.impls import fast_dispatch as FD, losses
    scores = torch.softmax(torch.randn(64, 4, device='cuda'), dim=1)
    plan, _ = FD.extract_critical(scores, 2)
    plan[2][1].add_(1)                                                # in place: the made slot map no longer fits
    ref = FD.RoutingPlan(plan[0], [x.clone() for x in plan[1]], [x.clone() for x in plan[2]], plan[3], plan[4])
    assert torch.equal(plan.slots.slot_map, ref.slots.slot_map)
    for kw in (dict(loss_fn=lambda s, i: losses.gshard_loss(s, i) * 2), dict(batch_prioritized_routing=True)):
        FD.extract_critical(scores, 2, **kw)
    FD.extract_critical(scores.half(), 2)
    from planmoe_b200.jit_kernels import gating
    monkeypatch.setattr(gating, 'use_fast_cumsum', False)             # the cumsum kernel knows no function transforms
    grad = torch.func.grad(lambda s: FD.extract_critical(s, 2)[1])(scores)
    assert torch.isfinite(grad).all()


@pytest.mark.parametrize('dtype', [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize('postscore', [True, False])
@pytest.mark.parametrize('S,E,k', [(1, 2, 2), (257, 5, 1), (300, 8, 3)])
def test_encode_and_decode_by_pick(dtype, postscore, S, E, k):
    """Gates handed over pick by pick (on one storage, and as tensors of their own) against the stacked, rounded ones."""
    from planmoe_b200.impls import fast_dispatch as FD
    from planmoe_b200.ops import dispatch as D
    torch.manual_seed(S)
    x = torch.randn(S, 64, device='cuda').to(dtype)
    dy = torch.randn(S, 64, device='cuda').to(dtype)
    scores = torch.softmax(torch.randn(S, E, device='cuda'), dim=1)
    out = []
    for form in ('made', 'separate', 'stacked'):
        xl, sl = x.clone().requires_grad_(), scores.clone().requires_grad_()
        plan, _ = FD.extract_critical(sl, k, capacity_factor=0.8)
        gates = [g * 1 for g in plan[3]] if form == 'separate' else plan[3]
        if form != 'made':
            plan = FD.RoutingPlan(plan[0], plan[1], plan[2], gates, plan[4], plan.slots)
        if form == 'stacked':
            g = plan.stacked_gates().to(dtype)
            slots = D.scatter(xl, plan.slots, None if postscore else g)
            y = D.gather(slots, plan.slots, g if postscore else None)
        else:
            y = FD.fast_decode(FD.fast_encode(xl, plan, postscore), plan, postscore)
        y.backward(dy)
        out.append((y.detach(), xl.grad, sl.grad))
    for got in out[:2]:
        assert torch.equal(got[0], out[2][0]) and torch.equal(got[1], out[2][1])
        # the stacked form rounds the gates' gradient to the data's type
        eps = torch.finfo(dtype).eps
        assert float((got[2] - out[2][2]).abs().max()) <= 4 * eps * float(out[2][2].abs().max()) + 1e-6


def _off(t, by=1):
    """The same values as a contiguous view that starts ``by`` elements into its storage."""
    room = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    view = room[by:].view(t.shape).copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16
    return view


@pytest.mark.parametrize('dtype', [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize('postscore', [True, False])
@pytest.mark.parametrize('gates32', [True, False])
def test_rows_off_the_vector_boundary(dtype, postscore, gates32):
    """Tokens, slots and gradients may start anywhere in their storage: the kernels get aligned copies."""
    from planmoe_b200.impls import fast_dispatch as FD
    torch.manual_seed(3)
    x = torch.randn(70, 64, device='cuda').to(dtype)
    dy = torch.randn(70, 64, device='cuda').to(dtype)
    scores = torch.softmax(torch.randn(70, 4, device='cuda'), dim=1)
    if not gates32:
        scores = scores.half()
    out = []
    for place in (lambda t: t, _off):
        xl, sl = place(x.clone()).requires_grad_(), scores.clone().requires_grad_()
        plan, _ = FD.extract_critical(sl, 2)
        slots = FD.fast_encode(xl, plan, postscore)
        held = place(slots.detach()).requires_grad_()
        y = FD.fast_decode(held, plan, postscore)
        y.backward(place(dy), retain_graph=True)
        slots.backward(place(held.grad))
        out.append((slots.detach(), y.detach(), held.grad, xl.grad, sl.grad))
    for u, v in zip(*out):
        assert torch.equal(u, v)


def test_kernels_refuse_rows_off_the_vector_boundary():
    """The bindings turn a misaligned base into an error on the host."""
    from planmoe_b200.ops import native
    lib = native.lib()
    x = _off(torch.randn(16, 64, device='cuda').bfloat16())
    good = x.clone()
    idx = torch.zeros(1, 16, dtype=torch.int32, device='cuda')
    loc = torch.arange(16, dtype=torch.int32, device='cuda').view(1, 16)
    smap = lib.build_slot_map(idx, loc, 1, 16)
    calls = [lambda: lib.dispatch_scatter(x, smap, None, 1, 16), lambda: lib.dispatch_gather(x, idx, loc, None, 16),
             lambda: lib.dispatch_gate_grad(x, good, idx, loc, 16), lambda: lib.dispatch_gate_grad(good, x, idx, loc, 16),
             lambda: lib.int8_encode(x), lambda: lib.int8_rows_encode(x), lambda: lib.colsum(x.view(1, 16, 64), 1, True),
             lambda: lib.int8_decode(_off(torch.zeros(16, 64, dtype=torch.uint8, device='cuda')), torch.ones(16, device='cuda'),
                                     torch.ones(16, device='cuda'), torch.bfloat16)]
    for call in calls:
        with pytest.raises(RuntimeError, match='aligned'):
            call()
    torch.cuda.synchronize()


@pytest.mark.parametrize('dtype,dim', [(torch.float32, 66), (torch.float32, 1), (torch.float16, 36), (torch.bfloat16, 7)])
@pytest.mark.parametrize('postscore', [True, False])
def test_rows_that_are_no_whole_vectors(dtype, dim, postscore):
    """Model dims whose rows the 16-byte kernels cannot move, against the same rows padded to whole vectors."""
    from planmoe_b200.impls import fast_dispatch as FD
    torch.manual_seed(dim)
    pad = torch.nn.functional.pad
    wide = (dim + 7) // 8 * 8
    x = torch.randn(70, dim, device='cuda').to(dtype)
    dy = torch.randn(70, dim, device='cuda').to(dtype)
    scores = torch.softmax(torch.randn(70, 4, device='cuda'), dim=1)
    out = []
    for padded in (False, True):
        xl = (pad(x, (0, wide - dim)) if padded else x.clone()).requires_grad_()
        sl = scores.clone().requires_grad_()
        plan, _ = FD.extract_critical(sl, 2, capacity_factor=0.8)
        slots = FD.fast_encode(xl, plan, postscore)
        y = FD.fast_decode(slots, plan, postscore)
        y.backward(pad(dy, (0, wide - dim)) if padded else dy)
        out.append((slots.detach()[..., :dim], y.detach()[..., :dim], xl.grad[..., :dim], sl.grad))
    for u, v in zip(out[0][:3], out[1][:3]):
        torch.testing.assert_close(u, v, rtol=2 * torch.finfo(dtype).eps, atol=1e-6)      # two products, added and rounded
    # the gates' gradient: `dim` products in another order, rounded to the data's type by the composite
    top = float(out[1][3].abs().max())
    assert float((out[0][3] - out[1][3]).abs().max()) <= (4 * torch.finfo(dtype).eps + 1e-5) * top
