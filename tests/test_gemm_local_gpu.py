"""The grouped GEMM of local operands: every epilogue and operand layout, at edges of its tiles."""

import pytest
import torch

from planmoe_b200.ops.gemm import ACT_CODES, EPI_BIAS_ACT, EPI_DACT, EPI_STORE, check_status, grouped_gemm

pytestmark = pytest.mark.gpu


def _rand(*shape, seed):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    return torch.randn(*shape, generator=gen, device='cuda').bfloat16()


def _close(got, want, k):
    # both round an fp32 sum of k products once: half a bf16 step of the value, and the sums' own rounding
    err = (got.double() - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -8 + 1e-5 * k ** 0.5 + 1e-30).all()), float(err.max())


# odd and even numbers of 256-row blocks, ragged rows, columns and contractions, fewer and more tiles than clusters, contractions
# shorter than, as long as and longer than the ring
SHAPES = [(1, 264, 64, 256), (3, 136, 448, 256), (2, 512, 8, 8), (3, 520, 72, 264), (1, 1024, 128, 512), (2, 776, 200, 1032), (5, 768, 320, 768),
          (9, 1288, 448, 520), (2, 4096, 264, 2048), (33, 264, 136, 72), (64, 512, 64, 256)]


@pytest.mark.parametrize('G,M,K,N', SHAPES)
@pytest.mark.parametrize('layout', ['fwd', 'dgrad', 'wgrad'])
def test_store(G, M, K, N, layout):
    if layout == 'wgrad':
        a, b = _rand(G, K, M, seed=1), _rand(G, K, N, seed=2)
        want = a.double().transpose(1, 2) @ b.double()
        got = grouped_gemm(a, True, b, True, EPI_STORE)
    elif layout == 'dgrad':
        a, b = _rand(G, M, K, seed=1), _rand(G, N, K, seed=2)
        want = a.double() @ b.double().transpose(1, 2)
        got = grouped_gemm(a, False, b, False, EPI_STORE)
    else:
        a, b, bias = _rand(G, M, K, seed=1), _rand(G, K, N, seed=2), _rand(G, N, seed=3)
        want = a.double() @ b.double() + bias.double().unsqueeze(1)
        got = grouped_gemm(a, False, b, True, EPI_STORE, bias=bias)
    check_status()
    _close(got, want, K)


@pytest.mark.parametrize('G,M,K,N', SHAPES)
@pytest.mark.parametrize('act', ['relu', 'gelu', 'silu', 'identity'])
def test_activation_and_its_backward(G, M, K, N, act):
    a, b, bias = _rand(G, M, K, seed=1), _rand(G, K, N, seed=2), _rand(G, N, seed=3)
    t = (a.double() @ b.double() + bias.double().unsqueeze(1)).requires_grad_()
    f = {'relu': torch.relu, 'gelu': torch.nn.functional.gelu, 'silu': torch.nn.functional.silu, 'identity': lambda x: x * 1}[act]
    want = f(t)
    deriv, = torch.autograd.grad(want.sum(), t)
    aux = torch.empty(G, M, N, dtype=torch.bfloat16, device='cuda')
    got = grouped_gemm(a, False, b, True, EPI_BIAS_ACT, ACT_CODES[act], bias=bias, aux=aux)
    alone = grouped_gemm(a, False, b, True, EPI_BIAS_ACT, ACT_CODES[act], bias=bias)
    check_status()
    away = t.detach().abs() > 1e-3                       # ReLU's derivative jumps where the sum's rounding decides
    _close(got, want.detach(), 4 * K)
    _close(torch.where(away, aux.double(), deriv), deriv, 4 * K)
    assert torch.equal(alone, got)
    # dH = (dY . W^T) * derivative, with its column sums
    dy, w = _rand(G, M, K, seed=4), _rand(G, N, K, seed=5)
    sums = torch.full((G, (M + 31) // 32, N), float('nan'), device='cuda')
    dh = grouped_gemm(dy, False, w, False, EPI_DACT, aux=aux, colsum=sums)
    check_status()
    _close(dh, (dy.double() @ w.double().transpose(1, 2)) * aux.double(), 4 * K)
    pad = torch.nn.functional.pad(dh.double(), (0, 0, 0, -M % 32)).view(G, -1, 32, N).sum(2)
    assert torch.allclose(sums.double(), pad, rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize('G,M,K,N', [(5, 1030, 72, 264), (8, 2560, 128, 1024), (64, 776, 64, 256)])
def test_used_rows(G, M, K, N):
    gen = torch.Generator().manual_seed(G)
    used = torch.randint(0, M + 1, (G,), generator=gen)
    used[:4] = torch.tensor([0, M, 256, 513])[:len(used[:4])]
    u = used.to('cuda', torch.int32)
    live = (torch.arange(M, device='cuda').unsqueeze(0) < u.unsqueeze(1)).unsqueeze(2)
    a, b = _rand(G, M, K, seed=1) * live, _rand(G, K, N, seed=2)
    out = torch.full((G, M, N), 7.0, dtype=torch.bfloat16, device='cuda')
    grouped_gemm(a, False, b, True, EPI_STORE, out=out, rows_used=u)
    end = ((used.clamp(min=1) + 255) // 256 * 256).clamp(max=M).cuda()
    inside = (torch.arange(M, device='cuda').unsqueeze(0) < end.unsqueeze(1)).unsqueeze(2)
    assert bool((torch.where(inside, torch.tensor(7.0, device='cuda').bfloat16(), out) == 7.0).all())   # behind: untouched
    _close(torch.where(inside, out, torch.zeros_like(out)), a.double() @ b.double(), K)
    d = _rand(G, M, N, seed=3) * live
    dw = grouped_gemm(a, True, d, True, EPI_STORE, rows_used=u)
    check_status()
    _close(dw, a.double().transpose(1, 2) @ d.double(), M)
