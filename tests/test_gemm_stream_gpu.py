"""The grouped GEMM for a handful of rows: edges of its tiles, groups without a token."""

import pytest
import torch

from planmoe_b200.ops.gemm import ACT_CODES, EPI_BIAS_ACT, EPI_STORE, check_status, grouped_gemm
from test_gemm_local_gpu import _close, _rand

pytestmark = pytest.mark.gpu

# contractions of one K block, of fewer blocks than the ring has stages, ragged, of many rounds of the ring; ragged columns; the most
# rows and tiles that it takes, and one more of either
SHAPES = [(1, 1, 8, 8), (2, 8, 64, 256), (3, 31, 520, 264), (4, 32, 1024, 3000), (8, 8, 4096, 1024), (4, 32, 72, 1032), (1, 32, 2056, 12288),
          (4, 33, 72, 1032), (1, 16, 256, 12800), (64, 16, 256, 2048)]


@pytest.mark.parametrize('G,M,K,N', SHAPES)
@pytest.mark.parametrize('act', ['relu', 'gelu', 'silu', 'identity'])
def test_rows(G, M, K, N, act):
    a, b, bias = _rand(G, M, K, seed=1), _rand(G, K, N, seed=2), _rand(G, N, seed=3)
    t = (a.double() @ b.double() + bias.double().unsqueeze(1)).requires_grad_()
    f = {'relu': torch.relu, 'gelu': torch.nn.functional.gelu, 'silu': torch.nn.functional.silu, 'identity': lambda x: x * 1}[act]
    want = f(t)
    deriv, = torch.autograd.grad(want.sum(), t)
    _close(grouped_gemm(a, False, b, True, EPI_STORE, bias=bias), t.detach(), K)
    _close(grouped_gemm(a, False, b, True, EPI_STORE), t.detach() - bias.double().unsqueeze(1), K)
    aux = torch.full((G, M, N), float('nan'), dtype=torch.bfloat16, device='cuda')
    got = grouped_gemm(a, False, b, True, EPI_BIAS_ACT, ACT_CODES[act], bias=bias, aux=aux)
    assert torch.equal(got, grouped_gemm(a, False, b, True, EPI_BIAS_ACT, ACT_CODES[act], bias=bias))
    check_status()
    _close(got, want.detach(), 4 * K)
    away = t.detach().abs() > 1e-3                       # ReLU's derivative jumps where the sum's rounding decides
    _close(torch.where(away, aux.double(), deriv), deriv, 4 * K)


@pytest.mark.parametrize('M', [7, 32])
def test_groups_without_a_token_read_no_weights(M):
    G, K, N = 6, 1032, 776
    used = torch.tensor([0, M, 1, 0, M // 2, 0])
    live = (torch.arange(M).unsqueeze(0) < used.unsqueeze(1)).unsqueeze(2).cuda()
    a, b, bias = _rand(G, M, K, seed=1) * live, _rand(G, K, N, seed=2), _rand(G, N, seed=3)
    b[used.cuda() == 0] = float('nan')
    got = grouped_gemm(a, False, b, True, EPI_STORE, bias=bias, rows_used=used.to('cuda', torch.int32))
    check_status()
    want = a.double() @ b.double().nan_to_num() + bias.double().unsqueeze(1)
    _close(got, want, K)


@pytest.mark.parametrize('G,M,K,N', SHAPES)
@pytest.mark.parametrize('act', ['gelu', 'identity'])
def test_bits_of_the_kernel_for_up_to_128_rows(G, M, K, N, act):
    """Every output adds its products up in the order of the kernel for up to 128 rows."""
    a, b, bias = _rand(G, M, K, seed=1), _rand(G, K, N, seed=2), _rand(G, N, seed=3)

    def run(**how):
        aux = torch.full((G, M, N), float('nan'), dtype=torch.bfloat16, device='cuda')
        return grouped_gemm(a, False, b, True, EPI_BIAS_ACT, ACT_CODES[act], bias=bias, aux=aux, **how), aux
    got, want = run(), run(cta_group=1)
    check_status()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
