"""The priority order at the edges of its sorted tiles of 1024 tokens, and below the sizes that are sorted."""

import pytest
import torch

from planmoe_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('S', [2, 8191, 8192, 9215, 9216, 9217, 12289])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
def test_order(S, dtype):
    logits = (torch.randn(S, 3, generator=torch.Generator().manual_seed(S)) * 2).round().cuda().to(dtype)    # few distinct keys
    logits[S // 2:S // 2 + 3] = float('nan')
    rank, perm = native.lib().importance_order(logits)
    assert torch.equal(rank[perm.long()].long(), torch.arange(S, device='cuda'))
    key = torch.softmax(logits.double(), 1).max(1).values.nan_to_num(0.0)
    along = key[perm.long()]
    assert bool((along[:-1] >= along[1:] - 1e-6).all())                            # best top score first, NaN last
    for row in logits[~logits.isnan().any(1)].unique(dim=0)[:5]:
        of = rank[(logits == row).all(1)]
        assert bool((of[1:] > of[:-1]).all())                                      # equal rows: token order
