"""int8 rows out of the local GEMM: unused capacity is neither computed nor read, and what is used is what a full pass gives."""

import pytest
import torch

from planmoe_b200 import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('S,E,K,cf,M,H', [(1000, 5, 2, 4.0, 256, 384), (65, 3, 1, 2.0, 128, 128), (2048, 2, 2, 1.0, 384, 256), (33, 16, 2, 1.0, 128, 192)])
def test_capacity_does_not_change_what_is_kept(S, E, K, cf, M, H):
    torch.manual_seed(0)
    with torch.device('cuda'):
        layer = moe.moe_layer(gate_type={'type': 'top', 'k': K, 'capacity_factor': cf, 'fp32_gate': True}, model_dim=M,
                              experts={'type': 'ffn', 'count_per_node': E, 'hidden_size_per_expert': H, 'activation_fn': 'gelu'}, compress_name='int8')
    layer = layer.cuda().bfloat16()
    layer.gates.float()
    x, dy = torch.randn(S, M, device='cuda').bfloat16(), torch.randn(S, M, device='cuda').bfloat16()

    def run(factor):
        xin = x.clone().requires_grad_()
        layer.zero_grad(set_to_none=True)
        y = layer(xin, capacity_factor=factor)
        y.backward(dy)
        return [y.detach(), xin.grad] + [p.grad for p in layer.experts.parameters()]
    if cf > 1.0:                                         # nothing is dropped at either capacity: the same rows, to the bit
        for a, b in zip(run(cf), run(2 * cf)):
            assert torch.equal(a, b)
    layer.compress_name = 'no'
    want = run(cf)
    layer.compress_name = 'int8'
    for a, b in zip(run(cf), want):                      # 255 steps of a row's range, twice: a few per cent of its norm
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 0.05
