"""A process that goes on with another GPU: limits of dynamic shared memory are told to each device."""

import os
import re

import pytest
import torch

import planmoe_b200
from planmoe_b200 import moe

KERNELS = os.path.join(os.path.dirname(planmoe_b200.__file__), 'csrc', 'kernels')
NGPU = torch.cuda.device_count() if torch.cuda.is_available() else 0


def test_no_launch_tells_the_process():
    """Only the helper, which knows the device, and the occupancy query for the first device set the limit."""
    found = []
    for name in sorted(os.listdir(KERNELS)):
        text = re.sub(r'//.*', '', open(os.path.join(KERNELS, name)).read()) if name.endswith(('.cu', '.cuh')) else ''
        for m in re.finditer(r'cudaFuncSetAttribute', text):
            heads = re.findall(r'^(?:\w[\w:<>*& ]*?)(\w+)\(', text[:m.start()], re.M)
            found.append((name, heads[-1]))
    assert sorted(found) == [('gemm_tcgen05.cu', 'max_pair_units'), ('launch.cuh', 'allow_smem')]


@pytest.mark.gpu
@pytest.mark.multigpu
@pytest.mark.skipif(NGPU < 2, reason="needs 2 GPUs")
@pytest.mark.parametrize('tokens', [16, 600])
def test_layers_on_two_devices(tokens):
    def run(device):
        torch.manual_seed(0)
        layer = moe.moe_layer(gate_type={'type': 'top', 'k': 2}, model_dim=128,
                              experts={'type': 'ffn', 'count_per_node': 4, 'hidden_size_per_expert': 256, 'activation_fn': 'gelu'})
        layer = layer.to(device).bfloat16()
        x = torch.randn(tokens, 128).to(device).bfloat16().requires_grad_()
        with torch.cuda.device(device):
            y = layer(x)
            (y.float().square().sum() + y.l_aux).backward()
        return [t.detach().cpu() for t in (y, x.grad, layer.experts.batched_fc1_w.grad)]
    for a, b in zip(run('cuda:0'), run('cuda:1')):
        assert torch.equal(a, b)
