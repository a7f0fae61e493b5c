"""Codec kernels at the edges of their forms: bases that rule the vector moves out, ragged last rows, blocks that end the
bit budget early or late.  The oracle is the serial CPU coder; streams are compared byte for byte."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _lib():
    from planmoe_b200.ops import native
    return native.lib()


def _values(kind, n, gen):
    x = torch.randn(n, generator=gen)
    if kind == 'relu':
        return torch.relu(x)
    if kind == 'sparse':                        # mostly empty blocks; planes run out before the bits do
        return torch.where(torch.rand(n, generator=gen) < 0.04, x, torch.zeros(()))
    if kind == 'wide':                          # exponents 60 apart inside a block
        return x * torch.exp2(torch.randint(-30, 30, (n,), generator=gen).float())
    if kind == 'tiny':
        return x * 1e-38
    x[::97] = float('inf')                      # blocks with a non-finite value are stored as zeros
    return x


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize('offset', [0, 1, 2, 4])
@pytest.mark.parametrize('kind', ['relu', 'sparse', 'wide', 'tiny', 'inf'])
def test_zfp_forms_match_the_serial_coder(dtype, offset, kind):
    lib = _lib()
    gen = torch.Generator().manual_seed(7)
    lead, rows, cols = 3, 37, 132                # 1 row in the last block row, a partial thread block
    n = lead * rows * cols
    x = _values(kind, n + offset, gen).to(dtype)
    x_cpu = x[offset:].view(lead, rows, cols)    # a contiguous view whose base is `offset` elements into its storage
    x_gpu = x.cuda()[offset:].view(lead, rows, cols)
    assert x_gpu.is_contiguous() and x_gpu.data_ptr() % 16 == (offset * x.element_size()) % 16
    for rate in (4, 8, 16):
        s_cpu, s_gpu = lib.zfp_encode(x_cpu.clone(), rate), lib.zfp_encode(x_gpu, rate)
        assert torch.equal(s_gpu.cpu(), s_cpu)
        y_cpu = lib.zfp_decode(s_cpu, lead, rows, cols, rate, dtype)
        y_gpu = lib.zfp_decode(s_gpu, lead, rows, cols, rate, dtype)
        assert torch.equal(y_gpu.cpu(), y_cpu)
        shifted = torch.empty(s_gpu.numel() + 4, dtype=torch.uint8, device='cuda')[4:].view_as(s_gpu).copy_(s_gpu)
        assert torch.equal(lib.zfp_decode(shifted, lead, rows, cols, rate, dtype), y_gpu)
