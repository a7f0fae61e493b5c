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


@pytest.mark.parametrize('sym', [2, 4])
@pytest.mark.parametrize('nbytes', [16, 48, 2032, 2048, 2064, 6160, 40960])
@pytest.mark.parametrize('kind', ['zeros', 'period', 'few', 'relu', 'random', 'runs'])
def test_lz_forms_match_the_serial_coder(sym, nbytes, kind):
    """Tail blocks of every raggedness, matches of the greatest length and distance, codes that start on any byte."""
    lib = _lib()
    gen = torch.Generator().manual_seed(3)
    slices, n = 3, nbytes // sym
    if kind == 'zeros':
        v = torch.zeros(slices, n, dtype=torch.int32)
    elif kind == 'period':                       # matches reach back exactly 32 symbols, and 33 (too far)
        v = torch.stack([torch.arange(n) % p for p in (32, 33, 31)]).int()
    elif kind == 'few':
        v = torch.randint(0, 3, (slices, n), generator=gen).int()
    elif kind == 'relu':
        x = torch.relu(torch.randn(slices, n, generator=gen))
        v = x.view(torch.int32) if sym == 4 else x.bfloat16().view(torch.int16).int()
    elif kind == 'random':
        v = torch.randint(-2 ** 31, 2 ** 31 - 1, (slices, n), generator=gen, dtype=torch.int64).int()
    else:                                        # runs of uneven length, some longer than a match can be
        v = torch.repeat_interleave(torch.arange(slices * n), torch.randint(1, 90, (slices * n,), generator=gen))
        v = v[:slices * n].view(slices, n).int()
    raw = (v if sym == 4 else v.to(torch.int16)).contiguous().view(torch.uint8).view(slices, -1)
    p_cpu, n_cpu = lib.lz_encode(raw, sym)
    p_gpu, n_gpu = lib.lz_encode(raw.cuda(), sym)
    assert torch.equal(n_gpu.cpu(), n_cpu)
    for s in range(slices):
        used = int(n_cpu[s])
        assert torch.equal(p_gpu[s, :used].cpu(), p_cpu[s, :used])
    assert torch.equal(lib.lz_decode(p_gpu, n_gpu, raw.size(1), sym).cpu(), raw)
    assert torch.equal(lib.lz_decode(p_cpu.cuda(), n_cpu.cuda(), raw.size(1), sym).cpu(), raw)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize('name', ['int8', 'zfp', 'lz'])
def test_codecs_take_tensors_off_the_vector_boundary(name, dtype):
    from planmoe_b200.parallel import codecs
    codec = codecs.get_compressor(name)
    x = torch.relu(torch.randn(4 * 24 * 64 + 1, device='cuda')).to(dtype)
    off = x[1:].view(4, 24, 64)
    assert off.is_contiguous() and off.data_ptr() % 16
    a, b = codec.compress(off, 4), codec.compress(off.clone(), 4)
    assert torch.equal(codec.decompress(a), codec.decompress(b))
    if name != 'lz':                             # behind a slice's code an lz wire holds anything
        for u, v in zip(a.wires, b.wires):
            assert torch.equal(u, v)
    if name == 'int8':                           # so may the wire
        room = torch.empty(a.wires[0].numel() + 1, dtype=torch.uint8, device='cuda')
        moved = codecs.Packed([room[1:].view_as(a.wires[0]).copy_(a.wires[0])] + a.wires[1:], a.meta)
        assert torch.equal(codec.decompress(moved), codec.decompress(b))


@pytest.mark.parametrize('device', ['cpu', 'cuda'])
@pytest.mark.parametrize('damage', ['far', 'long', 'backwards'])
def test_lz_blocks_with_a_damaged_header_are_left_alone(device, damage):
    """Offsets that point outside the slice, or enclose no code, are not followed; the other blocks decode."""
    lib = _lib()
    raw = torch.randint(0, 3, (2, 4 * 2048), generator=torch.Generator().manual_seed(1)).to(torch.uint8).to(device)
    payload, sizes = lib.lz_encode(raw, 2)
    head = payload.view(torch.int32)[1]          # {blocks, offset of block 0, 1, 2, 3, end}
    good = {'far': [0, 1], 'long': [0, 1, 2], 'backwards': [0, 2, 3]}[damage]
    if damage == 'far':                          # block 2 and what follows it
        head[4] = head[5] = 0x7ffffff0
    elif damage == 'long':
        head[5] = head[5] + 100000
    else:                                        # block 1 would end before it begins, block 2 starts where it did
        head[2] = head[3] + 4
    out = lib.lz_decode(payload, sizes, raw.size(1), 2)
    assert torch.equal(out[0], raw[0])
    for b in good:
        if damage == 'backwards' and b == 0:
            continue                             # its code now runs into block 1's
        assert torch.equal(out[1, b * 2048:(b + 1) * 2048], raw[1, b * 2048:(b + 1) * 2048])
    with pytest.raises(RuntimeError, match='header'):
        lib.lz_decode(payload[:, :16].contiguous(), sizes, raw.size(1), 2)
