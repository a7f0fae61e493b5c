"""What a user of this framework has it do, as timed cases: the MoE layer's training step and its inference forward, the
stand-alone routing + encode / decode pair, and the payload codecs, over the sizes that they are used at.

``listed()`` names the cases, ``draw()`` makes more of the same ranges, ``prepare()`` builds what a program holds before
the call, ``run()`` is one pass through the public entry points, ``exact()`` restates it in 64 bits with plain torch.
"""

import math

import torch
import torch.nn.functional as F

from planmoe_b200 import moe
from planmoe_b200.impls.fast_dispatch import extract_critical, fast_decode, fast_encode
from planmoe_b200.ops import native
from planmoe_b200.parallel import codecs

_DTYPES = {'bf16': torch.bfloat16, 'fp16': torch.float16, 'fp32': torch.float32}
_ACTS = {'gelu': F.gelu, 'relu': F.relu, 'silu': F.silu}
_AUX = 0.01            # weight of the balance loss in the training step
_CODEC_SLICES = 8      # destination ranks a codec's tensor is split over


def _layer_case(name, mode, tokens, dim, hidden, experts, top_k, cf, act, dtype='bf16', wire='no', fp32_gate=True, prio=False):
    return dict(name=name, kind='layer', mode=mode, tokens=tokens, dim=dim, hidden=hidden, experts=experts, top_k=top_k,
                cf=cf, act=act, dtype=dtype, wire=wire, fp32_gate=fp32_gate, prio=prio)


def listed():
    return [
        # the benchmark's layer: 16 x 512 tokens a rank, two experts a GPU, every token goes to both
        _layer_case('train_8k_tokens_2_experts', 'train', 8192, 2048, 2048, 2, 2, 1.0, 'gelu', fp32_gate=False),
        # the MoE block of the GPT model at its default sizes, eight sequences of 1024 tokens on one GPU
        _layer_case('train_gpt_block', 'train', 8192, 1024, 4096, 8, 2, 1.25, 'gelu'),
        # the benchmark's layer with int8 rows on the wire
        _layer_case('train_int8_wire', 'train', 8192, 2048, 2048, 2, 2, 1.0, 'gelu', wire='int8', fp32_gate=False),
        # a batch of uneven sequences, one pick a token, capacity sized to the busiest expert (as in the fairseq integration)
        _layer_case('train_ragged_top1_dynamic', 'train', 3001, 768, 3072, 5, 1, 0.0, 'relu'),
        # a large model's layer: the arithmetic of the experts is nearly all of the step
        _layer_case('train_16k_tokens_wide', 'train', 16384, 4096, 4096, 8, 2, 1.0, 'silu'),
        # a small layer, as in tests and first experiments: launches and host work count
        _layer_case('train_small', 'train', 256, 256, 512, 4, 2, 1.0, 'relu'),
        # the 32-bit layer of the CPU check (4 x 128 tokens), on the GPU: routing, encode and decode outside the fused path
        _layer_case('train_fp32', 'train', 512, 256, 512, 8, 2, 1.0, 'relu', dtype='fp32'),
        # a decoding step: a handful of tokens meet every expert's weights
        _layer_case('infer_16_tokens', 'infer', 16, 1024, 4096, 8, 2, 2.0, 'gelu'),
        # prefill / evaluation of a long batch, best-scored tokens claim their slots first
        _layer_case('infer_16k_tokens_prio', 'infer', 16384, 2048, 2048, 16, 2, 1.25, 'gelu', prio=True),
        # routing, encode and decode around a user's own experts, forward and backward
        dict(name='dispatch_fp16', kind='dispatch', tokens=8192, dim=2048, experts=16, top_k=2, cf=1.0, dtype='fp16'),
        # codecs on expert activations (about half of the values are zeros): pack and unpack
        dict(name='codec_zfp', kind='codec', codec='zfp', rows=8192, cols=4096, dtype='bf16'),
        dict(name='codec_lz', kind='codec', codec='lz', rows=8192, cols=4096, dtype='bf16'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['train', 'train', 'train', 'infer', 'infer', 'fp32', 'dispatch', 'codec'])
    if kind in ('train', 'infer'):
        lo = 16 if kind == 'infer' else 64
        tokens = _log_int(rng, lo, 16384)
        dim, hidden = 64 * _log_int(rng, 4, 64), 64 * _log_int(rng, 4, 64)
        experts = rng.choice([1, 2, 3, 4, 5, 8, 8, 12, 16, 32])
        while experts > 1 and experts * dim * hidden > 8 * 4096 * 4096:
            experts //= 2
        top_k = min(experts, rng.choice([1, 2, 2, 2, 4]))
        while top_k > 1 and tokens * top_k * dim * hidden > 16384 * 2 * 4096 * 4096:
            top_k -= 1
        cf = rng.choice([1.0, 1.0, 1.25, 2.0, 0.0])
        wire = 'int8' if kind == 'train' and dim % 128 == 0 and rng.random() < 0.15 else 'no'
        case = _layer_case(None, kind, tokens, dim, hidden, experts, top_k, cf, rng.choice(['gelu', 'relu', 'silu']),
                           wire=wire, fp32_gate=not (top_k == experts and cf >= 1.0 and rng.random() < 0.5),
                           prio=rng.random() < 0.15)
        del case['name']
        return case
    if kind == 'fp32':
        case = _layer_case(None, 'train', _log_int(rng, 64, 4096), 2 * _log_int(rng, 32, 512), _log_int(rng, 64, 1024),
                           rng.choice([2, 4, 7, 8, 16]), rng.choice([1, 2, 2]), rng.choice([1.0, 1.25]),
                           rng.choice(['gelu', 'relu']), dtype='fp32')
        del case['name']
        return case
    if kind == 'dispatch':
        return dict(kind='dispatch', tokens=_log_int(rng, 128, 16384), dim=8 * _log_int(rng, 16, 512),
                    experts=rng.choice([2, 4, 8, 16, 24, 64]), top_k=rng.choice([1, 2, 2]), cf=rng.choice([1.0, 1.25, 2.0]),
                    dtype=rng.choice(['bf16', 'fp16', 'fp32']))
    return dict(kind='codec', codec=rng.choice(['int8', 'zfp', 'lz']), rows=_CODEC_SLICES * _log_int(rng, 16, 1024),
                cols=16 * _log_int(rng, 8, 256), dtype=rng.choice(['bf16', 'bf16', 'fp16', 'fp32']))


def _capacity(case):
    """Slots an expert has, before alignment (dynamic capacity: what an even split needs)."""
    per_expert = -(-case['tokens'] // case['experts'])
    return case['top_k'] * int((case['cf'] or 1.0) * per_expert)


def prepare(case, seed):
    dev = torch.device('cuda')
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    dtype = _DTYPES[case['dtype']]

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    if case['kind'] == 'codec':
        x = torch.relu(normal(case['rows'], case['cols'])).to(dtype)
        return dict(kind='codec', x=x.view(_CODEC_SLICES, -1, case['cols']), codec=codecs.get_compressor(case['codec']),
                    name=case['codec'])
    x = normal(case['tokens'], case['dim']).to(dtype)
    dy = normal(case['tokens'], case['dim']).to(dtype)
    if case['kind'] == 'dispatch':
        logits = normal(case['tokens'], case['experts'])
        return dict(kind='dispatch', x=x.requires_grad_(), logits=logits.requires_grad_(), dy=dy, top_k=case['top_k'],
                    cf=case['cf'])
    with torch.device(dev):
        layer = moe.moe_layer(
            gate_type={'type': 'top', 'k': case['top_k'], 'capacity_factor': case['cf'], 'fp32_gate': case['fp32_gate']},
            model_dim=case['dim'],
            experts={'type': 'ffn', 'count_per_node': case['experts'], 'hidden_size_per_expert': case['hidden'],
                     'activation_fn': case['act']},
            seeds=(int(seed), int(seed) + 1, int(seed) + 2), compress_name=case['wire'],
            batch_prioritized_routing=case['prio'])
    layer = layer.to(dev).to(dtype)
    if case['fp32_gate']:
        layer.gates.float()
    train = case['mode'] == 'train'
    layer.train(train)
    return dict(kind='layer', layer=layer, x=x.requires_grad_(train), dy=dy, train=train)


def run(state):
    if state['kind'] == 'codec':
        packed = state['codec'].compress(state['x'], _CODEC_SLICES)
        out = state['codec'].decompress(packed)
        if state['name'] == 'lz':       # the slices' headers; what lies behind a slice's last code byte is not part of it
            _cap, _at, header = native.lib().lz_layout(state['x'][0].numel() * state['x'].element_size())
            return packed.wires[0][:, :header], out
        return tuple(packed.wires) + (out,)
    x, dy = state['x'], state['dy']
    x.grad = None
    if state['kind'] == 'dispatch':
        logits = state['logits']
        logits.grad = None
        crit, l_aux = extract_critical(F.softmax(logits, dim=1), state['top_k'], capacity_factor=state['cf'])
        slots = fast_encode(x, crit)
        y = fast_decode(slots, crit)
        torch.autograd.backward([y, l_aux], [dy, torch.full_like(l_aux, _AUX)])
        return slots.detach(), y.detach(), l_aux.detach(), x.grad, logits.grad
    layer = state['layer']
    if not state['train']:
        with torch.no_grad():
            return layer(x)
    layer.zero_grad(set_to_none=True)
    y = layer(x)
    l_aux = y.l_aux
    torch.autograd.backward([y, l_aux], [dy, torch.full_like(l_aux, _AUX)])
    ex = layer.experts
    return (y.detach(), l_aux.detach(), x.grad, layer.gates[0].wg.weight.grad, ex.batched_fc1_w.grad, ex.batched_fc1_bias.grad,
            ex.batched_fc2_w.grad, ex.batched_fc2_bias.grad)


def work(case):
    item = 4 if case['dtype'] == 'fp32' else 2
    if case['kind'] == 'codec':
        raw = case['rows'] * case['cols'] * item
        # the tensor in, its packed form out and in again (8 bits a value; lz: about what zeros compress to), the tensor out
        wire = raw * 0.75 if case['codec'] == 'lz' else case['rows'] * case['cols']
        return dict(bytes=2 * raw + 2 * wire, flops=0)
    tokens, dim, experts = case['tokens'], case['dim'], case['experts']
    rows = min(tokens * case['top_k'], experts * _capacity(case))
    if case['kind'] == 'dispatch':
        slots = experts * _capacity(case)
        # x, dy in; slots, y, dx out; logits in, their gradient out; the picked rows again for the gates' gradients
        return dict(bytes=(4 * tokens * dim + slots * dim + rows * dim) * item + 8 * tokens * experts, flops=0)
    weights = experts * 2 * dim * case['hidden'] * item
    gemm = 2.0 * 2.0 * rows * dim * case['hidden']
    if case['mode'] == 'infer':
        used = min(1.0, rows / experts)
        return dict(bytes=2 * tokens * dim * item + used * weights, flops=gemm)
    return dict(bytes=4 * tokens * dim * item + 3 * weights, flops=3 * gemm)


def tolerance(case):
    if case['kind'] == 'codec':
        # bytes and what they decode to; int8 may round a tie the other way
        return {'rel': 4e-3, 'differ': 1e-4} if case['codec'] == 'int8' else 'exact'
    if case['kind'] == 'dispatch':
        return {'rel': 1e-5 if case['dtype'] == 'fp32' else 2e-3 if case['dtype'] == 'fp16' else 1.5e-2}
    if case['dtype'] == 'fp32':
        return {'rel': 1e-5}
    return {'rel': 3e-2 if case['wire'] == 'int8' else 1.5e-2, 'max': 0.3}


# ------------------------------------------------------------------------------------ the same in 64 bits
def _route64(logits, top_k, cf, alignment, prio=False):
    """(picked experts [S, k], slot of each pick, kept, normalised gates, capacity, balance loss)"""
    S, E = logits.shape
    scores = F.softmax(logits, dim=1)
    picks = torch.topk(scores.detach(), min(top_k, E), dim=1).indices
    order = torch.argsort(-scores.detach().max(dim=1).values, stable=True) if prio else torch.arange(S, device=logits.device)
    slot, base = torch.empty_like(picks), 0
    for k in range(picks.size(1)):
        hot = F.one_hot(picks[order, k], E)
        at = hot.cumsum(0) - 1 + base
        slot[order, k] = at.gather(1, picks[order, k:k + 1]).view(-1)
        base = base + hot.sum(0, keepdim=True)
    gates = scores.gather(1, picks)
    if picks.size(1) > 1:
        gates = gates / gates.sum(1, keepdim=True)
    cap = picks.size(1) * int(cf * -(-S // E)) if cf > 0 else int(slot.max()) + 1
    cap = max(cap, 1)
    cap += -cap % alignment
    frac = F.one_hot(picks[:, 0], E).to(scores.dtype).sum(0)
    l_aux = (scores.sum(0) * frac).sum() * E / (S * S)
    return picks, slot, slot < cap, gates, cap, l_aux


def exact(case, seed):
    if case['kind'] == 'codec':
        state = prepare(case, seed)
        x = state['x'].double()
        if case['codec'] == 'lz':
            return None, x
        if case['codec'] == 'zfp':
            return None
        lo, hi = x.amin(-1, keepdim=True), x.amax(-1, keepdim=True)
        return None, (hi - lo).squeeze(-1), lo.squeeze(-1), None
    state = prepare(case, seed)
    x = state['x'].detach().double().requires_grad_()
    dy = state['dy'].double()
    if case['kind'] == 'dispatch':
        logits = state['logits'].detach().double().requires_grad_()
        picks, slot, kept, gates, cap, l_aux = _route64(logits, case['top_k'], case['cf'], 1)
        slots = x.new_zeros(case['experts'] * cap, case['dim'])
        y = torch.zeros_like(x)
        for k in range(picks.size(1)):
            at = (picks[:, k] * cap + slot[:, k])[kept[:, k]]
            slots = slots.index_add(0, at, x[kept[:, k]])
        for k in range(picks.size(1)):
            at = (picks[:, k] * cap + slot[:, k])[kept[:, k]]
            rows = torch.nonzero(kept[:, k]).view(-1)
            y = y.index_add(0, rows, slots[at] * gates[rows, k:k + 1])
        gx, gl = torch.autograd.grad([y, l_aux], [x, logits], [dy, torch.full_like(l_aux, _AUX)])
        return slots.detach().view(case['experts'], cap, -1), y.detach(), l_aux.detach(), gx, gl
    layer, ex = state['layer'], state['layer'].experts
    names = [layer.gates[0].wg.weight, ex.batched_fc1_w, ex.batched_fc1_bias, ex.batched_fc2_w, ex.batched_fc2_bias]
    wg, w1, b1, w2, b2 = params = [p.detach().double().requires_grad_(state['train']) for p in names]
    del layer, ex, names, state
    with torch.set_grad_enabled(case['mode'] == 'train'):
        picks, slot, kept, gates, cap, l_aux = _route64(x @ wg.t(), case['top_k'], case['cf'], 4, case['prio'])
        y = torch.zeros_like(x)
        for e in range(case['experts']):
            t, k = torch.nonzero((picks == e) & kept, as_tuple=True)
            h = _ACTS[case['act']](x[t] @ w1[e] + b1[e])
            y = y.index_add(0, t, (h @ w2[e] + b2[e]) * gates[t, k].unsqueeze(1))
    if case['mode'] == 'infer':
        return y
    gx, *gp = torch.autograd.grad([y, l_aux], [x] + params, [dy, torch.full_like(l_aux, _AUX)])
    return (y.detach(), l_aux.detach(), gx) + tuple(gp)
