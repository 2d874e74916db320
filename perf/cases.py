"""Performance cases of the block-sparse operations, measured through the package's public classes.

A case describes one call that a training or inference program makes over and over with a layout it
keeps: SparseSelfAttention and MultiheadAttention, the MatMul -> Softmax -> MatMul chain that the
attention replaces, Softmax and MatMul on their own, and the block-sparse Linear layer.  listed()
names twelve of them, draw() gives more of the same families over the whole range of sizes, data
types, block sizes, layouts and masks.  Inputs are synthetic, drawn on the GPU from a seed.
"""
import math

import torch

from torch_blocksparse_b200 import (Linear, MatMul, MultiheadAttention, Softmax, SparseSelfAttention, SparsityConfig,
                                    layouts)

DTYPES = {'fp32': torch.float32, 'fp16': torch.float16, 'bf16': torch.bfloat16}
# Another correct implementation keeps 32-bit sums but may add in another order and round an
# intermediate (scores, probabilities, their gradients) to the storage type at another place.
TOLERANCE = {'fp32': {'rel': 1e-5}, 'fp16': {'rel': 3e-3}, 'bf16': {'rel': 1e-2}}


def listed():
    return [
        # One short sequence, forward only: what a serving program calls per layer; all latency.
        dict(name='attention_infer_short', op='attention', dtype='fp16', train=False, batch=1, heads=12, length=1024,
             head_dim=64, block=64, layout='fixed', masks='none'),
        # SparsityConfig() as it comes (block 16, windows of 64): a small model's training step.
        dict(name='attention_train_default', op='attention', dtype='fp16', train=True, batch=4, heads=8, length=2048,
             head_dim=64, block=16, layout='config', masks='none'),
        # A padded batch of sequences whose length is no multiple of 64, sliding window.
        dict(name='attention_train_ragged', op='attention', dtype='bf16', train=True, batch=3, heads=10, length=2016,
             head_dim=64, block=32, layout='band', masks='padding'),
        # Relative position bias, key padding and a causal mask together, batch 4.
        dict(name='attention_train_masked', op='attention', dtype='fp16', train=True, batch=4, heads=16, length=4096,
             head_dim=64, block=64, layout='fixed', masks='all'),
        # The benchmark's workload: long sequences, fixed layout, local windows of 4 blocks.
        dict(name='attention_train_8k', op='attention', dtype='fp16', train=True, batch=8, heads=16, length=8192,
             head_dim=64, block=64, layout='fixed', masks='none'),
        # The benchmark's BigBird-style workload at a batch of 4: the longest sequences, head_dim 128.
        dict(name='attention_train_bigbird', op='attention', dtype='bf16', train=True, batch=4, heads=16, length=16384,
             head_dim=128, block=128, layout='bigbird', masks='none'),
        # The drop-in for torch.nn.MultiheadAttention, projections included.
        dict(name='mha_train', op='mha', dtype='bf16', train=True, batch=4, heads=16, length=2048, head_dim=64, block=32,
             layout='fixed', masks='none'),
        # The three operations of the reference one after the other, as programs written for it do.
        dict(name='chain_train', op='chain', dtype='fp16', train=True, batch=2, heads=8, length=2048, head_dim=64,
             block=32, layout='fixed', masks='padding'),
        # The benchmark's softmax: every optional input, in place.
        dict(name='softmax_masked', op='softmax', dtype='fp16', train=False, batch=8, heads=16, length=4096, block=64,
             layout='band', masks='all'),
        # The benchmark's smallest product, with both gradients: FP32, block 16.
        dict(name='matmul_sdd_fp32', op='matmul', dtype='fp32', train=True, batch=4, heads=2, mode='sdd', m=256, n=512,
             k=384, block=16, density=0.5, trans_a=True, trans_b=False),
        # The benchmark's large products of small blocks, with both gradients.
        dict(name='matmul_dsd_fp16', op='matmul', dtype='fp16', train=True, batch=8, heads=8, mode='dsd', m=2048, n=2048,
             k=2048, block=32, density=0.25, trans_a=False, trans_b=False),
        # A feed-forward layer with a block-sparse weight, on a number of tokens that is a multiple of nothing.
        dict(name='linear_train', op='linear', dtype='bf16', train=True, tokens=4093, n_in=1024, n_out=4096, block=32,
             density=0.25),
    ]


# ---- drawn cases ------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_tokens(rng, block, head_dims, longest):
    """Fields that every attention-like case has; lengths are whole blocks, odd counts among them."""
    layout = rng.choice(['fixed', 'fixed', 'fixed_bi', 'band', 'bigbird'])
    nb = _log(rng, max(8, 256 // block), min(longest // block, 512))
    if layout.startswith('fixed'):
        nb = max(8, nb // 4 * 4)                 # whole windows of 4 blocks
    return dict(dtype=rng.choice(['fp16', 'bf16']), train=rng.random() < 0.7, batch=_log(rng, 1, 8),
                heads=rng.choice([2, 4, 6, 8, 10, 12, 16]), length=nb * block, head_dim=rng.choice(head_dims), block=block,
                layout=layout)


def _draw(rng):
    op = rng.choices(['attention', 'mha', 'chain', 'softmax', 'matmul', 'linear'], [5, 1, 2, 1, 3, 1])[0]
    block = rng.choice([16, 32, 64, 64, 128])
    if op == 'attention':
        masks = rng.choice(['none', 'none', 'padding', 'all'])
        c = _draw_tokens(rng, block, [32, 64, 64, 64, 96, 128, 128], 4096 if masks == 'all' else 16384)
        return dict(op=op, **c, masks=masks)
    if op == 'mha':
        c = _draw_tokens(rng, block, [32, 64, 64, 128], 4096)
        return dict(op=op, **c, masks=rng.choice(['none', 'padding']))
    if op == 'chain':
        c = _draw_tokens(rng, block, [32, 64, 64, 80, 128], 4096)
        c['dtype'] = rng.choice(['fp32', 'fp16', 'fp16', 'bf16'])
        return dict(op=op, **c, masks=rng.choice(['none', 'padding', 'all']))
    if op == 'softmax':
        c = _draw_tokens(rng, block, [64], 4096)
        c['dtype'] = rng.choice(['fp32', 'fp16', 'bf16'])
        c['train'] = False
        del c['head_dim']
        return dict(op=op, **c, masks=rng.choice(['none', 'padding', 'all']))
    if op == 'matmul':
        mode = rng.choice(['sdd', 'dsd', 'dds'])
        train = rng.random() < 0.6
        size = {d: max(block, _log(rng, 128, 4096) // block * block) for d in 'mnk'}
        # the dimension no block covers: a multiple of 16 where a product reduces over it, else anything
        free = {'sdd': 'k', 'dsd': 'n', 'dds': 'm'}[mode]
        size[free] = _log(rng, 64, 4096)
        if mode == 'sdd' or train:
            size[free] = max(16, size[free] // 16 * 16)
        return dict(op=op, dtype=rng.choice(['fp32', 'fp16', 'fp16', 'bf16']), train=train, batch=_log(rng, 1, 8),
                    heads=rng.choice([1, 2, 4, 8]), mode=mode, **size, block=block, density=rng.choice([0.1, 0.25, 0.5]),
                    trans_a=rng.random() < 0.5, trans_b=rng.random() < 0.5)
    return dict(op=op, dtype=rng.choice(['fp16', 'bf16']), train=rng.random() < 0.7, tokens=_log(rng, 64, 16384),
                n_in=block * max(1, _log(rng, 256, 4096) // block), n_out=block * max(1, _log(rng, 256, 8192) // block),
                block=block, density=rng.choice([0.1, 0.25, 0.5]))


def _cost(case):
    """Work in bytes, with operations at 200 per byte (FP32 ones run without tensor cores: 10)."""
    w = work(case)
    return max(w['bytes'], w['flops'] / (10 if case['dtype'] == 'fp32' else 200))


def draw(rng):
    most = max(_cost(c) for c in listed()) / 4
    while True:
        case = _draw(rng)
        if _cost(case) <= most:
            return case


# ---- layouts ----------------------------------------------------------------------------------
def _layout(case):
    if case['op'] in ('matmul', 'linear'):
        if case['op'] == 'linear':
            heads, rows, cols = 1, case['n_in'], case['n_out']
        else:
            rows, cols = {'sdd': ('m', 'n'), 'dsd': ('m', 'k'), 'dds': ('k', 'n')}[case['mode']]
            flip = case['trans_a'] if case['mode'] == 'dsd' else case['trans_b'] if case['mode'] == 'dds' else False
            heads, rows, cols = case['heads'], case[cols if flip else rows], case[rows if flip else cols]
        shape = (heads, rows // case['block'], cols // case['block'])
        lay = torch.bernoulli(torch.full(shape, case['density']), generator=torch.Generator().manual_seed(0)).long()
        lay[:, 0, 0] = 1                         # no head without a block
        return lay
    heads, nb = case['heads'], case['length'] // case['block']
    if case['layout'] == 'config':               # what SparsityConfig() describes
        return layouts.fixed(heads, nb, 64 // case['block'])
    if case['layout'] == 'fixed':
        return layouts.fixed(heads, nb, 4)
    if case['layout'] == 'fixed_bi':
        return layouts.fixed(heads, nb, 4, 'bidirectional')
    if case['layout'] == 'band':
        return layouts.causal_band(heads, nb, 4, 1)
    return layouts.bigbird(heads, nb, 3, 3, 2, seed=0)


# ---- inputs -----------------------------------------------------------------------------------
class _Inputs:
    """Tensors on the GPU from one seed."""

    def __init__(self, seed, dtype):
        self.gen = torch.Generator('cuda').manual_seed(seed)
        self.dtype = DTYPES[dtype]

    def normal(self, *shape, scale=1.0):
        return (torch.randn(shape, generator=self.gen, device='cuda') * scale).to(self.dtype)

    def leaf(self, *shape, scale=1.0):
        return self.normal(*shape, scale=scale).requires_grad_()

    def padding(self, batch, length, mode):
        """Valid lengths uniform in [length / 2, length]: 1 / 0 for 'mul', 0 / -inf for 'add'."""
        n = torch.randint(length // 2, length + 1, (batch, 1), generator=self.gen, device='cuda')
        seen = torch.arange(length, device='cuda')[None, :] < n
        if mode == 'mul':
            return seen.to(self.dtype)
        return torch.zeros((batch, length), dtype=self.dtype, device='cuda').masked_fill(~seen, float('-inf'))

    def masks(self, case):
        """(keyword arguments, (key_padding_mask_mode, attn_mask_mode)) of an attention or softmax call."""
        z, h, length = case['batch'], case['heads'], case['length']
        if case['masks'] == 'none':
            return {}, ('add', 'mul')
        if case['masks'] == 'padding':
            return dict(key_padding_mask=self.padding(z, length, 'mul')), ('mul', 'mul')
        # (a causal mask: every layout has the diagonal blocks, so every query sees itself)
        return dict(rpe=self.normal(h, length, length, scale=0.1), key_padding_mask=self.padding(z, length, 'add'),
                    attn_mask=torch.ones((length, length), dtype=self.dtype, device='cuda').tril()), ('add', 'mul')


def prepare(case, seed):
    g = _Inputs(seed, case['dtype'])
    op, block, lay = case['op'], case['block'], _layout(case)
    s = dict(op=op, train=case['train'])
    if op in ('attention', 'chain', 'softmax'):
        z, h, length = case['batch'], case['heads'], case['length']
        s['masks'], modes = g.masks(case)
        if op == 'softmax':
            s['x'] = g.normal(z, int(lay.sum()), block, block)
            s['softmax'] = Softmax(lay, block)
            s['scale'] = 0.125
            s['masks'].update(key_padding_mask_mode=modes[0], attn_mask_mode=modes[1])
            return s
        make = g.leaf if s['train'] else g.normal
        s['q'], s['k'], s['v'] = (make(z, h, length, case['head_dim']) for _ in range(3))
        s['dout'] = g.normal(z, h, length, case['head_dim'])
        if op == 'attention':
            if case['layout'] == 'config':
                s['module'] = SparseSelfAttention(SparsityConfig(), key_padding_mask_mode=modes[0], attn_mask_mode=modes[1])
            else:
                s['module'] = SparseSelfAttention(layout=lay, block=block, key_padding_mask_mode=modes[0],
                                                  attn_mask_mode=modes[1])
            return s
        s['sdd'] = MatMul(lay, block, 'sdd', trans_a=False, trans_b=True)
        s['softmax'] = Softmax(lay, block)
        s['dsd'] = MatMul(lay, block, 'dsd', trans_a=False, trans_b=False)
        s['scale'] = case['head_dim'] ** -0.5
        s['masks'].update(key_padding_mask_mode=modes[0], attn_mask_mode=modes[1])
    elif op == 'mha':
        z, length, width = case['batch'], case['length'], case['heads'] * case['head_dim']
        mode = 'mul' if case['masks'] == 'padding' else 'add'
        mha = MultiheadAttention(width, case['heads'], lay, block, key_padding_mask_mode=mode).to('cuda', g.dtype)
        with torch.no_grad():
            for p in mha.parameters():
                p.copy_(g.normal(*p.shape, scale=width ** -0.5))
        mha.requires_grad_(s['train'])
        s['module'], s['params'] = mha, list(mha.parameters())
        s['x'] = g.normal(length, z, width).requires_grad_(s['train'])
        s['dout'] = g.normal(length, z, width)
        s['padding'] = g.padding(z, length, 'mul') if case['masks'] == 'padding' else None
    elif op == 'matmul':
        z, h, m, n, k = (case[f] for f in ('batch', 'heads', 'm', 'n', 'k'))
        make = g.leaf if s['train'] else g.normal
        shape = {'a': (z, h, k, m) if case['trans_a'] else (z, h, m, k), 'b': (z, h, n, k) if case['trans_b'] else (z, h, k, n),
                 'c': (z, h, m, n)}
        shape[{'sdd': 'c', 'dsd': 'a', 'dds': 'b'}[case['mode']]] = (z, int(lay.sum()), block, block)
        s['a'], s['b'] = (make(*shape[f], scale=k ** -0.5) for f in 'ab')
        s['dout'] = g.normal(*shape['c'], scale=k ** -0.5)
        s['matmul'] = MatMul(lay, block, case['mode'], trans_a=case['trans_a'], trans_b=case['trans_b'])
    else:
        layer = Linear(case['n_in'], case['n_out'], block, lay).to('cuda', g.dtype)
        with torch.no_grad():
            layer.weight.copy_(g.normal(*layer.weight.shape, scale=case['n_in'] ** -0.5))
        s['layer'] = layer.requires_grad_(s['train'])
        s['x'] = g.normal(case['tokens'], case['n_in']).requires_grad_(s['train'])
        s['dout'] = g.normal(case['tokens'], case['n_out'])
    return s


# ---- one pass ---------------------------------------------------------------------------------
def run(s):
    op = s['op']
    if op == 'softmax':
        with torch.no_grad():
            return s['softmax'](s['x'], scale=s['scale'], **s['masks'])
    with torch.set_grad_enabled(s['train']):
        if op == 'attention':
            inputs = (s['q'], s['k'], s['v'])
            out = s['module'](*inputs, **s['masks'])
        elif op == 'chain':
            inputs = (s['q'], s['k'], s['v'])
            w = s['softmax'](s['sdd'](s['q'], s['k']), scale=s['scale'], **s['masks'])
            out = s['dsd'](w, s['v'])
        elif op == 'mha':
            inputs = (s['x'], *s['params'])
            out, _ = s['module'](s['x'], s['x'], s['x'], key_padding_mask=s['padding'])
        elif op == 'matmul':
            inputs = (s['a'], s['b'])
            out = s['matmul'](*inputs)
        else:
            inputs = (s['x'], s['layer'].weight)
            out = s['layer'](s['x'])
    if not s['train']:
        return out
    return (out, *torch.autograd.grad(out, inputs, s['dout']))


# ---- what a pass cannot do without -------------------------------------------------------------
def work(case):
    op, block, nnz, e = case['op'], case['block'], int(_layout(case).sum()), DTYPES[case['dtype']].itemsize
    passes = 3 if case['train'] else 1           # a product's gradients are two more products of its size
    if op in ('attention', 'chain', 'mha', 'softmax'):
        z, h, length = case['batch'], case['heads'], case['length']
        masks = {'none': 0, 'padding': z * length, 'all': nnz * block * block + z * length + length * length}[case['masks']]
        if op == 'softmax':
            return dict(bytes=e * (2 * z * nnz * block * block + masks), flops=0)
        d = case['head_dim']
        width = h * d
        flops = passes * 4 * z * nnz * block * block * d
        if op == 'mha':
            tokens = e * z * length * width          # x, out and, in training, dout and dx
            weights = e * (4 * width * width + 4 * width)
            return dict(bytes=(4 if case['train'] else 2) * tokens + (2 if case['train'] else 1) * weights + e * masks,
                        flops=flops + passes * 8 * z * length * width * width)
        return dict(bytes=e * ((8 if case['train'] else 4) * z * length * width + masks), flops=flops)
    if op == 'matmul':
        z, h, m, n, k = (case[f] for f in ('batch', 'heads', 'm', 'n', 'k'))
        sizes = {'a': z * h * m * k, 'b': z * h * k * n, 'c': z * h * m * n}
        sizes[{'sdd': 'c', 'dsd': 'a', 'dds': 'b'}[case['mode']]] = z * nnz * block * block
        free = {'sdd': k, 'dsd': n, 'dds': m}[case['mode']]
        return dict(bytes=(2 if case['train'] else 1) * e * sum(sizes.values()), flops=passes * 2 * z * nnz * block * block * free)
    t = case['tokens']
    return dict(bytes=(2 if case['train'] else 1) * e * (t * (case['n_in'] + case['n_out']) + nnz * block * block),
                flops=passes * 2 * t * nnz * block * block)


def tolerance(case):
    return TOLERANCE[case['dtype']]
