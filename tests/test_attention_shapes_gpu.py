"""The tcgen05 attention at head dimensions below the two it is compiled for and at sequences that end
inside a chunk of 64 rows, against the CPU oracle (tolerances of tests/util.py)."""
import pytest
import torch

from tests.test_attention_gpu import check, no_device_side_timeout, rand_qkv  # noqa: F401
from torch_blocksparse_b200 import SparseSelfAttention, tables

pytestmark = pytest.mark.gpu


def layout_of(H, nb, seed):
    g = torch.Generator().manual_seed(seed)
    layout = (torch.rand((H, nb, nb), generator=g) > 0.5).long()
    layout[:, :, 0] = 1
    layout[0, nb - 1, :] = 0                  # the last block-row without any block
    layout[1, :, nb - 1] = 0                  # and the last block-column
    return layout


def masks_of(which, Z, H, L, dtype, seed):
    if which == 'none':
        return {}, 'add', 'mul'
    g = torch.Generator().manual_seed(seed)
    keep = torch.rand((Z, L), generator=g) > 0.3
    keep[:, 0] = True
    if which == 'padding':
        return dict(key_padding_mask=keep.to(dtype)), 'mul', 'mul'
    rpe = (0.5 * torch.randn((H, L, L), generator=g)).to(dtype)[None].repeat(Z, 1, 1, 1)
    kpm = torch.where(keep, 0.0, float('-inf')).to(dtype)
    if which == 'causal':
        return dict(rpe=rpe, key_padding_mask=kpm, attn_mask=torch.tril(torch.ones((L, L))).to(dtype)), 'add', 'mul'
    seen = (torch.rand((L, L), generator=g) > 0.2)
    seen[:, 0] = True
    return dict(rpe=rpe, key_padding_mask=kpm, attn_mask=torch.where(seen, 0.0, float('-inf')).to(dtype)), 'add', 'add'


@pytest.mark.parametrize('which', ['none', 'padding', 'causal', 'all'])
@pytest.mark.parametrize('D,block', [(8, 64), (32, 16), (32, 128), (40, 64), (72, 32), (80, 64), (96, 64), (120, 128)])
def test_head_dimensions(D, block, which):
    Z, H, nb = 2, 2, max(4, 256 // block)
    dtype = torch.bfloat16 if D in (72, 120) else torch.float16
    q, k, v, do = rand_qkv(Z, H, nb * block, D, dtype, seed=D)
    kw, km, am = masks_of(which, Z, H, nb * block, dtype, seed=D)
    check(layout_of(H, nb, D), block, q, k, v, do, True, km, am, **kw)


@pytest.mark.parametrize('which', ['none', 'padding', 'causal', 'all'])
@pytest.mark.parametrize('block,nb', [(16, 5), (16, 6), (16, 11), (32, 5), (32, 7)])
@pytest.mark.parametrize('D', [64, 128, 96, 32])
def test_sequences_that_end_inside_a_chunk(block, nb, D, which):
    Z, H = 2, 2
    q, k, v, do = rand_qkv(Z, H, nb * block, D, torch.float16, seed=nb)
    kw, km, am = masks_of(which, Z, H, nb * block, torch.float16, seed=nb)
    check(layout_of(H, nb, nb), block, q, k, v, do, True, km, am, **kw)


def test_operands_tensor_maps_cannot_describe():
    """Head dimensions only the tcgen05 kernels take: broadcast operands and masks off the 16-byte grid
    are copied."""
    Z, H, L, D, block = 3, 2, 256, 32, 32
    layout = layout_of(H, L // block, 3)
    q, k, v, do = rand_qkv(1, H, L, D, torch.float16, seed=1)
    mod = SparseSelfAttention(layout=layout, block=block, key_padding_mask_mode='mul')
    pad = torch.ones(Z, L + 1, dtype=torch.float16, device='cuda')[:, 1:]
    qe, ke, ve = (t.cuda().expand(Z, -1, -1, -1).requires_grad_() for t in (q, k, v))
    o = mod(qe, ke, ve, key_padding_mask=pad)
    # (the same kernel on operands and a mask that need no copy: the same bits)
    one = mod(q.cuda(), k.cuda(), v.cuda(), key_padding_mask=torch.ones(1, L, dtype=torch.float16, device='cuda'))
    assert torch.equal(o, one.expand(Z, -1, -1, -1))
    o.sum().backward()                        # (an expanded gradient)


@pytest.mark.parametrize('block,nb', [(16, 5), (16, 7), (16, 33), (32, 3), (32, 65)])
def test_tile_lists_of_ragged_layouts_device_against_host(block, nb):
    layout = layout_of(2, nb, nb)
    want, got = tables.build_attn_tiles(layout, block), tables.build_attn_tiles_device(layout.cuda(), block)
    assert torch.equal(want.hdr, got.hdr) and torch.equal(want.host, got.host[:want.host.numel()])
    tables.validate_device_buffer(got.on('cuda'), tiles=True)


@pytest.mark.parametrize('which', ['none', 'padding', 'causal'])
@pytest.mark.parametrize('D', [96, 128])
def test_tiles_of_few_chunks(D, which):
    """Two groups of warps on alternating chunks: tiles of 1 to 9 chunks of keys (a second group with
    nothing to do, rings that do and do not wrap), and of queries in the gradients."""
    Z, H, nb = 2, 2, 17
    layout = torch.zeros((H, nb, nb), dtype=torch.long)
    for i in range(nb):
        layout[0, i, :i // 2 + 1] = 1
        layout[1, :i // 2 + 1, nb - 1 - i] = 1
    q, k, v, do = rand_qkv(Z, H, nb * 64, D, torch.float16, seed=D)
    kw, km, am = masks_of(which, Z, H, nb * 64, torch.float16, seed=5)
    check(layout, 64, q, k, v, do, True, km, am, **kw)


@pytest.mark.parametrize('D', [32, 64, 96])
def test_profiled_calls_take_the_same_operands(D, monkeypatch):
    """With an event pair around every kernel a call gives the same bits, on operands that have to be copied too."""
    from torch_blocksparse_b200 import fused
    Z, H, L, block = 2, 2, 256, 32
    q, k, v, do = rand_qkv(1, H, L, D, torch.float16, seed=1)
    mod = SparseSelfAttention(layout=layout_of(H, L // block, 3), block=block, key_padding_mask_mode='mul')
    pad = torch.ones(Z, L + 1, dtype=torch.float16, device='cuda')[:, 1:]
    rpe = 0.1 * torch.randn(H, L, L + 1, device='cuda').half()[..., 1:]
    xs = [t.cuda().expand(Z, -1, -1, -1).requires_grad_() for t in (q, k, v)]
    results = []
    for profile in (None, []):
        monkeypatch.setattr(fused, 'PROFILE', profile)
        o = mod(*xs, rpe=rpe, key_padding_mask=pad)
        results.append((o, *torch.autograd.grad(o, xs, do.cuda().expand(Z, -1, -1, -1))))
    assert len(fused.PROFILE) == 4
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize('which', ['none', 'padding'])
@pytest.mark.parametrize('D,block', [(128, 64), (96, 32), (128, 128), (64, 64)])
def test_results_do_not_depend_on_the_order_of_tiles(D, block, which):
    """More tiles than SMs, taken over by running CTAs in any order: the bits of every batch entry are those it has
    alone, where each CTA runs one tile, call after call."""
    Z, H, L = 6, 4, 2560
    q, k, v, do = (t.cuda() for t in rand_qkv(Z, H, L, D, torch.float16, seed=D))
    kw, km, am = masks_of(which, Z, H, L, torch.float16, seed=2)
    kw = {n: t.cuda() for n, t in kw.items()}
    mod = SparseSelfAttention(layout=layout_of(H, L // block, 7), block=block, key_padding_mask_mode=km, attn_mask_mode=am)

    def results(z):
        xs = [t[z].clone().requires_grad_() for t in (q, k, v)]
        o = mod(*xs, **{n: t[z] for n, t in kw.items()})
        return (o, *torch.autograd.grad(o, xs, do[z]))
    alone = [results(slice(z, z + 1)) for z in range(Z)]
    for _ in range(3):
        for i, got in enumerate(results(slice(0, Z))):
            assert torch.equal(got, torch.cat([one[i] for one in alone]))
