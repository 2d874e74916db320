"""The native module behind the public classes (csrc/torch/ops.cpp): what the other tests do not
reach through them."""
import copy
import pickle

import pytest
import torch

from torch_blocksparse_b200 import MatMul, Softmax, SparseSelfAttention

LAYOUT = torch.tril(torch.ones((2, 4, 4), dtype=torch.long))


def test_owners_of_native_operations_copy_and_pickle():
    """Operations are per object and device; copies start without them."""
    for op, args in ((MatMul(LAYOUT, 16, 'sdd'), (torch.zeros(1, 2, 64, 16), torch.zeros(1, 2, 16, 64))),
                     (Softmax(LAYOUT, 16), (torch.zeros(1, 20, 16, 16),))):
        with pytest.raises(RuntimeError, match='CUDA tensors only'):
            op(*args)
        assert len(op._ops) == 1
        assert len(copy.deepcopy(op)._ops) == 0 and len(pickle.loads(pickle.dumps(op))._ops) == 0
    assert copy.deepcopy(SparseSelfAttention(layout=LAYOUT, block=16))._attn == {}


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float32, torch.float16, torch.bfloat16])
def test_timed_calls_and_versions(dtype):
    """bench=True times the forward; the softmax marks its operand as modified, with and without grad."""
    a, b = torch.randn(2, 2, 64, 32, device='cuda', dtype=dtype), torch.randn(2, 2, 32, 64, device='cuda', dtype=dtype)
    mm = MatMul(LAYOUT, 16, 'sdd', bench=True)
    w = mm(a.requires_grad_(), b)
    assert mm.time_c > 0 and torch.equal(w, MatMul(LAYOUT, 16, 'sdd')(a, b))
    sm = Softmax(LAYOUT, 16, bench=True)
    for x in (w, w.detach().clone()):
        before = x._version
        y = sm(x)
        assert y is x and x._version > before and sm.time_y > 0


@pytest.mark.gpu
@pytest.mark.parametrize('block', [32, 64, 128])
@pytest.mark.parametrize('heads', [1, 2])
@pytest.mark.parametrize('free', [8, 72, 120, 136, 250, 264, 520])
@pytest.mark.parametrize('trans', [False, True])
def test_products_with_ragged_free_dimensions(product_family, block, heads, free, trans):
    """dsd, dds and sdd at widths around the tiles of 128 and 256 columns and the 64 of a K stage, with
    batch and heads of one (whose strides carry no meaning), against an FP32 dense product."""
    g = torch.Generator().manual_seed(block + free)
    nb = 5
    layout = (torch.rand((heads, nb, nb), generator=g) > 0.5).long()
    layout[:, 0, 0] = 1
    n = nb * block
    idx = layout.nonzero()

    def dense(s):                                       # block format -> [1, heads, n, n]
        d = torch.zeros(1, heads, nb, block, nb, block, device='cuda')
        d[:, idx[:, 0], idx[:, 1], :, idx[:, 2]] = s.float().transpose(0, 1)
        return d.reshape(1, heads, n, n)
    rand = lambda *shape: torch.randn(shape, generator=g).half().cuda()
    s = rand(1, len(idx), block, block)
    # FP16 results of FP32 sums: one rounding (2^-11) of values of about sqrt(n)
    close = lambda got, want: torch.testing.assert_close(got.float(), want, rtol=1e-3, atol=2e-3 * n ** 0.5)
    x = rand(1, heads, free, n) if trans else rand(1, heads, n, free)
    xn = x.transpose(2, 3) if trans else x
    close(MatMul(layout, block, 'dsd', trans_b=trans)(s, x), dense(s) @ xn.float())
    x = rand(1, heads, n, free) if trans else rand(1, heads, free, n)
    xn = x.transpose(2, 3) if trans else x
    close(MatMul(layout, block, 'dds', trans_a=trans)(x, s), xn.float() @ dense(s))
    k = max(16, free // 16 * 16)
    a, b = rand(1, heads, n, k), rand(1, heads, n, k) if trans else rand(1, heads, k, n)
    want = a.float() @ (b.transpose(2, 3) if trans else b).float()
    close(dense(MatMul(layout, block, 'sdd', trans_b=trans)(a, b)), want * dense(torch.ones_like(s)))


@pytest.mark.gpu
@pytest.mark.parametrize('block', [16, 32, 128])
@pytest.mark.parametrize('rows', [1, 7, 129, 1000])
def test_linear_with_any_number_of_rows(product_family, block, rows):
    """Forward and both gradients of Linear against the dense layer."""
    from torch_blocksparse_b200 import Linear
    g = torch.Generator().manual_seed(rows)
    layout = (torch.rand((3, 4), generator=g) > 0.4).long()
    layout[0, 0] = 1
    lin = Linear(3 * block, 4 * block, block, layout).to('cuda', torch.float16)
    x = torch.randn((2, rows, 3 * block), generator=g).half().cuda().requires_grad_()
    dy = torch.randn((2, rows, 4 * block), generator=g).half().cuda()
    idx = layout.nonzero()
    w = torch.zeros(3, block, 4, block, device='cuda')
    w[idx[:, 0], :, idx[:, 1]] = lin.weight.detach().float()
    w = w.reshape(3 * block, 4 * block)
    y = lin(x)
    dx, dw = torch.autograd.grad(y, (x, lin.weight), dy)
    x2, dy2 = x.detach().float().reshape(-1, 3 * block), dy.float().reshape(-1, 4 * block)
    want_dw = (x2.T @ dy2).reshape(3, block, 4, block)[idx[:, 0], :, idx[:, 1]]
    for got, want in ((y, (x2 @ w).view_as(y)), (dx, (dy2 @ w.T).view_as(dx)), (dw, want_dw)):
        torch.testing.assert_close(got.float(), want, rtol=2e-3, atol=2e-3 * float(want.pow(2).mean().sqrt() + 1e-3))


@pytest.mark.gpu
@pytest.mark.parametrize('grad', [False, True])
def test_forward_mode_tangents_are_refused(grad):
    """No operation has a forward-mode derivative: a dual tensor is an error, with and without gradients on."""
    import torch.autograd.forward_ad as fwd
    from torch_blocksparse_b200 import Linear, MatMul, Softmax, SparseSelfAttention
    lay = torch.ones((1, 2, 2), dtype=torch.long)
    make = lambda *s: torch.randn(s, device='cuda', dtype=torch.float16)
    layer = Linear(64, 64, 32, lay).to('cuda', torch.float16)
    layer.requires_grad_(grad)
    with torch.set_grad_enabled(grad), fwd.dual_level():
        x, q, rows = (fwd.make_dual(make(*s), make(*s)) for s in ((1, 4, 32, 32), (1, 1, 64, 64), (5, 64)))
        for call in (lambda: MatMul(lay, 32, 'sdd')(q, make(1, 1, 64, 64)), lambda: Softmax(lay, 32)(x), lambda: layer(rows),
                     lambda: SparseSelfAttention(layout=lay, block=32)(q, make(1, 1, 64, 64), make(1, 1, 64, 64))):
            with pytest.raises((RuntimeError, NotImplementedError)):
                call()


def test_recorded_calls_replay_with_gradients():
    """torch.jit.trace on CPU: an operation whose result the tracer cannot see (raw memory) is replayed on new
    inputs, with plain and absent arguments, and the trace passes the tracer's own check."""
    from torch_blocksparse_b200 import tracing

    class Op:
        def run(self, a, mask, b, factor):
            class Hidden(torch.autograd.Function):
                @staticmethod
                def forward(ctx, a, b):
                    ctx.save_for_backward(a, b)
                    out = torch.empty((a.size(0), b.size(1)))
                    out.numpy()[...] = factor * (a.detach().numpy() @ b.detach().numpy())
                    return out

                @staticmethod
                def backward(ctx, g):
                    a, b = ctx.saved_tensors
                    return factor * (g @ b.T), factor * (a.T @ g)
            return Hidden.apply(a, b)
    op = Op()
    g = torch.Generator().manual_seed(0)
    draw = lambda grad: [torch.randn((3, 3), generator=g).requires_grad_(grad) for _ in range(2)]
    call = lambda a, b: tracing.call(op, 'run', tracing.call(op, 'run', a, None, b, 2.0), None, b, 0.5) + a
    for grad in (True, False):
        traced = torch.jit.trace(call, draw(grad))
        a, b = draw(True)
        want = (a @ b) @ b + a
        torch.testing.assert_close(traced(a, b), want)
        dy = torch.randn((3, 3), generator=g)
        torch.testing.assert_close(torch.autograd.grad(traced(a, b), (a, b), dy), torch.autograd.grad(want, (a, b), dy))
    with pytest.raises(RuntimeError, match='torch.jit.trace'):
        torch.jit.trace(lambda x: Softmax(LAYOUT, 16)(x * 1), torch.zeros(1, 20, 16, 16), check_trace=False)


@pytest.mark.gpu
@pytest.mark.parametrize('which', ['matmul', 'linear', 'attention', 'masked'])
def test_traced_calls_run_their_kernels_again(which):
    """A trace of the public classes, replayed on inputs it was not recorded with: the same bits as the call itself,
    and the same gradients."""
    from torch_blocksparse_b200 import Linear
    g = torch.Generator('cuda').manual_seed(0)
    draw = lambda *s: torch.randn(s, generator=g, device='cuda', dtype=torch.float16).requires_grad_()
    if which == 'matmul':
        mod, shapes = MatMul(LAYOUT, 16, 'sdd', trans_b=True), [(2, 2, 64, 32)] * 2
    elif which == 'linear':
        mod, shapes = Linear(64, 64, 16, LAYOUT[0]).to('cuda', torch.float16), [(5, 64)]
    else:
        mod, shapes = SparseSelfAttention(layout=LAYOUT, block=64, key_padding_mask_mode='mul'), [(2, 2, 256, 64)] * 3
    mask = {}
    if which == 'masked':
        mask['key_padding_mask'] = (torch.arange(256, device='cuda') < torch.tensor([[200], [256]], device='cuda')).half()

    class Call(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.mod = mod

        def forward(self, *xs):
            return self.mod(*xs, **mask) * 1
    call = Call()
    traced = torch.jit.trace(call, [draw(*s) for s in shapes])
    xs = [draw(*s) for s in shapes]
    want, got = call(*xs), traced(*xs)
    assert torch.equal(got, want)
    dy = torch.randn_like(want)
    for a, b in zip(torch.autograd.grad(got, xs, dy), torch.autograd.grad(want, xs, dy)):
        assert torch.equal(a, b)
    with torch.no_grad():
        assert torch.equal(traced(*xs), want)


def test_operands_of_another_type_or_device_are_refused():
    """Before anything is launched: kernels read every operand through a pointer, as the type of the first."""
    zeros = lambda *s, dtype=torch.float16, device='cpu': torch.zeros(s, dtype=dtype, device=device)
    from torch_blocksparse_b200 import Linear
    q = zeros(1, 2, 64, 96)
    att = SparseSelfAttention(layout=LAYOUT, block=16)
    for other in (dict(dtype=torch.bfloat16), dict(dtype=torch.float32)):
        for args in ((q, zeros(1, 2, 64, 96, **other), q), (q, q, zeros(1, 2, 64, 96, **other))):
            with pytest.raises(ValueError, match='must be Half'):
                att(*args)
        with pytest.raises(ValueError, match='same dtype'):
            MatMul(LAYOUT, 16, 'sdd')(zeros(1, 2, 64, 16), zeros(1, 2, 16, 64, **other))
    elsewhere = dict(device='meta')
    for args, kw in (((q, zeros(1, 2, 64, 96, **elsewhere), q), {}), ((q, q, zeros(1, 2, 64, 96, **elsewhere)), {}),
                     ((q, q, q), dict(rpe=zeros(2, 64, 64, **elsewhere))),
                     ((q, q, q), dict(key_padding_mask=zeros(2, 64, **elsewhere)))):
        with pytest.raises(RuntimeError, match='is on meta'):
            att(*args, **kw)
    x = zeros(1, 20, 16, 16)
    for name, shape in (('rpe', (2, 64, 64)), ('key_padding_mask', (1, 64)), ('attn_mask', (64, 64))):
        with pytest.raises(RuntimeError, match='is on meta'):
            Softmax(LAYOUT, 16)(x, **{name: zeros(*shape, **elsewhere)})
    with pytest.raises(ValueError, match=r'\[Z, H, L, D\]'):
        from torch_blocksparse_b200 import fused
        op = fused.Attention(MatMul(LAYOUT, 16, 'sdd').meta, None, 16, torch.device('cpu'))
        fused.attention(op, q, q[..., :64], q, 1.0)
    with pytest.raises(RuntimeError, match='CUDA tensors only'):
        Linear(64, 64, 16, LAYOUT[0])(zeros(3, 64))


@pytest.mark.gpu
def test_operands_on_the_host_are_refused_beside_a_device():
    zeros = lambda *s, device='cuda': torch.zeros(s, dtype=torch.float16, device=device)
    from torch_blocksparse_b200 import Linear
    q = zeros(1, 2, 64, 64)
    lin = Linear(64, 64, 16, LAYOUT[0])
    for call in (lambda: MatMul(LAYOUT, 16, 'sdd')(q, zeros(1, 2, 64, 64, device='cpu')), lambda: lin(zeros(3, 64)),
                 lambda: SparseSelfAttention(layout=LAYOUT, block=16)(q, q, zeros(1, 2, 64, 64, device='cpu')),
                 lambda: SparseSelfAttention(layout=LAYOUT, block=16)(q, q, q, key_padding_mask=zeros(2, 64, device='cpu')),
                 lambda: Softmax(LAYOUT, 16)(zeros(1, 20, 16, 16), attn_mask=zeros(64, 64, device='cpu'))):
        with pytest.raises(RuntimeError, match='cpu'):
            call()
    with pytest.raises(ValueError, match='graphed step'):
        SparseSelfAttention(layout=LAYOUT, block=16).graphed(q, q.bfloat16(), q, q)


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float16, torch.float32])
@pytest.mark.parametrize('free', [1, 2, 13, 33])
@pytest.mark.parametrize('block', [16, 64])
@pytest.mark.parametrize('where', ['whole', 'transposed', 'unaligned', 'odd rows', 'every other', 'expanded'])
def test_widths_of_views(product_family, dtype, free, block, where):
    """Dense operands of dsd and dds whose width is no multiple of 16 bytes, as views of any orientation, alignment
    and row distance: what cannot be read where it lies is copied, never refused."""
    g = torch.Generator('cuda').manual_seed(free)
    H, nb = 2, 3
    n = nb * block
    layout = torch.ones((H, nb, nb), dtype=torch.long)
    layout[0, 1] = 0
    idx = layout.nonzero()
    rand = lambda *s: torch.randn(s, generator=g, device='cuda', dtype=dtype)
    s = rand(2, len(idx), block, block)
    d = torch.zeros(2, H, nb, block, nb, block, device='cuda')
    d[:, idx[:, 0], idx[:, 1], :, idx[:, 2]] = s.float().transpose(0, 1)
    d = d.reshape(2, H, n, n)

    def view(rows, cols):
        if where == 'whole':
            return rand(2, H, rows, cols)
        if where == 'transposed':
            return rand(2, H, cols, rows).transpose(2, 3)
        if where == 'unaligned':
            return rand(2 * H * cols * rows + 1)[1:].view(2, H, cols, rows).transpose(2, 3)
        if where == 'odd rows':
            return rand(2, H, cols, rows + 1)[..., :rows].transpose(2, 3)
        if where == 'every other':
            return rand(2, H, 2 * rows, 2 * cols)[:, :, ::2, ::2]
        return rand(1, H, cols, rows).transpose(2, 3).expand(2, -1, -1, -1)
    # FP16 results of FP32 sums: one rounding (2^-11) of values of about sqrt(n); FP32 against TF32-free FP32 sums
    tol = dict(rtol=1e-3, atol=2e-3 * n ** 0.5) if dtype == torch.float16 else dict(rtol=1e-4, atol=1e-4)
    close = lambda got, want: torch.testing.assert_close(got.float(), want, **tol)
    x = view(n, free)
    close(MatMul(layout, block, 'dsd')(s, x), d @ x.float())
    close(MatMul(layout, block, 'dsd', trans_b=True)(s, x.transpose(2, 3)), d @ x.float())
    x = view(free, n)
    close(MatMul(layout, block, 'dds')(x, s), x.float() @ d)
    close(MatMul(layout, block, 'dds', trans_a=True)(x.transpose(2, 3), s), x.float() @ d)


@pytest.mark.gpu
@pytest.mark.parametrize('which', ['rpe', 'key_padding_mask', 'attn_mask'])
@pytest.mark.parametrize('op', ['softmax', 'attention 64', 'attention 96', 'chain'])
def test_biases_that_need_gradients_or_carry_tangents(op, which):
    """With a gradient needed by a bias or a mask alone the result can be differentiated (the bias receives
    nothing); a tangent on it is an error."""
    import torch.autograd.forward_ad as fwd
    make = lambda *s: torch.ones(s, device='cuda', dtype=torch.float16)
    shape = {'rpe': (2, 64, 64), 'key_padding_mask': (1, 64), 'attn_mask': (64, 64)}[which]
    if op == 'softmax':
        call = lambda t: Softmax(LAYOUT, 16)(make(1, 20, 16, 16), **{which: t})
    else:
        D = 96 if op == 'attention 96' else 64
        q = make(1, 2, 64, D)
        call = lambda t: SparseSelfAttention(layout=LAYOUT, block=16, fused=op != 'chain')(q, q, q, **{which: t})
    t = make(*shape).requires_grad_()
    out = call(t)
    assert out.requires_grad
    out.sum().backward()
    assert t.grad is None or not bool(t.grad.any())
    with torch.no_grad():
        assert not call(t).requires_grad
        with fwd.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
            call(fwd.make_dual(make(*shape), make(*shape)))


def test_attributes_changed_between_calls_are_read():
    """MatMul, Softmax and attention objects keep native operations that copy their attributes."""
    def used(obj, *args):
        """The operation `obj` calls (on CPU tensors, which it refuses)."""
        with pytest.raises((RuntimeError, ValueError), match='CUDA tensors only'):
            obj(*args)
        op, = obj._ops.values()
        return op
    mm, x = MatMul(LAYOUT, 16, 'sdd'), torch.zeros(1, 2, 64, 16)
    ops = [used(mm, x, x)]
    assert used(mm, x, x) is ops[0]
    mm.bench = False
    assert used(mm, x, x) is ops[0]                     # (nothing that the operation holds)
    for name, value in (('trans_a', True), ('trans_b', True), ('mode', 'dsd'), ('block', 32)):
        setattr(mm, name, value)
        ops.append(used(mm, x, x))
    assert len(set(map(id, ops))) == 5
    sm, y = Softmax(LAYOUT, 16), torch.zeros(1, 20, 16, 16)
    first = used(sm, y)
    sm.block = 32
    assert used(sm, y) is not first
    q = torch.zeros(1, 2, 64, 64, dtype=torch.float16)
    att = SparseSelfAttention(layout=LAYOUT, block=16)
    with pytest.raises(RuntimeError, match='CUDA tensors only'):
        att(q, q, q)
    first, = att._attn.values()
    att.block = 32                                       # (its tables are those of block 16)
    with pytest.raises((RuntimeError, ValueError), match='does not fit|CUDA tensors only'):
        att(q, q, q)
    second, = att._attn.values()
    assert second is not first and second.block == 32


@pytest.mark.gpu
def test_products_after_an_attribute_changed():
    from torch_blocksparse_b200 import Linear
    g = torch.Generator('cuda').manual_seed(0)
    a = torch.randn((1, 2, 64, 64), generator=g, device='cuda')
    mm = MatMul(LAYOUT, 16, 'sdd')
    plain = mm(a, a)
    mm.trans_b = True
    assert torch.equal(mm(a, a), MatMul(LAYOUT, 16, 'sdd', trans_b=True)(a, a)) and not torch.equal(mm(a, a), plain)
    lin = Linear(64, 64, 16, LAYOUT[0]).cuda()
    x = a[0, 0].requires_grad_()
    w = lin.weight
    for trans in (False, True):
        lin.matmul.trans_b = trans
        y = lin(x)
        want = MatMul(LAYOUT[:1], 16, 'dds', trans_b=trans)(x[None, None], w[None])[0, 0]
        assert torch.equal(y, want)
        for got, ref in zip(torch.autograd.grad(y, (x, w), a[0, 1]), torch.autograd.grad(want, (x, w), a[0, 1])):
            torch.testing.assert_close(got, ref)


def test_objects_saved_before_they_had_native_operations():
    """Whole modules in files of an earlier version have no cache of native operations."""
    from torch_blocksparse_b200 import Linear, MultiheadAttention
    x = torch.zeros(1, 2, 64, 64, dtype=torch.float16)
    att, mha = SparseSelfAttention(layout=LAYOUT, block=16), MultiheadAttention(128, 2, LAYOUT, 16).half()
    with pytest.raises(RuntimeError, match='CUDA tensors only'):
        att(x, x, x)
    for obj, calls in ((MatMul(LAYOUT, 16, 'sdd'), (x, x)), (Softmax(LAYOUT, 16), (torch.zeros(1, 20, 16, 16),)),
                       (Linear(64, 64, 16, LAYOUT[0]), (torch.zeros(3, 64),)), (att, (x, x, x)), (mha, (torch.zeros(64, 1, 128).half(),) * 3)):
        old = copy.deepcopy(obj)
        parts = list(old.modules()) if isinstance(old, torch.nn.Module) else [old]
        parts += [getattr(m, 'matmul') for m in parts if hasattr(m, 'matmul')]
        parts += [o for m in parts for ops in getattr(m, 'ops', {}).values() for o in ops]
        for m in parts:
            m.__dict__.pop('_ops', None)
            m.__dict__.pop('_attn', None)
        with pytest.raises(RuntimeError, match='CUDA tensors only'):
            pickle.loads(pickle.dumps(old))(*calls)


@pytest.mark.parametrize('op,block,Z,heads,nb,density,free,trans,want', [
    # sdd: padded or few tiles, the set-up and the union cost more than the products
    ('sdd', 32, 1, 1, 32, 0.25, 64, 0, 0), ('sdd', 32, 4, 8, 128, 0.25, 32, 0, 0), ('sdd', 64, 1, 1, 16, 0.25, 48, 0, 0),
    ('sdd', 32, 4, 8, 32, 0.5, 320, 0, 1), ('sdd', 32, 4, 8, 32, 0.5, 336, 0, 1), ('sdd', 64, 4, 8, 64, 0.5, 80, 0, 1),
    # whole tiles of several entries and heads, and block 128
    ('sdd', 32, 2, 2, 8, 0.1, 64, 0, 1), ('sdd', 128, 1, 1, 8, 0.1, 16, 0, 1), ('dsd', 32, 2, 2, 8, 0.1, 128, 0, 1),
    # dsd and dds, narrow and wide
    ('dsd', 32, 1, 12, 32, 0.25, 64, 0, 0), ('dsd', 32, 1, 12, 32, 0.25, 320, 1, 1), ('dds', 64, 1, 1, 16, 0.25, 64, 1, 0),
    ('dds', 32, 1, 1, 128, 0.25, 4093, 0, 1), ('dds', 64, 1, 1, 64, 0.5, 2000, 1, 1), ('dsd', 16, 2, 2, 8, 0.5, 128, 0, 0)])
def test_kernel_family_by_size(op, block, Z, heads, nb, density, free, trans, want):
    """The family measured as the faster one at sizes well away from where the two are level."""
    import ctypes
    from torch_blocksparse_b200 import _lib, tables
    g = torch.Generator().manual_seed(0)
    meta = tables.build_meta((torch.rand((heads, nb, nb), generator=g) < density).long())
    got = ctypes.c_int(-1)
    _lib.check(_lib.lib().bsp_matmul_prefers_tcgen05(('sdd', 'dsd', 'dds').index(op), block, Z, free, trans, meta.hdr.data_ptr(),
                                                     ctypes.byref(got)))
    assert got.value == want


def test_kernel_family_arguments():
    import ctypes
    from torch_blocksparse_b200 import _lib, tables
    meta, out, L = tables.build_meta(LAYOUT), ctypes.c_int(-1), _lib.lib()
    for args in ((3, 32, 1, 64, 0, meta.hdr.data_ptr()), (0, 48, 1, 64, 0, meta.hdr.data_ptr()), (0, 32, 1, 0, 0, meta.hdr.data_ptr()),
                 (0, 32, 0, 64, 0, meta.hdr.data_ptr()), (0, 32, 1, 64, 0, None)):
        assert L.bsp_matmul_prefers_tcgen05(*args, ctypes.byref(out)) == _lib.ERR_INVALID
    assert L.bsp_matmul_use_tcgen05(3) == _lib.ERR_INVALID
