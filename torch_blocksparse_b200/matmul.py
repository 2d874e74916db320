"""Block-sparse matrix multiplication with the reference's Python interface.

Mirrors torch_blocksparse/matmul.py:
  MatMul(layout, block, mode, trans_a=False, trans_b=False, bench=False)   (matmul.py:643-659)
  MatMul.__call__(a, b)                                                    (matmul.py:670-690)
  MatMul.make_lut(dtype, device)                                           (matmul.py:611-641)
  _sparse_matmul: the table builders of the autograd function              (matmul.py:281-458)

mode 'sdd': sparse = op(a) @ op(b);  'dsd': dense = op(a_sparse) @ op(b);
'dds': dense = op(a) @ op(b_sparse).  Dense tensors are [Z, H, rows, cols],
sparse ones [Z, nnz, block, block] in layout.nonzero() order.

All arithmetic runs in the native CUDA library; there is no other code path.  The products, their
gradients and the checks of the operands are in csrc/torch/ops.cpp.
"""
import math

import torch

from . import _lib, tables, tracing
from .tracing import recording

_DTYPES = {torch.float32: _lib.F32, torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}


def _dtype_code(t):
    if t.dtype not in _DTYPES:
        raise ValueError('unsupported dtype %s (float32, float16 and bfloat16 are)' % t.dtype)
    return _DTYPES[t.dtype]


def _stream(t):
    return torch.cuda.current_stream(t.device).cuda_stream


def _require_cuda(*ts):
    for t in ts:
        if not t.is_cuda:
            raise RuntimeError('torch_blocksparse_b200 runs on CUDA tensors only (got a %s tensor)' % t.device)


class _sparse_matmul:
    """Table builders under the names and with the results of the reference's autograd function."""

    @staticmethod
    def make_sdd_lut(layout, block, dtype, device):
        """matmul.py:281-297."""
        return tables.make_sdd_lut(layout, block, device)

    @staticmethod
    def make_dxx_lut(layout, block, step, trans, device, transform=None):
        """matmul.py:372-458 (`transform` other than identity is not supported)."""
        if transform is not None:
            raise NotImplementedError('make_dxx_lut: only the identity transform is supported')
        return tables.make_dxx_lut(layout, block, step, trans, device)


class MatMul(_lib.WithOps):

    _op_attributes = frozenset(('block', 'mode', 'trans_a', 'trans_b'))

    def make_lut(self, dtype, device):
        """The reference-format tables for c, da and db (matmul.py:611-641), cached
        per (dtype, device):
        (c_lut, c_num_locks, c_width, c_packs, da_..., db_...)."""
        key = (dtype, device)
        if key in self.lut_cache:
            return self.lut_cache[key]
        layout, block = self.layout, self.block
        step = 8 if dtype == torch.float32 else 16
        sdd = lambda: tables.make_sdd_lut(layout, block, device)
        dxx = lambda trans: tables.make_dxx_lut(layout, block, step, trans, device)
        if self.mode == 'sdd':
            c, da, db = sdd(), dxx(True), dxx(False)
        elif self.mode == 'dsd':
            c, da, db = dxx(not self.trans_a), sdd(), dxx(self.trans_a)
        else:
            c, da, db = dxx(self.trans_b), dxx(not self.trans_b), sdd()
        self.lut_cache[key] = tuple(c) + tuple(da) + tuple(db)
        return self.lut_cache[key]

    def __init__(self, layout, block, mode, trans_a=False, trans_b=False, bench=False):
        if mode not in ['sdd', 'dsd', 'dds']:
            raise NotImplementedError('Supported modes are: sdd, dsd, dds')
        self.lut_cache = dict()
        self.trans_a = trans_a
        self.trans_b = trans_b
        self.mode = mode
        self.spdims = layout.shape
        self.block = block
        self.layout = layout
        self.bench = bench
        self.time_c = None
        self.time_da = None
        self.time_db = None
        self._meta = None
        self._ops = _lib.OpCache()           # native operation per device index

    @property
    def meta(self):
        """Execution metadata of the layout (built on first use)."""
        if self._meta is None:
            self._meta = tables.build_meta(self.layout)
        return self._meta

    def _op(self, device):
        """The native operation with this object's tables on `device`."""
        ops, meta = self._ops, self.meta
        op = _lib.ops().MatMulOp(meta.hdr, meta.on(device), self.block, self.mode, self.trans_a, self.trans_b)
        ops[-1 if device.index is None else device.index] = op
        return op

    def __call__(self, a, b):
        op = self._ops.get(a.get_device()) or self._op(a.device)
        if recording() is not None:
            return tracing.call(op, '__call__', a, b)
        if not self.bench:
            return op(a, b)
        times = _lib.ops().Times()
        c = op(a, b, times)
        self.time_c, self.time_da, self.time_db = times.c, None, None
        return c


class Linear(torch.nn.Module):
    """y = x . W with a block-sparse weight (torch_blocksparse/matmul.py:693-709).

    The reference's class cannot be constructed: it calls MatMul with its
    arguments in the wrong order (matmul.py:702).  This is the layer it
    describes: `weight` holds the nonzero blocks of an [in_features,
    out_features] matrix as [nnz, block, block] (Kaiming-uniform, as the
    reference initialises it), `layout` is [in_features / block, out_features /
    block] (a leading singleton head dimension is accepted), and forward is the
    'dds' product.  Inputs of any rank [..., in_features] are flattened to rows.
    There is no bias, as in the reference.
    """

    def __init__(self, in_features, out_features, block, layout, bench=False):
        super().__init__()
        if layout.dim() == 2:
            layout = layout.unsqueeze(0)
        if layout.dim() != 3 or layout.size(0) != 1:
            raise ValueError('Linear: layout must be [in_features / block, out_features / block]')
        if in_features % block or out_features % block:
            raise ValueError('Linear: in_features and out_features must be multiples of block %d' % block)
        if tuple(layout.shape[1:]) != (in_features // block, out_features // block):
            raise ValueError('Linear: layout %s does not fit %d x %d features with block %d'
                             % (tuple(layout.shape[1:]), in_features, out_features, block))
        self.in_features = in_features
        self.out_features = out_features
        self.block = block
        self.weight = torch.nn.Parameter(torch.empty(int(layout.sum()), block, block))
        self.reset_parameters()
        self.matmul = MatMul(layout, block, 'dds', trans_a=False, trans_b=False, bench=bench)

    def reset_parameters(self):
        torch.nn.init.kaiming_uniform_(self.weight, a=math.sqrt(5))

    def forward(self, input):
        if input.size(-1) != self.in_features:
            raise ValueError('Linear: expected %d input features, got %d' % (self.in_features, input.size(-1)))
        mm = self.matmul
        op = mm._ops.get(input.get_device()) or mm._op(input.device)
        if recording() is not None:
            return tracing.call(op, 'linear', input, self.weight, None)
        times = _lib.ops().Times() if mm.bench else None
        y = op.linear(input, self.weight, times)
        if times is not None:
            mm.time_c = times.c
        return y
