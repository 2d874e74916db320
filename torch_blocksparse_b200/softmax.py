"""Block-sparse softmax with the reference's Python interface.

Mirrors torch_blocksparse/softmax.py:
  Softmax(layout, block, bench=False)                                  (softmax.py:338-343)
  Softmax.__call__(x, scale=1., rpe=None, key_padding_mask=None, attn_mask=None,
                   key_padding_mask_mode='add', attn_mask_mode='add')  (softmax.py:345-361)
  _sparse_softmax: the table builder of the autograd function          (softmax.py:201-221)

Semantics kept from the reference: the result overwrites `x` and `x` itself
is returned (softmax.py:301,313); the backward overwrites the incoming
gradient and returns it (softmax.py:325-326); rpe and the masks receive no
gradient; masks in 'mul' mode turn 0 into -inf and anything else into 0.
rpe is addressed as [Z, H, M, N] (softmax.py:50-55); a 3-D [H, M, N] tensor is
accepted as well and broadcast over the batch.  The checks, the autograd
function and the launches are in csrc/torch/ops.cpp.
"""
import torch

from . import _lib, tables
from .tracing import recording


class _sparse_softmax:

    @staticmethod
    def make_lut(layout, block, device):
        """softmax.py:201-221: returns (lut, maxlut).  A layout in device memory gets its table
        there (from the metadata built on the device), without a copy to the host."""
        if layout.is_cuda and torch.device(device).type == 'cuda':
            return tables.make_softmax_lut_device(layout, device)
        return tables.make_softmax_lut(layout, device)


class Softmax(_lib.WithOps):

    _op_attributes = frozenset(('block', 'spdims'))

    def make_lut(self, device):
        """Table cache per device (softmax.py:332-336)."""
        key = (device, )
        if key not in self.lut_cache:
            # (one table per layout content and device for the whole process: ops on the same layout share it)
            self.lut_cache[key] = tables._cached('softmax_lut', self.layout, (str(device),),
                                                 lambda: _sparse_softmax.make_lut(self.layout, self.block, device))
        return self.lut_cache[key]

    def __init__(self, layout, block, bench=False):
        self.spdims = layout.shape
        self.layout = layout
        self.block = block
        self.bench = bench
        self.lut_cache = dict()
        self.time_y = None
        self._ops = _lib.OpCache()           # native operation per device index

    def _op(self, device):
        """The native operation with this object's table on `device`."""
        ops = self._ops
        lut, maxlut = self.make_lut(device)
        op = _lib.ops().SoftmaxOp(lut, maxlut, *self.spdims, self.block)
        ops[-1 if device.index is None else device.index] = op
        return op

    def __call__(self, x, scale=1., rpe=None, key_padding_mask=None, attn_mask=None,
                 key_padding_mask_mode='add', attn_mask_mode='add'):
        if recording() is not None:
            raise RuntimeError('Softmax works in place, which torch.jit.trace cannot replay')
        op = self._ops.get(x.get_device()) or self._op(x.device)
        times = _lib.ops().Times() if self.bench else None
        x = op(x, scale, rpe, key_padding_mask, attn_mask, key_padding_mask_mode, attn_mask_mode, times)
        if times is not None:
            self.time_y = times.c
        return x
