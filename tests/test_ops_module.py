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
