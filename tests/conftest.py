import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line('markers', 'gpu: needs a CUDA device (run with -m gpu on a B200)')


def pytest_collection_modifyitems(config, items):
    import torch
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason='no CUDA device')
    for item in items:
        if 'gpu' in item.keywords:
            item.add_marker(skip)


@pytest.fixture(params=[1, 2], ids=['by size', 'tcgen05'])
def product_family(request):
    """MatMul on the kernels its size speaks for, and on tcgen05 wherever they cover it."""
    from torch_blocksparse_b200 import _lib
    _lib.check(_lib.lib().bsp_matmul_use_tcgen05(request.param))
    yield request.param
    _lib.check(_lib.lib().bsp_matmul_use_tcgen05(1))
