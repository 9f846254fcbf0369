"""The grid build either side of the sizes where its passes take more entries per thread
and count their tiles in a kernel of their own, and of a block's and a trip's entries;
order and offsets must equal the oracle's."""
import ctypes

import numpy as np
import pytest

import oracle as O
from twoscalesplit_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


@pytest.mark.parametrize("n,dims", [(1, (1, 1)), (255, (3, 5)), (257, (64, 33)), (1025, (2048, 1)), (149999, (400, 371)),
                                    (150000, (45, 46)), (150001, (400, 371)), (152577, (2049, 97)), (623617, (1, 7))])
def test_build_sizes(n, dims):
    import torch
    rng = np.random.default_rng(n)
    cell = 0.25
    pos = (rng.uniform(-0.1, 1.1, size=(n, 2)) * np.array(dims) * cell).astype(np.float32)
    ids = rng.permutation(3 * n)[:n].astype(np.int32)
    lib = _abi.load_library()
    ws = ctypes.c_size_t(0)
    assert lib.tss_grid_workspace_size(n, *dims, ctypes.byref(ws)) == 0
    p, i = torch.from_numpy(pos).cuda(), torch.from_numpy(ids).cuda()
    order = torch.empty(n, dtype=torch.int32, device="cuda")
    off = torch.empty(dims[0] * dims[1] + 1, dtype=torch.int32, device="cuda")
    work = torch.full((ws.value,), 0x5a, dtype=torch.uint8, device="cuda")  # nothing in it is zero beforehand
    o_order, o_off = O.grid(pos, ids, (0.0, 0.0), cell, dims)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for _ in range(2):  # and on the workspace as the first build left it
        order.fill_(-1)
        off.fill_(-1)
        assert lib.tss_grid_build(ptr(p), ptr(i), n, 0.0, 0.0, cell, *dims, ptr(order), ptr(off), ptr(work), ws.value,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert np.array_equal(order.cpu().numpy(), o_order)
        assert np.array_equal(off.cpu().numpy(), o_off)
