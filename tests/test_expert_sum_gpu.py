"""The sum of a token's expert rows without a residual: the bits of a sum in the order of k, for whole and ragged rows, and refusals."""
import ctypes as C

import pytest
import torch

from atoma_infer_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,top,width,offset", [(1, 1, 4, 0), (3, 4, 1024, 0), (5, 5, 1028, 0), (2, 9, 4096, 0), (7, 6, 1027, 0), (4, 3, 64, 1), (1, 64, 33, 0)])
def test_rows_in_order(dtype, T, top, width, offset):
    """offset: rows that do not start on 16 bytes, which are taken value by value."""
    g = torch.Generator().manual_seed(T + top + width)
    n = T * top + 3
    flat = torch.randn(n * width + offset, generator=g).to(dtype).to(DEV)
    rows = flat[offset:].view(n, width)
    place = torch.randperm(n, generator=g)[:T * top].to(torch.int32).to(DEV)
    out = torch.full((T + 1, width), 7.0, device=DEV)
    L = _lib.lib()
    L.atoma_expert_rows_sum(C.c_void_p(rows.data_ptr()), C.c_void_p(place.data_ptr()), C.c_void_p(out.data_ptr()), T, top, width, 1 if dtype == torch.bfloat16 else 2, None)
    torch.cuda.synchronize()
    picked = rows[place.long()].float().view(T, top, width)
    want = torch.zeros(T, width, device=DEV)
    for k in range(top):
        want = want + picked[:, k]
    assert torch.equal(out[:T], want) and bool((out[T] == 7.0).all())


def test_refusals():
    L = _lib.lib()
    x = torch.zeros(64, device=DEV)
    p = C.c_void_p(x.data_ptr())
    for args in ((None, p, p, 1, 1, 4, 2), (p, p, p, 1, 65, 4, 2), (p, p, p, 1, 0, 4, 2), (p, p, p, 1, 1, 1 << 20, 2), (p, p, p, 1, 1, 4, 7)):
        L.atoma_expert_rows_sum(*args, None)
        assert L.atoma_last_status() != 0, args
