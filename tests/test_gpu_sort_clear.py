"""The sort clears the caller's accumulation buffer: every byte of it and no byte beside it, at any alignment."""
import pytest
import torch

from flydsl_b200 import _lib
from flydsl_b200.kernels.moe_sorting_kernel import moe_sorting_flydsl

pytestmark = pytest.mark.gpu
GUARD = 64


# 40 pairs: one block sorts; 10000 pairs: three launches.  16384 bytes is one clearing block's share, 24 MB more than all
# clearing blocks of one pass
@pytest.mark.parametrize("T", [20, 5000])
@pytest.mark.parametrize("size", [1, 7, 15, 16, 17, 16384 + 3, 24 * 1024 * 1024 + 5])
def test_clears_exactly_the_buffer(T, size):
    E, k, U = 8, 2, 16
    ids = torch.stack([torch.arange(T) % E, (torch.arange(T) + 1) % E], 1).to(torch.int32).cuda()
    tw = torch.ones((T, k), device="cuda")
    cap = T * k + E * U - k
    i32 = dict(dtype=torch.int32, device="cuda")
    out = (torch.empty(cap, **i32), torch.empty(cap, device="cuda"), torch.empty((cap + U - 1) // U, **i32), torch.empty(2, **i32))
    for offset in (0, 1, 2, 8, 15):
        raw = torch.full((GUARD + offset + size + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
        lo, hi = GUARD + offset, GUARD + offset + size
        moe_sorting_flydsl(ids, tw, *out, raw[lo:hi], E, U)
        torch.cuda.synchronize()
        assert int(torch.count_nonzero(raw[lo:hi])) == 0, offset
        assert bool((raw[:lo] == 0xA5).all()) and bool((raw[hi:] == 0xA5).all()), offset
    assert _lib.device_status() == 0
