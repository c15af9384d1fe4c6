"""aq_mlp_backward refuses layer sizes below one before it touches the device,
as aq_mlp_forward does: zero is a multiple of every tile size, so such sizes
would pass the whole-network kernels' rule and write nothing or, negative, out
of bounds."""
import ctypes as C

import pytest

from autoquantizer_b200 import _lib


@pytest.mark.parametrize("dims", [(0, 64, 12), (64, 0, 12), (64, 64, 0), (-64, 64, 12), (64, -64, 12)])
def test_sizes_below_one(dims):
    p = C.c_void_p(256)  # never read
    L = _lib.lib()
    assert L.aq_mlp_backward(*dims, p, p, 1, p, p, p, None) == -1
    assert L.aq_mlp_forward(*dims, p, p, p, 1, p, p, None) == -1
