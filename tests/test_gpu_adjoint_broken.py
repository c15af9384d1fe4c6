"""A backward pass that ends with an error (here: queued on a stream that is
being captured, where its wait is not permitted, so nothing of it runs) leaves
the next run right, to 1e-9 of the run before (f64, atomic sums in different
orders)."""
import ctypes as C

import numpy as np
import pytest

from autoquantizer_b200 import _lib, scenes
from autoquantizer_b200.adjoint import ek_seed
from test_gpu_adjoint import _setup

pytestmark = pytest.mark.gpu


def test_run_after_a_broken_backward_pass():
    import torch

    cfg, vals = scenes.falling_block_3d(n=500, n_grid=16)
    s, adj, s0 = _setup(cfg, vals)
    T = 4

    def run():
        sT = adj.forward(s0, T, 4)
        seed = ek_seed(sT, 3, s.p_mass, s.g)
        g0, sens = adj.backward(seed)
        return [sT.cpu().numpy(), g0.cpu().numpy(), sens], seed

    first, seed = run()
    g0 = torch.empty_like(seed)
    sens = (C.c_double * s.n_slots())()
    rt = C.CDLL("libcudart.so.12")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle, graph = C.c_void_p(st.cuda_stream), C.c_void_p()
    assert rt.cudaStreamBeginCapture(handle, 2) == 0  # relaxed: this stream only
    rc = _lib.lib().aq_adjoint_backward(adj._h, C.c_void_p(seed.data_ptr()), C.c_void_p(g0.data_ptr()), sens, handle)
    rt.cudaStreamEndCapture(handle, C.byref(graph))
    rt.cudaGetLastError()
    assert rc == -3
    again, _ = run()
    for a, b in zip(first, again):
        assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a))
    adj.close()
