"""The whole-network kernels and the layer-by-layer ones over sizes on both
sides of their rule and of their tiles (16 rows, 64 columns of k, 256-row
segments of the batch), against the numpy oracle: 2e-3 relative to the
largest value, the bf16 bound of test_gpu_mlp.py."""
import ctypes as C

import numpy as np
import pytest

import mlp_oracle as MO
from autoquantizer_b200 import surrogate as SG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 15, 17, 256, 257, 1000])
@pytest.mark.parametrize("dims", [(64, 128, 12), (64, 64, 1), (128, 192, 70), (64, 512, 3), (48, 128, 12),
                                  (64, 100, 5), (64, 64, 129)])
def test_forward_and_gradient(dims, B):
    m = SG.MLP(1, *dims)
    p = m.p.cpu().numpy()
    rng = np.random.default_rng(B)
    x = rng.normal(size=(B, dims[0])).astype(np.float32)
    dy = rng.normal(size=(B, dims[2])).astype(np.float32)
    y, yo = m.forward_raw(x).cpu().numpy(), MO.forward(p, x, dims)[0]
    assert np.max(np.abs(y - yo)) < 2e-3 * max(1.0, np.abs(yo).max())
    g, go = m.grad_raw(x, dy).cpu().numpy(), MO.backward(p, x, dy, dims)
    assert np.max(np.abs(g - go)) < 2e-3 * np.abs(go).max()


def test_inference_without_saved_activations():
    import torch
    from autoquantizer_b200 import _lib

    m = SG.MLP(seed=2)
    x = torch.randn(33, SG.N_IN, device="cuda")
    y = torch.empty(33, SG.N_OUT, device="cuda")
    _lib.check(_lib.lib().aq_mlp_forward(*m.dims, C.c_void_p(m.p.data_ptr()), C.c_void_p(m.pb.data_ptr()),
                                         C.c_void_p(x.data_ptr()), 33, C.c_void_p(y.data_ptr()), None,
                                         _lib.stream_ptr()))
    assert torch.equal(y, m.forward_raw(x))
