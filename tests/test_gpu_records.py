"""The bulk record kernels at the edges of their 32-record groups: values
stored into grouped storage, appended behind a partly filled group, words and
state read back in particle order and the per-slot statistics, against
aq_encode's and aq_decode's contiguous records (codes and values equal bit
for bit, whole numbers both) and numpy sums (1e-12: FP64 sums in another
order)."""
import ctypes as C

import numpy as np
import pytest

from autoquantizer_b200 import _lib, scenes
from autoquantizer_b200.mpm_solver import MPMSolver
from test_gpu_codec import gpu_decode, gpu_encode

pytestmark = pytest.mark.gpu


def _cfg(kind, n):
    if kind == "2d_fluid":
        return scenes.dam_break_2d(n=n, n_grid=64)[0]
    if kind == "2d_raw":
        cfg = scenes.elastic_block_2d(n=4, n_grid=64)[0]
        cfg.n_particles = n
        return cfg
    return scenes.mixed_boxes_3d(n=n, n_grid=32, quantized=kind != "3d_raw",
                                 precision="f64" if kind == "3d_raw64" else "f32")[0]


@pytest.mark.parametrize("n,more", [(1, 1), (31, 2), (32, 33), (33, 64), (100, 7)])
@pytest.mark.parametrize("kind", ["2d_fluid", "2d_raw", "3d_quant", "3d_raw"])
def test_store_append_fetch(kind, n, more):
    import torch

    cfg = _cfg(kind, n + more)
    s = MPMSolver(cfg)
    ns = s.n_slots()
    rng = np.random.default_rng(n)
    vals = rng.normal(0.4, 0.2, (n + more, ns)).astype(np.float32)
    if s.has_mat:
        vals[:, -1] = rng.integers(0, 4, n + more)
    s.set_particles(torch.from_numpy(vals[:n]).cuda())
    L = s.layout()
    want = gpu_encode(L, vals, seed=int(cfg.seed), step=-1, f64=False)
    assert np.array_equal(s.words(), want[:n])
    t = torch.from_numpy(vals[n:]).cuda()
    _lib.check(_lib.lib().aq_sim_append(s._sim, C.c_void_p(t.data_ptr()), 0, more, _lib.stream_ptr()))
    s.current_idx = n + more
    assert np.array_equal(s.words(), want)
    for f64 in (False, True):
        assert np.array_equal(s.state_values(f64), gpu_decode(L, want, f64))
    # records in, in another order of storage after a substep's binning, and out again
    s.set_words(want)
    assert np.array_equal(s.words(), want)
    state = s.state_values(True)
    for ref in (None, torch.from_numpy(vals).cuda(), torch.from_numpy(vals.astype(np.float64)).cuda()):
        st = s.field_stats(reference=ref)
        cols = [np.abs(state).sum(0), state.sum(0), (state ** 2).sum(0)]
        if ref is not None:
            cols.append(np.abs(state - vals.astype(np.float64)).sum(0))
        for k, c in zip((0, 1, 2, 4), cols):
            assert np.all(np.abs(st[:, k] - c) <= 1e-12 * np.maximum(1.0, np.abs(state).sum(0) + (state ** 2).sum(0)))
        assert np.array_equal(st[:, 3], np.abs(state).max(0))


@pytest.mark.parametrize("n,ns", [(1, 1), (3, 25), (257, 24), (40, 300), (5, 1024)])
def test_state_error_shapes(n, ns):
    import torch

    rng = np.random.default_rng(ns)
    a, b = rng.normal(size=(n, ns)), rng.normal(size=(n, ns)).astype(np.float32)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    sq, mx = (C.c_double * ns)(), (C.c_double * ns)()
    _lib.check(_lib.lib().aq_state_error(C.c_void_p(ta.data_ptr()), 1, C.c_void_p(tb.data_ptr()), 0, n, ns, sq, mx,
                                         _lib.stream_ptr()))
    d = np.abs(a - b)
    assert np.allclose(np.array(sq[:]), (d * d).sum(0), rtol=1e-12, atol=0)
    assert np.array_equal(np.array(mx[:]), d.max(0))
