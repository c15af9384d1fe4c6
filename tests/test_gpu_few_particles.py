"""Few particles on a large grid must not take longer than many: the passes
clear a grid as they go, with more thread blocks than the particles need.
Three times the time of 1,000 (adjoint: 2,000) particles on the same grid is
allowed; median of nine calls."""
import numpy as np
import pytest

from autoquantizer_b200 import scenes
from autoquantizer_b200.adjoint import Adjoint, ek_seed
from autoquantizer_b200.mpm_solver import MPMSolver

pytestmark = pytest.mark.gpu


def _median_ms(f):
    import torch

    for _ in range(3):
        f()
    ts = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        b.synchronize()
        ts.append(a.elapsed_time(b))
    return float(np.median(ts))


def _substeps_ms(n, n_grid):
    cfg, vals = scenes.falling_block_3d(n=n, n_grid=n_grid)
    cfg.dt = 1e-5
    s = MPMSolver(cfg)
    s.set_particles(vals)
    return _median_ms(lambda: s.substeps(16))


@pytest.mark.parametrize("n,n_grid", [(1, 128), (64, 256)])
def test_substeps(n, n_grid):
    few, many = _substeps_ms(n, n_grid), _substeps_ms(1000, n_grid)
    assert few <= 3 * many, (few, many)


def _adjoint_ms(n, n_grid):
    import torch

    cfg, vals = scenes.falling_block_3d(n=n, n_grid=n_grid)
    cfg.dt = 1e-5
    s = MPMSolver(cfg)
    s.set_particles(vals)
    adj = Adjoint(s._params())
    s0 = torch.from_numpy(np.ascontiguousarray(vals[:, :s.n_slots()])).cuda().float()

    def run():
        sT = adj.forward(s0, 8, 8)
        adj.backward(ek_seed(sT, 3, s.p_mass, s.g))

    ms = _median_ms(run)
    adj.close()
    return ms


def test_adjoint():
    few, many = _adjoint_ms(64, 128), _adjoint_ms(2000, 128)
    assert few <= 3 * many, (few, many)
