"""Substeps captured into a CUDA graph: every replay advances the state as the
same call made directly, and a direct call after replays goes on from there.

One capture holds two re-binnings (so the record buffers are back in their
places at its end) and two chains whose substeps add up to no multiple of
three (the grids rotate through three roles).  In f64: 1e-9 relative to the
largest value of a slot, for atomic sums in different orders."""
import numpy as np
import pytest

from autoquantizer_b200 import scenes
from autoquantizer_b200.mpm_solver import MPMSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_grid", [(4900, 128),     # several passes a launch
                                      (112896, 512),   # one pass a launch
                                      (1024, 3000)])   # two grids, cleared by a memset
def test_replays_match_direct_calls(n, n_grid):
    import torch

    def solver():
        cfg, vals = scenes.elastic_block_2d(n=n, n_grid=n_grid)
        cfg.precision = "f64"
        cfg.sort_interval = 4
        cfg.dt = 2e-5 if n_grid < 3000 else 1e-6
        s = MPMSolver(cfg)
        s.set_particles(vals)
        s.substeps(8)  # the next call re-bins first
        return s

    a, b = solver(), solver()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.substeps(8)
    for _ in range(4):
        g.replay()
    a.substeps(8)
    b.substeps(40)
    x, y = a.state_values(), b.state_values()
    scale = np.maximum(1.0, np.abs(y).max(0))
    assert np.max(np.abs(x - y) / scale) < 1e-9
    assert a.status()[0] == b.status()[0] == 0
