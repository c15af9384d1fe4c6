"""The adjoint's warp tiles and segment buffers at their edges, in f64.

  tiles     particles so far apart that a warp's box of nodes does not fit
            its tile (gathered from and scattered to the grid directly), and
            particle counts around a warp's 32: the forward state against
            MPMSolver's substeps and the gradient against central differences
            (_fd_check's tolerances)
  segments  every split of a run into checkpoint segments, the last one kept
            from the forward pass, against bisection checkpointing, and a
            second backward pass of the same run: 1e-9 relative (atomic sums
            in different orders)
"""
import numpy as np
import pytest

from autoquantizer_b200 import scenes
from autoquantizer_b200.adjoint import ek_seed
from test_gpu_adjoint import _fd_check, _setup

pytestmark = pytest.mark.gpu


def _forward_matches_solver(cfg, vals, T):
    s, adj, s0 = _setup(cfg, vals)
    sT = adj.forward(s0, T, 2).cpu().numpy()
    adj.close()
    s.substeps(T)
    ref = s.state_values()
    scale = np.maximum(1.0, np.abs(ref).max(0))
    assert np.max(np.abs(sT - ref) / scale) < 1e-9


def _spread(cfg, vals, lo, hi):
    """The scene's particles moved to independent uniform positions, with a
    small random velocity so that no velocity component is exactly zero."""
    rng = np.random.default_rng(11)
    d, n = cfg.dim, vals.shape[0]
    vals[:, :d] = lo + (hi - lo) * rng.random((n, d))
    vals[:, d:2 * d] = rng.normal(size=(n, d))
    return cfg, vals


@pytest.mark.parametrize("dim", [2, 3])
def test_boxes_beyond_the_tile(dim):
    make = (lambda: scenes.elastic_block_2d(n=400, n_grid=64)) if dim == 2 else \
        (lambda: scenes.falling_block_3d(n=300, n_grid=48))
    _forward_matches_solver(*_spread(*make(), 0.15, 0.85), T=3)
    cfg, vals = _spread(*make(), 0.15, 0.85)
    cfg.dt = 2e-5
    _fd_check(cfg, vals, T=4, every=2)


@pytest.mark.parametrize("n", [1, 31, 33, 65])
@pytest.mark.parametrize("dim", [2, 3])
def test_particle_counts(dim, n):
    if dim == 2:
        cfg, vals = scenes.elastic_block_2d(n=81, n_grid=32)
        cfg.n_particles = n
        vals = vals[:n]
    else:
        cfg, vals = scenes.falling_block_3d(n=n, n_grid=16)
    cfg, vals = _spread(cfg, vals, 0.45, 0.6)
    _forward_matches_solver(cfg, vals.copy(), T=3)
    cfg.dt = 2e-5
    _fd_check(cfg, vals, T=5, every=2)


@pytest.mark.parametrize("T,every", [(1, 1), (5, 1), (6, 3), (7, 3), (4, 9), (16, 16)])
def test_segments_match_bisection(T, every):
    cfg, vals = scenes.falling_block_3d(n=500, n_grid=16)
    cfg, vals = _spread(cfg, vals, 0.4, 0.65)
    s, adj, s0 = _setup(cfg, vals)

    def run(e):
        sT = adj.forward(s0, T, e)
        g = adj.backward(ek_seed(sT, 3, s.p_mass, s.g))
        again = adj.backward(ek_seed(sT, 3, s.p_mass, s.g))
        for a, b in ((g[0].cpu().numpy(), again[0].cpu().numpy()), (g[1], again[1])):
            assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a)) + 1e-300
        return sT.cpu().numpy(), g[0].cpu().numpy(), g[1]

    for a, b in zip(run(every), run(0)):
        assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a)) + 1e-300
