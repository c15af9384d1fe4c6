"""Work items and pass chains of the fused substep at their edges, against
the oracle from the same records (compare_states: 2e-5 relative for f32
state, 1e-8 for f64, plus one quantization step).

  items   a block's records in one part, in equal parts, with a remainder:
          counts around one unit (32) and one item (64), and a crowded cell
          block split over many CTAs
  passes  chains longer than one launch makes (AQ_PASS_MAX), whose last
          launch holds one pass, and chains continued by later calls
  grids   a grid too large for a third copy: one pass a launch, cleared by
          a memset
"""
import numpy as np
import pytest

from autoquantizer_b200 import scenes
from helpers import compare_states, twin

pytestmark = pytest.mark.gpu


def _scene(dim, n, quantized):
    if dim == 2:
        if quantized:
            return scenes.dam_break_2d(n=n, n_grid=64)
        cfg, vals = scenes.elastic_block_2d(n=int(np.ceil(np.sqrt(n))) ** 2, n_grid=64)
        cfg.n_particles = n
        return cfg, vals[:n]
    return scenes.mixed_boxes_3d(n=n, n_grid=32, quantized=quantized)


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 4099])
@pytest.mark.parametrize("dim,quantized", [(2, False), (2, True), (3, False), (3, True)])
def test_item_sizes_match_oracle(dim, quantized, n):
    cfg, vals = _scene(dim, n, quantized)
    s, o = twin(cfg, vals)
    for k in (1, 2):
        s.substeps(k)
        o.substeps(k)
        compare_states(s, o, 2e-5)
        o.set_words(s.words())
    assert s.status()[0] == o.flags == 0


def test_crowded_block_is_split_over_items():
    # 20,000 particles in two cell blocks: over a hundred items of one block
    cfg, vals = scenes.falling_block_3d(n=20000, n_grid=32)
    rng = np.random.default_rng(3)
    vals[:, :3] = 0.5 + rng.random((20000, 3)) * np.array([4.0, 4.0, 8.0]) / 32
    cfg.precision = "f64"
    s, o = twin(cfg, vals)
    s.substeps(3)
    o.substeps(3)
    compare_states(s, o, 1e-8)


@pytest.mark.parametrize("calls", [(17,), (34,), (16, 1, 3), (40,)])
def test_pass_chains_match_oracle(calls):
    cfg, vals = scenes.falling_block_3d(n=5000, n_grid=32)
    cfg.precision = "f64"
    cfg.sort_interval = 36
    s, o = twin(cfg, vals)
    for k in calls:
        s.substeps(k)
        o.substeps(k)
    assert s.step_count() == sum(calls)
    compare_states(s, o, 1e-8)
    assert s.status()[0] == 0


def test_grid_without_a_third_copy_matches_oracle():
    cfg, vals = scenes.elastic_block_2d(n=1024, n_grid=3000)  # 288 MB of f64 nodes
    cfg.precision = "f64"
    cfg.dt = 1e-6
    s, o = twin(cfg, vals)
    s.substeps(3)
    o.substeps(3)
    compare_states(s, o, 1e-8)
