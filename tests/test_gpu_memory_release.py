"""What a destroyed simulator held goes back to the device: all but 1 GiB at
once, and that too after release_memory.  64 MB are left for the pool's own
granularity and for what other code of the process maps meanwhile."""
import gc

import pytest

import autoquantizer_b200 as aq
from autoquantizer_b200 import scenes
from autoquantizer_b200.mpm_solver import MPMSolver

pytestmark = pytest.mark.gpu

MB, GB = 1 << 20, 1 << 30


def test_memory_of_a_destroyed_simulator():
    import torch

    def free():
        return torch.cuda.mem_get_info()[0]

    def solver():
        # three 268 MB grids, and 4 million records twice with their scratch
        cfg, vals = scenes.falling_block_3d(n=1000, n_grid=256)
        cfg.n_particles = 4_000_000
        s = MPMSolver(cfg)
        s.set_particles(vals)
        s.substeps(1)
        torch.cuda.synchronize()
        return s

    solver()._drop_sim()  # kernels compiled and loaded
    gc.collect()  # nothing of earlier tests is freed meanwhile
    torch.cuda.empty_cache()
    aq.release_memory()
    before = free()
    s = solver()
    assert before - free() > 1.5 * GB
    s._drop_sim()
    torch.cuda.empty_cache()
    assert before - free() < GB + 64 * MB
    aq.release_memory()
    assert before - free() < 64 * MB


def test_streamed_simulator_holds_two_grids():
    import torch

    from autoquantizer_b200.streamed import StreamedSolver

    cfg, vals = scenes.falling_block_3d(n=1000, n_grid=256)
    s = MPMSolver(cfg)
    s.set_particles(vals)
    StreamedSolver(s, 1000).close()  # kernels compiled and loaded
    gc.collect()  # nothing of earlier tests is freed meanwhile
    torch.cuda.empty_cache()
    aq.release_memory()
    before = torch.cuda.mem_get_info()[0]
    st = StreamedSolver(s, 1000)
    held = before - torch.cuda.mem_get_info()[0]
    st.close()
    grid = 16 * 256 ** 3
    cells = 2 * 4 * 256 ** 3  # per-cell counts and offsets of the binning
    assert 2 * grid <= held < 2 * grid + cells + 64 * MB, held
