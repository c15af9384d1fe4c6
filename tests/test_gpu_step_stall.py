"""A substep launch that gives up waiting for its own blocks (here because the
wait's limit is one cycle) is an error wherever the state is used, and the
state set anew runs on from clean grids."""
import ctypes as C

import numpy as np
import pytest

from autoquantizer_b200 import _lib, scenes
from helpers import compare_states, twin

pytestmark = pytest.mark.gpu


def test_stalled_launch_is_an_error_until_the_state_is_set():
    import torch

    cfg, vals = scenes.falling_block_3d(n=5000, n_grid=32)
    cfg.precision = "f64"
    s, o = twin(cfg, vals)
    L = _lib.lib()
    assert L.aq_sim_wait_limit(s._sim, 0) == -1
    words = s.words()
    s.substeps(3)
    o.substeps(3)
    compare_states(s, o, 1e-8)  # the default limit is not reached
    _lib.check(L.aq_sim_wait_limit(s._sim, 1))
    s.substeps(5)
    torch.cuda.synchronize()
    ns, d = s.n_slots(), C.c_double
    assert L.aq_sim_check(s._sim) == -7
    assert s.status()[0] & _lib.AQ_ST_STALLED
    out = torch.empty((5000, 32), dtype=torch.float64, device="cuda")
    p = C.c_void_p(out.data_ptr())
    assert L.aq_sim_substeps(s._sim, 1, _lib.stream_ptr()) == -7
    assert L.aq_sim_get_state(s._sim, p, 1, _lib.stream_ptr()) == -7
    assert L.aq_sim_get_words(s._sim, p, _lib.stream_ptr()) == -7
    assert L.aq_sim_grid_mass(s._sim, p, _lib.stream_ptr()) == -7
    assert L.aq_sim_loss(s._sim, 0, C.byref(d()), _lib.stream_ptr()) == -7
    assert L.aq_sim_field_stats(s._sim, None, 0, (d * (5 * ns))(), _lib.stream_ptr()) == -7
    for read in (s.state_values, s.words, s.compute_loss, s.field_stats):
        with pytest.raises(_lib.AqError):
            read()
    _lib.check(L.aq_sim_wait_limit(s._sim, 1 << 34))
    s.set_words(words)
    o.set_words(words)
    assert L.aq_sim_check(s._sim) == 0 and not s.status()[0] & _lib.AQ_ST_STALLED
    s.substeps(5)
    o.substeps(5)
    compare_states(s, o, 1e-8)


def test_stall_found_by_the_read_that_waits_for_it():
    cfg, vals = scenes.falling_block_3d(n=5000, n_grid=32)
    s, _ = twin(cfg, vals)
    _lib.check(_lib.lib().aq_sim_wait_limit(s._sim, 1))
    s.substeps(5)
    with pytest.raises(_lib.AqError):
        s.state_values()
    s.set_particles(np.asarray(vals))
    s.substeps(5)
    assert np.isfinite(s.state_values()).all()
