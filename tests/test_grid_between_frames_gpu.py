"""The grid between two frames: its output fields are those of the last output
step, zero where that step had no nodes, whatever ran in this memory before."""
import numpy as np
import pytest

import slab
from test_blocks import CFG, DX, Z, _release

pytestmark = pytest.mark.gpu


def _context(prec):
    s = slab.Slab(Z, DX)
    s.set_params(dict(CFG, output_dt=5.0, total_time=20.0), prec)
    return s


def _wide(s):
    """A run that leaves output fields over a large part of the terrain."""
    s.upload_release(_release(24.0))
    s.initial_pass()
    s.advance_to_frame()


def _between(s):
    """4.5 s of steps without output after the t = 0 pass: the flow reaches tiles that it was not in."""
    s.upload_release(_release(16.0))
    s.initial_pass()
    before = s.grid()
    assert s.advance_steps(450) == 450
    after = s.grid()
    assert after["i_off"] + after["Nx"] > before["i_off"] + before["Nx"] + 4  # nodes: the front has moved on
    return after


@pytest.mark.parametrize("prec", [slab.FP32_SPLIT, slab.FP64_PLAIN])
def test_grid_between_frames_after_another_run(prec):
    s = _context(prec)
    _wide(s)
    used = _between(s)  # the same engine
    s.close()
    s = _context(prec)
    _wide(s)
    s.close()
    s = _context(prec)  # a new one in the memory of the last
    new = _between(s)
    s.close()
    for g in (used, new):
        m = g["mass"]
        assert (m > 0).any() and (m == 0).any()
        # where the t = 0 pass had no nodes every output field is zero
        front = np.arange(g["Nx"]) * DX + g["i_off"] * DX > 60.0 + 16.0 + 3 * DX
        assert front.any()
        for k in ("h", "mass", "vz", "F", "a"):
            assert not g[k][front].any(), k
    for k in used:
        assert np.allclose(used[k], new[k], rtol=1e-9, atol=1e-12), k
