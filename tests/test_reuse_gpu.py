"""A context that uploads again runs on the path, step graphs and buffers of the
run before: its results, launch counts and error behaviour are a new
context's, whatever the sizes of the runs before it."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu

N, DX = 96, 2.0
CFG = dict(gravity=9.81, rho=300.0, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=0.25, total_time=5.0, friction="VOELLMY",
           voellmy_mu=0.2, voellmy_xi=1000.0)
I = np.arange(N)
Z = -0.4 * I[:, None] * DX + 0.3 * np.sin(0.3 * I)[None, :]


def _release(r, h0):
    return {"type": "ELLIPSE", "center": (60.0, 96.0), "rx": r, "ry": 0.7 * r, "rotation_deg": 20.0, "h0": h0}


def _run(s, rel, frames):
    s.upload_release(rel)
    s.initial_pass()
    for _ in range(frames):
        s.advance_to_frame()
    P, (hm, vm) = s.particles(), s.max_maps()
    return [P[k] for k in ("x", "v", "vz", "h", "A", "mass", "z")] + [hm, vm], s.state(), s.kernel_launches()


@pytest.mark.parametrize("prec", [slab.FP32_SPLIT, slab.FP64_PLAIN])
def test_runs_on_a_used_context_equal_fresh_ones(prec):
    runs = [(_release(20.0, 1.5), 2), (_release(9.0, 2.0), 1), (_release(35.0, 1.0), 3), (_release(9.0, 2.0), 1), (_release(9.0, 2.5), 2)]
    s = slab.Slab(Z, DX)
    s.set_params(CFG, prec)
    for rel, frames in runs:
        got, state, launches = _run(s, rel, frames)
        f = slab.Slab(Z, DX)
        f.set_params(CFG, prec)
        want, fstate, _ = _run(f, rel, frames)
        f.close()
        assert state == fstate
        for a, b in zip(got, want):
            if prec == slab.FP32_SPLIT:
                assert np.array_equal(a, b)
            else:  # its sums are atomics in arrival order: rounding apart, amplified over at most 75 steps
                assert np.abs(a - b).max() <= 1e-9 * max(1.0, np.abs(b).max())
        assert 0 < launches < 3000  # counted from this run's upload on
        with pytest.raises(slab.SlabError):  # a release over the terrain's edge: refused, and nothing of it is kept
            s.upload_release({**rel, "center": (2.0, 96.0)})
    s.close()
