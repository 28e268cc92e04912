"""Persistent steps of few and of many tiles (the grid update inside G2P or as a
phase of its own: Engine32::fused): bitwise the steps of separate kernels,
for one scenario, around the line between the two, and in a batch."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu

N = 1024
CFG = dict(gravity=9.81, rho=300.0, C_cfl=0.5, dt_max=0.02, flip_ratio=0.95, output_dt=0.2, total_time=10.0, friction="VOELLMY",
           voellmy_mu=0.2, voellmy_xi=1000.0)
I = np.arange(N)
Z = -0.5 * I[:, None] + 0.3 * np.sin(0.1 * I)[None, :]


def _rect(lx, ly, cx=400.0, cy=512.0):
    return {"type": "RECTANGLE", "center": (cx, cy), "Lx": lx, "Ly": ly, "rotation_deg": 0.0, "h0": 1.5}


@pytest.mark.parametrize("lx,ly", [(96.0, 96.0), (509.0, 507.0), (600.0, 640.0)])  # 144, about 4 096, 6 000 tiles
def test_one_scenario(lx, ly):
    out = []
    for persistent in (False, True):
        s = slab.Slab(Z, 1.0)
        s.set_params(CFG, slab.FP32_SPLIT)
        if persistent:
            s.set_persistent(True)
        s.upload_release(_rect(lx, ly))
        s.initial_pass()
        s.advance_to_frame()
        s.advance_steps(35)
        P = s.particles()
        g = s.grid()
        out.append([P[k] for k in ("x", "v", "vz", "h", "mass", "z")] + list(s.max_maps()) + [g[k] for k in ("h", "mass", "v", "vz", "F")])
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_batch_of_many_tiles():
    out = []
    for persistent in (False, True):
        b = slab.Batch(Z, 1.0, max_scenarios=3)
        if persistent:
            b.set_persistent(True)
        ids = [b.add_release(dict(CFG, total_time=t), r) for t, r in
               ((0.5, _rect(400.0, 430.0)), (0.9, _rect(380.0, 300.0, 500.0, 400.0)), (0.7, _rect(60.0, 60.0)))]
        b.run()
        out.append([x for k in ids for x in (b.particles(k)["x"], b.particles(k)["v"], *b.max_maps(k))])
        b.close()
    for a, c in zip(*out):
        assert np.array_equal(a, c)
