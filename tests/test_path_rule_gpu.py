"""Steps of 1 500 to 4 096 tiles of one scenario take the kernels of few tiles
or those of many by the heaviest tile's particle count, at upload and as the
flow changes. Either way the bits are those of persistent steps, which always
run the kernels of few tiles; the launches per step tell which ran."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu

DX, RHO = 1.0, 300.0
CFG = dict(gravity=9.81, rho=RHO, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=5.0, total_time=5.0, friction="VOELLMY",
           voellmy_mu=0.2, voellmy_xi=1000.0)


def _case(side, heavy):
    """side x side tiles of 12 particles each, and one with `heavy` more."""
    n = 8 * side + 70
    i = np.arange(n)
    z = -0.2 * i[:, None] * DX + 0.2 * np.sin(0.2 * i)[None, :]
    rng = np.random.default_rng(11)
    t = np.repeat(np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2), 12, 0)
    x = 24.0 + 8.0 * t + rng.uniform(0.6, 8.4, (len(t), 2))
    x = np.concatenate([x, 24.0 + 8.0 * (side // 2) + rng.uniform(1.0, 8.0, (heavy, 2))]) * DX
    m = len(x)
    h, A = rng.uniform(0.5, 2.0, m), np.full(m, DX * DX / 4.0)
    return z, {"x": x, "v": rng.normal(0.0, 0.5, (m, 2)), "vz": np.zeros(m), "h": h, "A": A, "mass": RHO * h * A, "z": np.zeros(m)}


# 1 369 tiles: few; 2 500 and 3 969: many; 2 500 and 3 844 with one of 700 or 1 000: few
@pytest.mark.parametrize("side,heavy,kernels", [(37, 0, 4), (50, 0, 5), (50, 700, 4), (63, 0, 5), (62, 1000, 4)])
def test_kernels_by_heaviest_tile(side, heavy, kernels):
    z, P = _case(side, heavy)
    out = []
    for persistent in (False, True):
        s = slab.Slab(z, DX)
        s.set_params(CFG, slab.FP32_SPLIT)
        s.set_persistent(persistent)
        s.upload(P)
        s.initial_pass()
        n0 = s.kernel_launches()
        s.advance_steps(32)
        if not persistent:
            assert (s.kernel_launches() - n0) // 32 == kernels
        s.advance_steps(40)
        out.append((s.particles(), s.max_maps(), s.state()))
        s.close()
    (Pa, ma, sa), (Pb, mb, sb) = out
    assert sa == sb
    for k in Pa:
        assert np.array_equal(Pa[k], Pb[k]), k
    for a, b in zip(ma, mb):
        assert np.array_equal(a, b)
