"""The grid update as a kernel of its own (steps of more than 4 096 tiles) and
inside G2P (fewer; persistent steps always) give the same bits: particles,
maxima and every grid member, on a full block of tiles, on scattered ones --
whose windows have nodes in grid tiles without particles -- and at the
terrain's far edges."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu

DX, RHO = 1.0, 300.0
CFG = dict(gravity=9.81, rho=RHO, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=0.08, total_time=5.0)
LAWS = {"COULOMB": dict(coulomb_mu=0.4), "VOELLMY": dict(voellmy_mu=0.2, voellmy_xi=1000.0),
        "MU_I": dict(mui_mu1=0.38, mui_mu2=0.64, mui_I0=0.279, mui_d=5e-4, mui_phi=0.6)}


def _case(kind):
    n = 563  # 71 tiles a side, the last one of 3 cells
    i = np.arange(n)
    z = -0.3 * i[:, None] * DX + 0.2 * np.sin(0.2 * i)[None, :]
    rng = np.random.default_rng(5)
    if kind == "block":
        x = rng.uniform(20.0, 555.0, (300000, 2))
    elif kind == "scattered":  # about 4 400 tiles, most with a particle or two, every other one empty
        t = rng.permutation(70 * 70)[:4400]
        x = np.stack([t // 70, t % 70], 1) * 8.0 + rng.uniform(1.0, 8.0, (4400, 2))
        x = np.concatenate([x, x[:500] + 0.3])
    else:  # up to the last cell whose stencil fits
        x = np.concatenate([rng.uniform(2.0, 560.4, (200000, 2)), [[560.4, 560.4], [2.0, 560.4]]])
    m = len(x)
    h = rng.uniform(0.5, 2.0, m)
    A = np.full(m, DX * DX / 4.0)
    return z, {"x": x, "v": rng.normal(0.0, 0.5, (m, 2)), "vz": np.zeros(m), "h": h, "A": A, "mass": RHO * h * A, "z": np.zeros(m)}


@pytest.mark.parametrize("kind,law", [("block", "VOELLMY"), ("scattered", "MU_I"), ("edges", "COULOMB")])
def test_grid_update_alone_equals_inside_g2p(kind, law):
    z, P = _case(kind)
    out = []
    for persistent in (False, True):
        s = slab.Slab(z, DX)
        s.set_params({**CFG, "friction": law, **LAWS[law]}, slab.FP32_SPLIT)
        s.set_persistent(persistent)
        s.upload(P)
        s.initial_pass()
        g = [s.grid()]
        s.advance_to_frame()
        g.append(s.grid())
        if kind != "edges":
            s.advance_steps(3)
            g.append({k: v for k, v in s.grid().items() if k in ("v", "flip", "Nx", "Ny", "i_off", "j_off")})
        out.append((s.particles(), s.max_maps(), g, s.state(), s.conservation()[1]))
        s.close()
    (Pa, ma, ga, sa, ca), (Pb, mb, gb, sb, cb) = out
    assert sa == sb and abs(ca - cb) <= 1e-12 * abs(cb)
    for k in Pa:
        assert np.array_equal(Pa[k], Pb[k]), k
    for a, b in zip(ma, mb):
        assert np.array_equal(a, b)
    for a, b in zip(ga, gb):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
