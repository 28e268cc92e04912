"""FP64: particles within half a cell of the terrain's first row and column of
nodes, whose stencil starts at node 0 as the reference's truncated base index
does, against the oracle. Tolerances as in test_plain64_gpu.py: 1e-12 relative
per step, over 20 steps 20 times that."""
import numpy as np
import pytest

import oracle as O
import slab

pytestmark = pytest.mark.gpu

N, DX = 24, 2.0
CFG = dict(gravity=9.81, rho=300.0, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=0.1, total_time=10.0, friction="COULOMB",
           coulomb_mu=0.1)


@pytest.mark.parametrize("corner", ["x", "y", "xy"])
def test_half_a_cell_from_the_first_nodes(corner):
    i = np.arange(N)
    z = -0.2 * i[:, None] * DX - 0.2 * i[None, :] * DX + 0.05 * np.sin(i)[:, None]  # falls away from both edges
    g = np.random.default_rng(5)
    n = 60
    near, inside = g.uniform(0.05, 0.45, n) * DX, g.uniform(4.0, 9.0, n) * DX
    x = np.stack([near if "x" in corner else inside, near[::-1] if "y" in corner else inside], 1)
    h, A = g.uniform(0.5, 1.5, n), np.full(n, DX * DX / 4)
    P = {"x": x, "v": np.abs(g.normal(0.0, 0.3, (n, 2))), "vz": np.zeros(n), "h": h, "A": A, "mass": 300.0 * h * A, "z": np.zeros(n)}
    s = slab.Slab(z, DX)
    s.set_params(CFG, slab.FP64_PLAIN)
    s.upload(P)
    s.initial_pass()
    o = O.Oracle(CFG, z, DX)
    o.set_particles(dict(P, theta=np.zeros(n)))
    o.t0()
    G, Go = s.grid(), o.grid()
    assert (G["Nx"], G["Ny"], G["i_off"], G["j_off"]) == (Go["Nx"], Go["Ny"], Go["i_off"], Go["j_off"])
    for k in ("mass", "h", "v"):
        np.testing.assert_allclose(G[k], Go[k], rtol=1e-12, atol=1e-12 * np.abs(Go[k]).max(), err_msg=k)
    for _ in range(20):
        assert s.advance_steps(1) == 1
        o.step()
    Q, Qo = s.particles(), o.particles_by_id()
    for k in ("x", "v", "h", "z"):
        np.testing.assert_allclose(Q[k], Qo[k], rtol=2e-11, atol=2e-11 * max(1.0, np.abs(Qo[k]).max()), err_msg=k)
    s.close()
