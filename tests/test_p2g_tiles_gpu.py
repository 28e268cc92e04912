"""P2G of one tile at the sizes where its kernel changes course: one particle,
the last fixed-point tile and the first cell-sorted one (48, 49), one pass of
candidates and its edges (320), several passes, all in one cell or spread. The
t = 0 grid against FP64_PLAIN, which the oracle pins.

Tolerance: a contribution m w has w <= 9/16 from a dozen FP32 roundings of
values below 2 and an offset rounded to FP32, so its error is below
16 u m (u = 2^-24); n of them summed one after the other add at most n u of
the sum of their sizes. So |error| <= (16 + n) u M for a node's mass, M the
mass of all particles, and the same with M max(h) and the force terms. Offsets
whose weights lie within 1e-4 of the 3e-3 cut-off are not drawn: there the two
arithmetics may differ by a whole contribution."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu

N, DX, RHO = 48, 1.0, 300.0
CFG = dict(gravity=9.81, rho=RHO, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=1.0, total_time=10.0, friction="COULOMB",
           coulomb_mu=0.4)


def _weights(u):
    f = u - np.floor(u - 0.5)
    return np.stack([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1.0) ** 2, 0.5 * (f - 0.5) ** 2], -1)


def _particles(n, spread, seed):
    """n particles with base cells in the tile of cells 16..23: over the tile, or all in one cell."""
    rng = np.random.default_rng(seed)
    out = np.zeros((0, 2))
    while len(out) < n:
        x = 16.5 + (8.0 if spread else 1.0) * rng.random((4 * n + 16, 2)) * 0.999 + (0.0 if spread else 3.0)
        w = _weights(x[:, 0])[:, :, None] * _weights(x[:, 1])[:, None, :]
        out = np.concatenate([out, x[(np.abs(w - 3e-3) > 1e-4).all((1, 2))]])
    x = out[:n] * DX
    h, A = rng.uniform(0.5, 3.0, n), np.full(n, DX * DX / 4.0)
    return {"x": x, "v": rng.normal(0.0, 2.0, (n, 2)), "vz": np.zeros(n), "h": h, "A": A, "mass": RHO * h * A, "z": np.zeros(n)}


@pytest.mark.parametrize("n,spread", [(1, True), (48, True), (48, False), (49, True), (192, True), (193, True), (319, True), (320, True),
                                      (321, False), (640, True), (641, True), (1500, True), (1500, False)])
def test_tile_sums_against_fp64(n, spread):
    i = np.arange(N)
    z = -0.3 * i[:, None] * DX + 0.2 * np.sin(0.7 * i)[None, :] + 0.1 * np.cos(0.5 * i)[:, None]
    P = _particles(n, spread, n)
    g = []
    for prec in (slab.FP32_SPLIT, slab.FP64_PLAIN):
        s = slab.Slab(z, DX)
        s.set_params(CFG, prec)
        s.upload(P)
        s.initial_pass()
        g.append(s.grid())
        s.close()
    a, b = g
    assert (a["Nx"], a["Ny"], a["i_off"], a["j_off"]) == (b["Nx"], b["Ny"], b["i_off"], b["j_off"])
    tol = (16 + n) * 2.0 ** -24
    M, hmax = P["mass"].sum(), P["h"].max()
    assert np.abs(a["mass"] - b["mass"]).max() <= tol * M
    assert np.abs(a["mass"] * a["h"] - b["mass"] * b["h"]).max() <= 2 * tol * M * hmax
    # force of one particle: m g cos^2 (slope + h / (2 dx) * weight gradient), slopes below 0.5, gradients below 1
    assert np.abs(a["F"] - b["F"]).max() <= tol * M * CFG["gravity"] * (0.5 + 0.5 * hmax / DX)
    assert (b["mass"] > 0).any()
