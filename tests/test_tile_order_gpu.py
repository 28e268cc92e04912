"""The order in which P2G and G2P take the tiles of a step. One scenario alone
takes them by size (uneven: 2 000 tiles of 1 to 1 000 particles) or in turn
(many: more than 16 per CTA); in a batch beside another one it takes fixed runs
of the list. A tile's sums do not depend on when it is computed, so the bits are
the same. Then one tile at the edges of P2G's passes of 384 candidates."""
import numpy as np
import pytest

import slab
import test_p2g_tiles_gpu as tiles

pytestmark = pytest.mark.gpu

DX, RHO = 1.0, 300.0
CFG = dict(gravity=9.81, rho=RHO, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=0.05, total_time=0.1, friction="COULOMB",
           coulomb_mu=0.4)


def _scenario(side, counts, seed):
    """counts[k] particles in the k-th of randomly drawn tiles of a side x side terrain of 8-cell tiles"""
    rng = np.random.default_rng(seed)
    t = np.repeat(rng.permutation(side * side)[:len(counts)], counts)
    x = np.clip(np.stack([t // side, t % side], 1) * 8.0 + rng.uniform(0.0, 8.0, (len(t), 2)), 2.0, 8.0 * side - 3.0)
    m = len(x)
    h, A = rng.uniform(0.5, 2.0, m), np.full(m, DX * DX / 8.0)
    return {"x": x, "v": rng.normal(0.0, 1.0, (m, 2)), "vz": np.zeros(m), "h": h, "A": A, "mass": RHO * h * A, "z": np.zeros(m)}


def _case(kind):
    rng = np.random.default_rng(11)
    if kind == "uneven":
        side, counts = 60, np.concatenate([rng.integers(1, 120, 1900), rng.integers(300, 1000, 90), [383, 384, 385, 768, 769, 1000]])
    else:
        side, counts = 150, rng.integers(5, 8, 150 * 150 - 40)
    i = np.arange(8 * side)
    return -0.3 * i[:, None] * DX + 0.2 * np.sin(0.2 * i)[None, :], _scenario(side, rng.permutation(counts), 12)


@pytest.mark.parametrize("kind", ["uneven", "many"])
def test_alone_equals_beside_another(kind):
    z, P = _case(kind)
    s = slab.Slab(z, DX)
    s.set_params(CFG, slab.FP32_SPLIT)
    s.upload(P)
    s.initial_pass()
    n = s.advance_steps(10 ** 9)
    b = slab.Batch(z, DX, max_scenarios=2)
    sid = b.add(CFG, P)
    b.add(CFG, {k: v[:7] for k, v in P.items()})
    b.run()
    assert b.state(sid)[2] == n and n > 5
    Pa, Pb = s.particles(), b.particles(sid)
    for k in Pa:
        assert np.array_equal(Pa[k], Pb[k]), k
    for a, c in zip(s.max_maps(), b.max_maps(sid)):
        assert np.array_equal(a, c)
    s.close()
    b.close()


def test_thread_per_cell_equals_thread_per_row():
    """Steps of more than 4 096 tiles sum with a thread per cell, in passes of
    288 candidates; persistent steps with three. The same operations in the same
    order: the same bits, also of the grid members of an output step."""
    rng = np.random.default_rng(21)
    counts = rng.permutation(np.concatenate([rng.integers(1, 120, 4300), [48, 49, 287, 288, 289, 575, 576, 577, 1000]]))
    P = _scenario(70, counts, 22)
    i = np.arange(8 * 70)
    out = []
    for persistent in (False, True):
        s = slab.Slab(-0.3 * i[:, None] * DX + 0.2 * np.sin(0.2 * i)[None, :], DX)
        s.set_params(CFG, slab.FP32_SPLIT)
        s.set_persistent(persistent)
        s.upload(P)
        s.initial_pass()
        g = s.grid()
        s.advance_to_frame()
        out.append((s.particles(), g, s.grid(), s.state()))
        s.close()
    (Pa, ga, fa, sa), (Pb, gb, fb, sb) = out
    assert sa == sb
    for a, b in ((Pa, Pb), (ga, gb), (fa, fb)):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n", [383, 384, 385, 768, 769])
def test_pass_edges_against_fp64(n):
    tiles.test_tile_sums_against_fp64(n, True)
