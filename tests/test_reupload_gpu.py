"""What a context's next upload takes over from the run before it, in the cases
where that run did not simply end: a persistent launch that gave up, uploads that
are never run, sizes that grow."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu

N, DX = 96, 2.0
CFG = dict(gravity=9.81, rho=300.0, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=0.25, total_time=5.0, friction="VOELLMY",
           voellmy_mu=0.2, voellmy_xi=1000.0)
I = np.arange(N)
Z = -0.4 * I[:, None] * DX + 0.3 * np.sin(0.3 * I)[None, :]


def _release(r):
    return {"type": "ELLIPSE", "center": (60.0, 96.0), "rx": r, "ry": 0.7 * r, "rotation_deg": 20.0, "h0": 1.5}


def _context(prec=slab.FP32_SPLIT):
    s = slab.Slab(Z, DX)
    s.set_params(CFG, prec)
    return s


def _run(s, r):
    s.upload_release(_release(r))
    s.initial_pass()
    _, _, steps = s.advance_to_frame()
    steps += s.advance_steps(40)
    P = s.particles()
    return [P[k] for k in ("x", "v", "vz", "h", "mass", "z")] + list(s.max_maps()), steps, s.state()


@pytest.mark.parametrize("waited", [True, False])
@pytest.mark.parametrize("persistent", [True, False])
def test_upload_after_a_persistent_launch_gave_up(waited, persistent):
    """The run that gave up ends with the upload: the next one is a new context's."""
    s = _context()
    s.set_persistent(True, limit_cycles=64)  # far below one phase: the early CTAs give up
    s.upload_release(_release(20.0))
    s.initial_pass()
    if waited:
        with pytest.raises(slab.SlabError) as ex:
            s.advance_steps(64)
        assert ex.value.code == 6  # SLAB_E_TIMEOUT
    else:
        s.advance_steps_async(64)
    s.set_persistent(persistent, limit_cycles=4_000_000_000)
    got, steps, state = _run(s, 20.0)
    s.close()
    f = _context()
    want, fsteps, fstate = _run(f, 20.0)
    f.close()
    assert (steps, state) == (fsteps, fstate) and steps > 40
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_uploads_without_an_initial_pass_do_not_grow_the_pool():
    """An upload that replaces one whose t = 0 pass was never run needs no more
    node blocks than the first. 400 of them: each adding its tiles to the
    estimate would ask for some 400 x 150 blocks of 2.8 KB, more than 160 MB."""
    torch = pytest.importorskip("torch")
    s = _context()
    want, steps, state = _run(s, 35.0)
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(400):
        s.upload_release(_release(35.0))
    grown = free0 - torch.cuda.mem_get_info()[0]
    got, steps2, state2 = _run(s, 35.0)
    s.close()
    assert grown < 32 << 20, grown
    assert (steps, state) == (steps2, state2)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def _host_particles(n, seed):
    rng = np.random.default_rng(seed)
    h, A = rng.uniform(0.5, 3.0, n), np.full(n, 1e-2)
    return {"x": rng.uniform(40.0, 150.0, (n, 2)), "v": np.zeros((n, 2)), "vz": np.zeros(n), "h": h, "A": A, "mass": 300.0 * h * A,
            "z": np.zeros(n)}


def test_a_larger_upload_fits_where_it_would_on_a_new_context():
    """FP64 particles are 72 bytes each. After 8 M of them (576 MB), with 312 MB
    of the device left, 12 M (864 MB) fit in the room of both, and not beside any
    64 MB array of the run before that is still there when the last new one of
    96 MB is asked for."""
    torch = pytest.importorskip("torch")
    small, large = _host_particles(8 << 20, 1), _host_particles(12 << 20, 2)
    s = _context(slab.FP64_PLAIN)
    s.upload(small)
    s.initial_pass()
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (312 << 20), dtype=torch.uint8, device="cuda")
    try:
        s.upload(large)
        s.initial_pass()
        assert s.conservation()[0] == pytest.approx(large["mass"].sum(), rel=1e-12)
    finally:
        del rest
        torch.cuda.empty_cache()
        s.close()


def test_the_tuner_starts_anew_with_another_size():
    """Launch shapes are measured on a run's first steps (15 of them, read when
    the next are enqueued), whatever the context ran before; steps of a run of
    another size are not taken together with them."""
    i = np.arange(104)
    z = -0.4 * np.arange(203)[:, None] * DX + 0.3 * np.sin(0.3 * i)[None, :]
    s = slab.Slab(z, DX)
    s.set_params({**CFG, "friction": "COULOMB", "coulomb_mu": 0.8, "total_time": 60.0}, slab.FP32_SPLIT)

    def start(r):
        s.upload_release(_release(r))
        s.initial_pass()

    def tunes():
        return s.launch_shapes()[1]

    start(20.0)
    s.advance_steps(64)
    assert tunes() == 1
    s.advance_steps(1200)  # measured again at growing distances
    n = tunes()
    assert n > 1
    start(40.0)
    s.advance_steps(64)
    assert tunes() == n + 1
    start(10.0)
    s.advance_steps(8)
    start(28.0)  # 8 steps measured, 7 to go: of another size
    s.advance_steps(8)
    s.advance_steps(4)
    assert tunes() == n + 1
    s.advance_steps(8)
    s.advance_steps(4)
    assert tunes() == n + 2
    s.close()
