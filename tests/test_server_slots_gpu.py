"""A request that cannot be admitted (its particles reach past the terrain) gives
its slot back, whether the slot is new or has served another one."""
import numpy as np
import pytest

import slab
from test_blocks import CFG, DX, N, Z, _release

pytestmark = pytest.mark.gpu

RUN = dict(CFG, total_time=0.2)


def _outside():
    x = np.array([[60.0, 96.0], [(N - 1) * DX - 0.1, 96.0]])
    one = np.ones(2)
    return {"x": x, "v": 0 * x, "vz": 0 * one, "h": one, "A": one, "mass": 300.0 * one, "z": 0 * one}


@pytest.mark.parametrize("first_fails", [True, False])
def test_slot_of_a_refused_request_serves_the_next(first_fails):
    s = slab.Server(Z, DX, max_scenarios=1)
    ids = []
    if not first_fails:
        ids.append(s.submit_release(RUN, _release(16.0)))
    bad = s.submit(RUN, _outside())
    ids += [s.submit_release(RUN, _release(16.0)) for _ in range(2)]
    s.drain()
    with pytest.raises(slab.SlabError):
        s.result(bad)
    got = [s.result(k) for k in ids]
    for g in got[1:]:
        for k in ("x", "v", "h", "h_max"):
            assert np.array_equal(g[k], got[0][k]), k
    s.close()


def test_batch_goes_on_after_a_refused_scenario():
    out = []
    for refused in (False, True):
        b = slab.Batch(Z, DX, max_scenarios=2)
        ids = [b.add_release(RUN, _release(16.0))]
        if refused:
            with pytest.raises(slab.SlabError):
                b.add(RUN, _outside())
        ids.append(b.add_release(RUN, _release(20.0)))
        b.run()
        out.append([b.particles(k)["x"] for k in ids] + [m for k in ids for m in b.max_maps(k)])
        b.close()
    for a, c in zip(*out):
        assert np.array_equal(a, c)
