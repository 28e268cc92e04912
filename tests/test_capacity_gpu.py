"""More active tiles than the work list can hold (2^31 floats of partial sums): an
error, and the tiles on the list read no partial sums of tiles past its end."""
import numpy as np
import pytest

import slab

pytestmark = pytest.mark.gpu


def test_more_active_tiles_than_the_work_list_holds():
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GiB of free device memory")
    tiles, n = 1800, 14400  # 3.24 M tiles of 8 x 8 cells, one particle in each but the outermost
    assert (tiles - 2) ** 2 > (2**31 - 1) // 700
    s = slab.Slab(np.zeros((n, n)), 1.0)
    s.set_params(dict(gravity=9.81, rho=300.0, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=1.0, total_time=10.0, friction="COULOMB",
                      coulomb_mu=0.4), slab.FP32_SPLIT)
    at = 8.0 * np.arange(1, tiles - 1) + 3.7
    x = np.stack(np.meshgrid(at, at, indexing="ij"), -1).reshape(-1, 2)
    one = np.ones(len(x))
    s.upload({"x": x, "v": 0 * x, "vz": 0 * one, "h": one, "A": 0.25 * one, "mass": 75.0 * one, "z": 0 * one})
    with pytest.raises(slab.SlabError) as ex:
        s.initial_pass()
    assert ex.value.code == 3  # SLAB_E_OOM
    s.upload({k: v[:4] for k, v in {"x": x, "v": 0 * x, "vz": 0 * one, "h": one, "A": 0.25 * one, "mass": 75.0 * one, "z": 0 * one}.items()})
    s.initial_pass()
    assert s.advance_steps(3) == 3
    assert np.abs(s.particles()["x"] - x[:4]).max() < 0.1
    s.close()
    slab.trim_memory()
