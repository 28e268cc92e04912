"""The step control (csrc/common.cuh) where a step is begun and not run: the launch
of an advance call's next steps failed, or time did not move on. The next call has
to begin the same step again; a box made of the cleared accumulators would reach
outside the terrain."""
import os
import subprocess

import numpy as np
import pytest

import slab
from test_blocks import CSRC, HERE, Z, DX, CFG, _cuda_include, _release


def test_a_step_begun_twice_keeps_its_box(tmp_path):
    exe = str(tmp_path / "control_driver")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "control_driver.cpp"), "-I", CSRC, "-I",
                    os.path.join(CSRC, "..", "..", "include"), "-I", _cuda_include()], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [slab.FP32_SPLIT, slab.FP64_PLAIN])
def test_steps_after_time_stood_still(prec):
    """With a vanishing Courant number time stops moving once the particles do;
    advance_to_frame gives up between two steps. What follows is what follows the
    same number of steps taken without giving up."""
    def context():
        s = slab.Slab(Z, DX)
        s.set_params(dict(CFG, C_cfl=1e-300), prec)
        s.upload_release(_release(20.0))
        s.initial_pass()
        return s

    a = context()
    with pytest.raises(slab.SlabError) as ex:
        a.advance_to_frame()
    assert ex.value.code == 6  # SLAB_E_TIMEOUT
    n = a.state()[3]
    assert a.advance_steps(2) == 2
    b = context()
    assert b.advance_steps(n + 2) == n + 2
    for s in (a, b):
        s.frame_capture(0)
    fa, fb = a.frame_wait(0), b.frame_wait(0)
    assert [fa[k] for k in ("Nx", "Ny", "i_off", "j_off")] == [fb[k] for k in ("Nx", "Ny", "i_off", "j_off")]
    assert fa["Nx"] > 0
    Pa, Pb = a.particles(), b.particles()
    for k in ("x", "v", "h", "mass"):
        if prec == slab.FP32_SPLIT:
            assert np.array_equal(Pa[k], Pb[k]), k
        else:  # the order of FP64 sums is free
            np.testing.assert_allclose(Pa[k], Pb[k], rtol=1e-9, atol=1e-9, err_msg=k)
    for s in (a, b):
        s.close()
