"""The memory blocks kept between calls (csrc/blocks.cu): who gets a released
block and when, the bounds, failed allocations, several threads. On the CPU over
a counting stand-in for the CUDA runtime (blocks_driver.cpp); on the GPU beside
another thread's stream capture, which a wait for the whole device would break."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

import slab

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "slab-pro_b200", "csrc")


def _cuda_include():
    nvcc = shutil.which("nvcc")
    homes = [os.environ.get("CUDA_HOME"), nvcc and os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "/usr/local/cuda"]
    for h in homes:
        if h and os.path.exists(os.path.join(h, "include", "cuda_runtime.h")):
            return os.path.join(h, "include")
    pytest.skip("no CUDA headers")


def test_rules_over_a_counting_runtime(tmp_path):
    exe = str(tmp_path / "blocks_driver")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, os.path.join(HERE, "blocks_driver.cpp"), "-x", "c++", os.path.join(CSRC, "blocks.cu"),
                    "-I", CSRC, "-I", os.path.join(os.path.dirname(CSRC), "..", "include"), "-I", _cuda_include(), "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


N, DX = 96, 2.0
CFG = dict(gravity=9.81, rho=300.0, C_cfl=0.5, dt_max=0.01, flip_ratio=0.95, output_dt=0.25, total_time=5.0, friction="VOELLMY",
           voellmy_mu=0.2, voellmy_xi=1000.0)
I = np.arange(N)
Z = -0.4 * I[:, None] * DX + 0.3 * np.sin(0.3 * I)[None, :]


def _release(r):
    return {"type": "ELLIPSE", "center": (60.0, 96.0), "rx": r, "ry": 0.7 * r, "rotation_deg": 20.0, "h0": 1.5}


def _run(s, r):
    s.upload_release(_release(r))
    s.initial_pass()
    s.advance_to_frame()
    P = s.particles()
    return [P[k] for k in ("x", "v", "h")] + list(s.max_maps())


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [slab.FP32_SPLIT, slab.FP64_PLAIN])
def test_uploads_beside_a_capture_of_another_thread(prec):
    """While this thread's stream is being captured, another thread uploads and
    runs releases of changing sizes, sets parameters and closes its context."""
    torch = pytest.importorskip("torch")
    sizes = [20.0, 9.0, 35.0, 14.0]

    def job(out):
        try:
            s = slab.Slab(Z, DX)
            for r in sizes:
                s.set_params(CFG, prec)
                out.append(_run(s, r))
            for r in sizes:
                out.append(_run(s, r))
            s.close()
        except Exception as e:  # noqa: BLE001 - handed to the main thread
            out.append(e)

    want, got = [], []
    job(want)  # (every module is loaded before the capture)
    a = torch.ones(1024, device="cuda")
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        b = a * 2.0
        t = threading.Thread(target=job, args=(got,))
        t.start()
        t.join()
        b += 1.0
    for w, o in zip(want, got):
        assert not isinstance(o, Exception), o
        for x, y in zip(w, o):
            if prec == slab.FP32_SPLIT:
                assert np.array_equal(x, y)
            else:  # its sums are atomics in arrival order: rounding apart, amplified over at most 25 steps
                assert np.abs(x - y).max() <= 1e-9 * max(1.0, np.abs(x).max())
    assert len(got) == len(want) == 2 * len(sizes)
    g.replay()
    torch.cuda.synchronize()
    assert float(b.sum()) == 3.0 * 1024


def _held(torch, free0):
    torch.cuda.synchronize()
    return free0 - torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
def test_kept_memory_is_given_back():
    """4 M particles take 80 bytes each and some 500 MB while they are sorted
    in. After the last context is closed at most 1 GiB stays, after a trim
    nothing; while the context lives, a small run and a trim leave what a
    context that only ever had the small run holds."""
    torch = pytest.importorskip("torch")
    n = 4 << 20
    rng = np.random.default_rng(3)
    h, A = rng.uniform(0.5, 3.0, n), np.full(n, 1e-2)
    P = {"x": rng.uniform(40.0, 150.0, (n, 2)), "v": np.zeros((n, 2)), "vz": np.zeros(n), "h": h, "A": A, "mass": 300.0 * h * A, "z": np.zeros(n)}
    few = {k: v[:1000] for k, v in P.items()}

    def context():
        s = slab.Slab(Z, DX)
        s.set_params(CFG, slab.FP32_SPLIT)
        return s

    s = context()
    s.upload(P)  # (every kernel is loaded)
    s.initial_pass()
    s.close()
    slab.trim_memory()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    s = context()
    s.upload(few)
    slab.trim_memory()
    small = _held(torch, free0)
    s.upload(P)
    slab.trim_memory()
    assert _held(torch, free0) > 80 * n
    s.upload(few)
    slab.trim_memory()
    assert _held(torch, free0) <= small + (8 << 20)
    s.upload(P)
    s.initial_pass()
    s.close()
    assert _held(torch, free0) <= (1 << 30) + (8 << 20)
    slab.trim_memory()
    assert _held(torch, free0) <= 8 << 20
