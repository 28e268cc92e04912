"""The step graphs (csrc/graphs.hpp) when something fails while a step is being
captured, over a stand-in for the CUDA runtime (graphs_driver.cpp)."""
import os
import subprocess

from test_blocks import CSRC, HERE, _cuda_include


def test_a_failed_capture_leaves_the_stream_usable(tmp_path):
    exe = str(tmp_path / "graphs_driver")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, os.path.join(HERE, "graphs_driver.cpp"), "-I", CSRC, "-I",
                    os.path.join(CSRC, "..", "..", "include"), "-I", _cuda_include()], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
