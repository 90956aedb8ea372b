"""Kernels that take more dynamic shared memory than the default launch on
every device of a process, not only on the first: the built launch code over
a CUDA runtime that keeps each device's limits. CPU only."""
import os
import subprocess

import pytest

import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shared_memory_limit_is_raised_on_every_device(tmp_path):
    objs = [os.path.join(build.OBJ_DIR, f"{n}.cu.o") for n in ("gol_kernels", "gol_local")]
    if not all(os.path.exists(o) for o in objs):
        pytest.skip("the engine's objects are not here (only its library)")
    exe = str(tmp_path / "launch_fake_cuda")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT}/include", f"-I{cuda}/include",
                    os.path.join(ROOT, "tests", "launch_fake_cuda.cpp"), *objs, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
