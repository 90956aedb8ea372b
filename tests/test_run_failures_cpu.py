"""gol_run when a CUDA call fails in a run on interleaved rows: the grid is a
valid one afterwards (or refused), never words in another order. The engine's
source is compiled over a CUDA runtime of host memory. CPU only."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fake_cuda") / "engine_fake_cuda")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    csrc = os.path.join(ROOT, "stencil-optimalizations_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffunction-sections", "-Wl,--gc-sections",
                    f"-I{ROOT}/include", f"-I{csrc}", f"-I{cuda}/include", "-x", "c++",
                    os.path.join(csrc, "gol_engine.cu"),
                    os.path.join(ROOT, "tests", "engine_fake_cuda.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", ["instantiate", "launch", "restore"])
def test_failed_run(engine, what):
    r = subprocess.run([engine, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
