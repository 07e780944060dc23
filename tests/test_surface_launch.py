"""Host side of the one-launch interface passes of an SOR sweep, on a fake CUDA runtime: what
the launch needs is set on every device of the process. No GPU is used."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("surface")
    csrc, cpp = os.path.join(ROOT, "hyteg-vara_b200", "csrc"), os.path.join(ROOT, "tests", "cpp")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cuda = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    objs = []
    for f in (os.path.join(csrc, "hyb_surface.cu"), os.path.join(cpp, "surface_launch.cu"), os.path.join(cpp, "fake_cudart.cpp")):
        objs.append(str(tmp / (os.path.basename(f) + ".o")))
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", csrc, "-c", "-o", objs[-1], f],
                       check=True)
    out = str(tmp / "surface_launch")
    subprocess.run(["g++", "-I", cuda, "-o", out] + objs, check=True)  # without the real runtime
    return out


@pytest.mark.parametrize("check", ["devices"])
def test_host_side(exe, check):
    r = subprocess.run([exe, check], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
