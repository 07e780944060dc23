"""Host side of the one-launch interface passes of an SOR sweep, on a fake CUDA runtime: what
the launch needs is set on every device of the process; a device, or a stream's part of one,
that cannot hold the grid is noticed before anything is launched or captured. On a GPU: a sweep
on a stream of 64 SMs, launched and captured, takes the launches per colour."""
import os
import subprocess
import sys

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


@pytest.mark.parametrize("check", ["devices", "fits", "stream", "silent"])
def test_host_side(exe, check):
    r = subprocess.run([exe, check], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def check_small_stream():
    import numpy as np
    from cuda.bindings import driver as cu, runtime as rt

    import hyteg_b200 as H
    import oracle as O

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]

    level = 4
    coords, tets = O.mesh_cuboid(2, 2, 2)
    st, orc = H.PrimitiveStorage(coords, tets, level), O.Oracle(coords, tets, level)
    A = H.P1ConstantLaplaceOperator(st, level, level)
    m, labels = st.colouring()
    sms = ok(cu.cuDeviceGetDevResource(0, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    part = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 64))[0][0]
    green = ok(cu.cuGreenCtxCreate(ok(cu.cuDevResourceGenerateDesc([part], 1)), 0,
                                   cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    small = int(ok(cu.cuGreenCtxStreamCreate(green, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0)))
    rng = np.random.default_rng(1)
    x0, b = rng.uniform(-1, 1, orc.n(level)), rng.uniform(-1, 1, orc.n(level))
    x, fb = H.P1Function("x", st, level, level), H.P1Function("b", st, level, level)
    fb.set(b, level)

    def sweep(stream):
        n = H.load().hyb_kernel_launch_count()
        A.smooth_sor(x, fb, 0.9, level, H.INNER | H.NEUMANN, stream=stream)
        return H.load().hyb_kernel_launch_count() - n

    ref = x0.copy()
    orc.sor_colored(ref, b, level, labels, m, relax=0.9, flag=1 | 4)
    for stream, captured, launches in ((None, False, 2), (small, False, m + 1), (small, True, m + 1)):
        x.set(x0, level)
        ok(rt.cudaStreamSynchronize(0) + (None,))  # the small stream does not wait for the default one
        if captured:
            ok(rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal) + (None,))
        assert sweep(stream) == launches
        if captured:
            run = ok(rt.cudaGraphInstantiate(ok(rt.cudaStreamEndCapture(stream)), 0))
            ok(rt.cudaGraphLaunch(run, stream) + (None,))
        ok(rt.cudaStreamSynchronize(stream or 0) + (None,))
        err = np.abs(x.get(level) - ref).max() / np.abs(ref).max()
        assert err <= 1e-11, (captured, err)  # the bound of the sweeps' parity tests


@pytest.mark.gpu
def test_stream_of_a_part_of_the_device():
    env = dict(os.environ, HYB_SURFACE_MIN_DOFS="0",
               PYTHONPATH=os.pathsep.join([os.path.join(ROOT, "oracle"), os.path.join(ROOT, "hyteg-vara_b200", "python")]))
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


if __name__ == "__main__":
    check_small_stream()
