"""The interface passes of a multicolour SOR sweep as one cooperative launch (hyb_surface.cu:
constant stencil, Inner | Neumann, many surface DoFs) through the C ABI against the CPU oracle.

The launch takes over at half a million surface DoFs; here HYB_SURFACE_MIN_DOFS lowers that in
a child process, so that it runs on: the smallest levels it takes (faces of 21 points), six
macro-tets (every face cut into row ranges, fewer blocks than SMs), the 48-tet cuboid (as many
ranges as SMs), a 144-tet box (several whole faces per block), level 7 and the spherical shell
(seven colours). Whole sweeps, forward and backward, relax 1 and 0.8. The rows are summed in
another order than the oracle's, in the sweep's precision: 1e-11 in FP64 (max norm, relative),
the bound of the sweeps' parity tests; 2e-5 for two FP32 sweeps."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def check(mesh, level):
    import hyteg_b200 as H
    import oracle as O

    if mesh == "shell":
        st = H.PrimitiveStorage.spherical_shell(3, 2, 0.55, 1.0, level)
        coords, tets = st.mesh()
    else:
        coords, tets = O.mesh_cuboid(*(int(c) for c in mesh))
        st = H.PrimitiveStorage(coords, tets, level)
    orc = O.Oracle(coords, tets, level)
    A = H.P1ConstantLaplaceOperator(st, level, level)
    m, labels = st.colouring()
    rng = np.random.default_rng(level)
    x0, b = rng.uniform(-1, 1, orc.n(level)), rng.uniform(-1, 1, orc.n(level))
    for dtype, np_dtype, tol in ((H.F64, np.float64, 1e-11), (H.F32, np.float32, 2e-5)):
        x0, b = x0.astype(np_dtype), b.astype(np_dtype)
        fx, fb = H.P1Function("x", st, level, level, dtype), H.P1Function("b", st, level, level, dtype)
        fb.set(b, level)
        for relax, order in ((1.0, (False, False)), (0.8, (True, False))):
            fx.set(x0, level)
            ref = x0.astype(np.float64)
            for backwards in order:
                n = H.load().hyb_kernel_launch_count()
                (A.smooth_sor_backwards if backwards else A.smooth_sor)(fx, fb, relax, level, H.INNER | H.NEUMANN)
                # one launch for the interfaces, one or four for the interiors
                assert H.load().hyb_kernel_launch_count() - n in (2, 5)
                orc.sor_colored(ref, b.astype(np.float64), level, labels, m, relax=relax, flag=1 | 4, backwards=backwards)
            err = np.abs(fx.get(level).astype(np.float64) - ref).max() / np.abs(ref).max()
            assert err <= tol, (dtype, relax, order, err)


@pytest.mark.gpu
@pytest.mark.parametrize("mesh,level", [("111", 3), ("221", 4), ("111", 6), ("111", 7), ("222", 6), ("432", 6), ("shell", 6)])
def test_interface_passes_match_oracle(mesh, level):
    env = dict(os.environ, HYB_SURFACE_MIN_DOFS="0",
               PYTHONPATH=os.pathsep.join([os.path.join(ROOT, "oracle"), os.path.join(ROOT, "hyteg-vara_b200", "python")]))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), mesh, str(level)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.gpu
def test_large_meshes_leave_the_one_launch_by_type():
    """848 inner faces at level 6 are six a block: 114 KB in FP32, which runs in one launch, and
    206 KB, more than the limit, in FP64, which takes a launch per colour. The two agree to the bound of
    the FP32 sweep above."""
    import hyteg_b200 as H

    level = 6
    st = H.PrimitiveStorage.cuboid(4, 4, 5, level)
    A = H.P1ConstantLaplaceOperator(st, level, level)
    m, _ = st.colouring()
    rng = np.random.default_rng(1)
    x0, b = (rng.uniform(-1, 1, st.num_dofs(level)).astype(np.float32) for _ in range(2))
    got = []
    for dtype, launches in ((H.F64, m + 4), (H.F32, 1 + 4)):
        fx, fb = H.P1Function("x", st, level, level, dtype), H.P1Function("b", st, level, level, dtype)
        fx.set(x0, level)
        fb.set(b, level)
        n = H.load().hyb_kernel_launch_count()
        A.smooth_sor(fx, fb, 0.8, level, H.INNER | H.NEUMANN)
        assert H.load().hyb_kernel_launch_count() - n == launches
        got.append(fx.get(level).astype(np.float64))
    assert np.abs(got[1] - got[0]).max() <= 2e-5 * np.abs(got[0]).max()


if __name__ == "__main__":
    check(sys.argv[1], int(sys.argv[2]))
