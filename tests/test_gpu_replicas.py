"""A DoF on a macro-face, -edge or -vertex is stored once per adjacent cell; the lanes that
compute it together read one replica and write all of them. The copies have to agree
afterwards: an operator application reads every cell's own copies, a download only the first,
so A x on the GPU has to match the oracle's A x of the downloaded x (1e-12 of its largest
entry in FP64, the bound of the apply's parity tests). After uploads, and after under-relaxed
sweeps and the additive prolongation, whose results depend on the old value, through each
route of the interface passes (chosen by environment variables, in a child process): the row
tables, a launch per colour without tables, one launch for all colours."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_barrier_over_the_active_mask():
    # the active mask is whatever lanes happen to run together: a barrier over it orders nothing
    csrc = os.path.join(ROOT, "hyteg-vara_b200", "csrc")
    for f in sorted(os.listdir(csrc)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, f)).read())
        assert not re.search(r"__syncwarp\s*\(\s*__activemask", text), f


def check(mesh, level):
    import hyteg_b200 as H
    import oracle as O

    coords, tets = O.mesh_cuboid(*(int(c) for c in mesh))
    st, orc = H.PrimitiveStorage(coords, tets, level), O.Oracle(coords, tets, level)
    A = H.P1ConstantLaplaceOperator(st, level - 1, level)
    flag = H.INNER | H.NEUMANN
    rng = np.random.default_rng(level)
    x, b, y = (H.P1Function(n, st, level - 1, level) for n in "xby")
    x.set(rng.uniform(-1, 1, orc.n(level)), level)
    x.set(rng.uniform(-1, 1, orc.n(level - 1)), level - 1)
    b.set(rng.uniform(-1, 1, orc.n(level)), level)

    def copies_agree(what):
        A.apply(x, y, level, flag)
        ref = orc.apply(x.get(level), level, flag=flag)
        err = np.abs(y.get(level) - ref).max() / np.abs(ref).max()
        assert err <= 1e-12, (what, err)

    copies_agree("upload")
    for what, step in (("forward", A.smooth_sor), ("backward", A.smooth_sor_backwards)):
        for relax in (0.8, 1.3):
            step(x, b, relax, level, flag)
            copies_agree((what, relax))
    before, coarse = x.get(level), x.get(level - 1)
    H.P1toP1LinearProlongation().prolongate_and_add(x, level - 1, flag)
    ref = orc.prolongate(coarse, level - 1, before.copy(), flag=flag, add=True)
    assert np.abs(x.get(level) - ref).max() <= 1e-12 * np.abs(ref).max()
    copies_agree("prolongate and add")


@pytest.mark.gpu
@pytest.mark.parametrize("mesh,level", [("111", 3), ("222", 4), ("222", 6)])
@pytest.mark.parametrize("route", ["tables", "colours", "one"])
def test_copies_of_interface_dofs_agree(mesh, level, route):
    env = dict(os.environ, HYB_SURFACE_MIN_DOFS="0" if route == "one" else str(1 << 30),
               PYTHONPATH=os.pathsep.join([os.path.join(ROOT, "oracle"), os.path.join(ROOT, "hyteg-vara_b200", "python")]))
    if route != "tables":
        env.update(HYB_ROW_TABLE_MAX_POINTS="0", HYB_ROW_IFACE_MAX_POINTS="0")
    r = subprocess.run([sys.executable, os.path.abspath(__file__), mesh, str(level)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


if __name__ == "__main__":
    check(sys.argv[1], int(sys.argv[2]))
