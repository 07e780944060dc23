"""The one-block CG (k_cg) at the limits of its lists, against the oracle's CG. A thread marks up
to 64 closure points (512 threads: 32768 points) and the block lists up to 512 groups of 32
operator rows; beyond either the passes look classes up, or run every group. 198 macro-tets at
level 3 fill the 64 points (32670), 199 need a 65th (32835), six at level 5 (39270 points, 930
groups of interior rows alone) exceed both, six at level 2 stay far below. With the level's row
table (a multigrid solve on the same operator builds it) and without. Five iterations from a
random start: the applies differ by 1e-13 of their largest entries and a step's scalars carry
that on, so 1e-10 of the iterate bounds the difference with room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,level", [(6, 2), (198, 3), (199, 3), (6, 5)])
@pytest.mark.parametrize("coefficient", ["constant", "nodal"])
@pytest.mark.parametrize("tables", [False, True])
def test_cg_lists_match_oracle(oracle_mod, cells, level, coefficient, tables):
    import hyteg_b200 as H

    O = oracle_mod
    coords, tets = O.mesh_cuboid((cells + 5) // 6, 1, 1)
    used, tets = np.unique(tets[:cells], return_inverse=True)
    coords, tets = coords[used], tets.reshape(cells, 4)
    st, orc = H.PrimitiveStorage(coords, tets, level), O.Oracle(coords, tets, level)
    op = 0
    if coefficient == "constant":
        A = H.P1ConstantLaplaceOperator(st, level - 1, level)
    else:
        k = [np.exp(np.sin(3.0 * orc.coords_of(lv)).sum(axis=1)) for lv in range(level + 1)]
        A = H.P1ElementwiseDivKGradOperator(st, level - 1, level, k[level - 1:])
        op = orc.op_divkgrad(k)
    if tables:
        u, f = H.P1Function("u", st, level - 1, level), H.P1Function("f", st, level - 1, level)
        H.GeometricMultigridSolver(st, A, level - 1, level).solve(u, f, level)
    rng = np.random.default_rng(cells + level)
    x, b = H.P1Function("x", st, level, level), H.P1Function("b", st, level, level)
    ref, rhs = rng.uniform(-1, 1, orc.n(level)), rng.uniform(-1, 1, orc.n(level))
    x.set(ref, level)
    b.set(rhs, level)
    it, conv = H.CGSolver(1e-30, 5).solve(A, x, b, level)
    orc.cg(ref, rhs, level, tol=1e-30, max_iter=5, op=op)
    assert (it, conv) == (5, False)
    assert np.abs(x.get(level) - ref).max() <= 1e-10 * np.abs(ref).max()
