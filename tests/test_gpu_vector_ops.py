"""Vector operations and canonical-order transfers of P1 functions against numpy, at closure
sizes that fill, exceed and fall short of the kernels' blocks (4 points to 6545 per cell)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [0, 1, 2, 4, 5])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_vector_operations_match_numpy(level, dtype):
    import hyb_inputs
    import hyteg_b200 as H

    st = H.PrimitiveStorage.cuboid(2, 1, 1, level)
    hd, nd, eps = (H.F64, np.float64, 1e-15) if dtype == "f64" else (H.F32, np.float32, 6e-8)
    n, xyz = st.num_dofs(level), st.dof_coords(level)
    inner = ((xyz > 1e-12) & (xyz < 1 - 1e-12)).all(axis=1)
    masks = {H.ALL: np.ones(n, bool), H.INNER | H.NEUMANN: inner, H.DIRICHLET: ~inner}
    rng = np.random.default_rng(level)
    v = [rng.uniform(-1, 1, n).astype(nd) for _ in range(3)]
    f = [H.P1Function("f", st, level, level, hd) for _ in range(4)]
    for fi, vi in zip(f, v):
        fi.set(vi, level)
        assert np.array_equal(fi.get(level), vi)
    # the device-side fill depends on positions alone: checks the canonical order itself
    f[3].fill_uniform_random(level, 7, 2 << level)
    assert np.array_equal(f[3].get(level), hyb_inputs.uniform_rhs(xyz, 7, 2 << level).astype(nd))
    for flag, mask in masks.items():
        start = rng.uniform(-1, 1, n).astype(nd)
        for k in range(1, 4):
            sc = [0.5, -1.25, 3.0][:k]
            want = sum(s * x.astype(np.float64) for s, x in zip(sc, v))
            f[3].set(start, level)
            f[3].assign(sc, f[:k], level, flag)
            got = f[3].get(level)
            assert np.abs(got - want)[mask].max(initial=0) <= 8 * eps * 5
            assert np.array_equal(got[~mask], start[~mask])
            f[3].set(start, level)
            f[3].add(sc, f[:k], level, flag)
            assert np.abs(f[3].get(level) - (start.astype(np.float64) + want))[mask].max(initial=0) <= 8 * eps * 6
        f[3].set(start, level)
        f[3].assign([2.0, 1.0], [f[3], f[0]], level, flag)  # the destination among the sources
        assert np.abs(f[3].get(level) - (2.0 * start.astype(np.float64) + v[0]))[mask].max(initial=0) <= 8 * eps * 3
        f[3].set(start, level)
        f[3].interpolate(1.5, level, flag)
        assert np.array_equal(f[3].get(level), np.where(mask, nd(1.5), start))
        want = float(np.dot(v[0].astype(np.float64)[mask], v[1].astype(np.float64)[mask]))
        assert abs(f[0].dot_global(f[1], level, flag) - want) <= 1e-13 * max(n, 10)
