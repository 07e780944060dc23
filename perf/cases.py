"""Performance cases of the P1 geometric-multigrid path.

Each case is work that a program built on this library does through its public Python binding
(a ctypes layer over the C ABI): solves to a tolerance, single multigrid cycles, smoothing,
Krylov steps, grid transfers, the curved-shell operator and a batch of served requests. Every
pass ends with the results in the caller's own device (served requests: host) memory in the
canonical DoF order, as a caller needs them.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  mesh, operator, functions and inputs of a case
    run(state)           one pass
    work(case)           bytes and flops one pass cannot do without
    exact(case, seed)    the pass's outputs in plain 64-bit torch, where there is such a value
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyteg-vara_b200", "python"))
import hyteg_b200 as H  # noqa: E402

FLAG = H.INNER | H.NEUMANN  # the unknowns of a solve


def listed():
    return [
        # the smallest call: one operator application on the six-tet cube, where launches count
        _case("apply", "apply_f64_cube1_l3", 1, 1, 1, 3),
        # one V(3,3) cycle used as a preconditioner on the CPU-sized reference problem (levels 0..5)
        _case("cycle", "cycle_f64_cube1_l5", 1, 1, 1, 5),
        # whole solve in double precision, ordinary size
        _case("solve", "solve_f64_cube2_l6", 2, 2, 2, 6, precision=64),
        # the headline solve: 48 macro-tets, 17 M unknowns, FP32 cycles in FP64 refinement
        _case("solve", "solve_mixed_cube2_l7", 2, 2, 2, 7, precision=32),
        # variable (lognormal) coefficient, 384 macro-tets: the heterogeneous-medium solve
        _case("solve", "solve_mixed_lognormal_cube4_l6", 4, 4, 4, 6, precision=32, coefficient="lognormal"),
        # pre-smoothing of a V(3,3) cycle on the finest level, double precision
        _case("smooth", "smooth_f64_cube2_l7", 2, 2, 2, 7),
        # a symmetric smoother (forward, then backward sweeps) in single precision
        _case("smooth", "smooth_symmetric_f32_cube4_l6", 4, 4, 4, 6, precision=32, symmetric=True),
        # smoothing with the variable coefficient on an elongated box
        _case("smooth", "smooth_lognormal_f64_box123_l6", 1, 2, 3, 6, coefficient="lognormal"),
        # one step of a user's own conjugate-gradient loop on the finest level
        _case("cg_step", "cg_step_f64_cube4_l6", 4, 4, 4, 6),
        # grid transfers between the two finest levels, both directions
        _case("transfer", "transfer_f64_box343_l6", 3, 4, 3, 6),
        # the curved-shell (blending) operator on the reference's spherical-shell mesh
        _case("shell", "shell_apply_f64_720_l4", 3, 4, 0, 4),
        # several small requests arriving together at the serving loop, mixed shapes and coefficients
        _case("serve", "serve_12_mixed", 2, 2, 2, 5, requests=12),
    ]


def _case(kind, name, nx, ny, nz, level, precision=64, coefficient="constant", symmetric=False, requests=0):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "level": level, "precision": precision, "coefficient": coefficient,
         "symmetric": symmetric, "requests": requests}
    if name:
        c["name"] = name
    return c


def draw(rng):
    kind = rng.choice(["apply", "cycle", "solve", "solve", "smooth", "smooth", "cg_step", "transfer", "shell", "serve"])
    if kind == "shell":
        return _case(kind, None, 3, rng.choice([2, 3, 4, 5]), 0, rng.choice([2, 3, 4]), coefficient=rng.choice(["constant", "radial"]))
    if kind == "serve":
        return _case(kind, None, rng.randint(1, 3), rng.randint(1, 2), rng.randint(1, 2), rng.choice([3, 4, 5]), requests=rng.randint(2, 12))
    variable = kind in ("solve", "smooth", "cycle", "apply") and rng.random() < 0.4
    most = 8.5e6 if variable else 17.0e6  # DoFs of the largest level
    while True:
        n = [rng.randint(1, 4) for _ in range(3)]
        level = rng.randint(2, 7)
        if n[0] * n[1] * n[2] * 8 ** level <= most:
            break
    return _case(kind, None, *n, level, precision=rng.choice([64, 32]), coefficient="lognormal" if variable else "constant",
                 symmetric=kind == "smooth" and rng.random() < 0.5)


# ---------------------------------------------------------------------------- inputs
def _uniform(seed, stream, n):
    """U[-1, 1) values: right-hand sides and iterates as the benchmark problems draw them."""
    return np.random.default_rng([seed, stream]).uniform(-1.0, 1.0, n)


def _field(seed, corr_len=0.2, modes=64):
    """Random Fourier features of a Gaussian random field of correlation length corr_len."""
    r = np.random.default_rng([seed, 99])
    return r.normal(0.0, 1.0 / corr_len, (modes, 3)), r.uniform(0.0, 2.0 * np.pi, modes)


def _dtype(case):
    return (H.F64, torch.float64) if case["precision"] == 64 else (H.F32, torch.float32)


def _function(st, name, level, dtype, values=None, inner_only=False, min_level=None):
    f = H.P1Function(name, st, level if min_level is None else min_level, level, dtype)
    if values is not None:
        t = torch.as_tensor(values).to(device="cuda", dtype=torch.float64 if dtype == H.F64 else torch.float32)
        f.set_device(t.data_ptr(), level)
        torch.cuda.synchronize()  # t is released on return
        if inner_only:
            f.interpolate(0.0, level, H.DIRICHLET)
    return f


def _operator(case, st, level, seed):
    if case["coefficient"] == "lognormal":
        w, ph = _field(seed)
        return H.P1ElementwiseDivKGradOperator.random_features(st, 0, level, w, ph, 1.0)
    return H.P1ConstantLaplaceOperator(st, 0, level)


def _requests(case, seed):
    """The request mix of a serving case: cubes up to nx, levels 3..level, both coefficients."""
    out = []
    for i in range(case["requests"]):
        c = (1 + i % case["nx"], 1 + i % case["ny"], 1 + (i // 2) % case["nz"])
        level = 3 + i % (case["level"] - 2)
        coeff = H.COEFF_LOGNORMAL if i % 3 == 1 else H.COEFF_CONSTANT
        out.append((H.Server.request(*c, level, coeff, 32 if i % 4 else 64, seed * 1000 + i), _box_dofs(*c, level)))
    return out


def prepare(case, seed):
    kind, L = case["kind"], case["level"]
    s = {"kind": kind, "level": L, "case": case}
    if kind == "serve":
        s["server"] = H.Server(40 << 30, max_active=16, max_level=L)
        s["requests"] = _requests(case, seed)
        run(s)  # a serving process keeps the meshes and hierarchies of earlier requests
        return s
    if kind == "shell":
        st = H.PrimitiveStorage.spherical_shell(case["nx"], case["ny"], 0.55, 1.0, L)
        s["A"] = H.P1ElementwiseBlendingDivKGradOperator(st, L, L, 5.0 if case["coefficient"] == "radial" else 0.0)
        n, hd, td = st.num_dofs(L), H.F64, torch.float64
    else:
        st = H.PrimitiveStorage.cuboid(case["nx"], case["ny"], case["nz"], L)
        n = st.num_dofs(L)
        hd, td = (H.F64, torch.float64) if kind in ("solve", "cycle") else _dtype(case)
        if kind != "transfer":
            s["A"] = _operator(case, st, L, seed)
    s["st"] = st
    new = lambda values=None, inner=False: _function(st, "f", L, hd, values, inner)  # noqa: E731
    out = lambda lvl=L: torch.empty(st.num_dofs(lvl), dtype=td, device="cuda")  # noqa: E731
    if kind in ("solve", "cycle"):
        s["x"] = _function(st, "x", L, H.F64, min_level=0)
        s["b"] = _function(st, "b", L, H.F64, _uniform(seed, 1, n), min_level=0)
        s["gmg"] = H.GeometricMultigridSolver(st, s["A"], 0, L, 3, 3, 1.0, coarse_tol=1e-12)
        s["out"] = out()
    elif kind in ("apply", "shell"):
        s["x"], s["y"], s["out"] = new(_uniform(seed, 1, n)), new(), out()
    elif kind == "smooth":
        s["x0"], s["b"], s["x"], s["out"] = new(_uniform(seed, 1, n), True), new(_uniform(seed, 2, n)), new(), out()
    elif kind == "cg_step":
        s["x"], s["r"], s["p"] = (new(_uniform(seed, k, n), True) for k in (1, 2, 3))
        s["ap"], s["x1"], s["r1"], s["p1"] = (new() for _ in range(4))
        s["out"] = [out() for _ in range(3)]
    elif kind == "transfer":
        s["r"] = _function(st, "r", L, hd, _uniform(seed, 1, n), min_level=L - 1)
        s["e"] = _function(st, "e", L, hd, min_level=L - 1)
        t = torch.as_tensor(_uniform(seed, 2, st.num_dofs(L - 1))).to(device="cuda", dtype=td)
        s["e"].set_device(t.data_ptr(), L - 1)
        s["out"] = [out(L - 1), out()]
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------- one pass
def run(s):
    kind, L = s["kind"], s["level"]
    if kind == "solve":
        s["x"].interpolate(0.0, L)
        history = s["gmg"].solve_to_tolerance(s["x"], s["b"], L, 1e-8, 60, s["case"]["precision"])
        s["x"].get_device(s["out"].data_ptr(), L)
        return {"x": s["out"], "cycles": len(history) - 1}
    if kind == "cycle":
        s["x"].interpolate(0.0, L)
        s["gmg"].solve(s["x"], s["b"], L)
        s["x"].get_device(s["out"].data_ptr(), L)
        return s["out"]
    if kind in ("apply", "shell"):
        s["A"].apply(s["x"], s["y"], L, FLAG)
        s["y"].get_device(s["out"].data_ptr(), L)
        return s["out"]
    if kind == "smooth":
        s["x"].assign([1.0], [s["x0"]], L)
        for _ in range(3):
            s["A"].smooth_sor(s["x"], s["b"], 1.0, L, FLAG)
            if s["case"]["symmetric"]:
                s["A"].smooth_sor_backwards(s["x"], s["b"], 1.0, L, FLAG)
        s["x"].get_device(s["out"].data_ptr(), L)
        return s["out"]
    if kind == "cg_step":
        s["A"].apply(s["p"], s["ap"], L, FLAG)
        rr, pap = s["r"].dot_global(s["r"], L, FLAG), s["p"].dot_global(s["ap"], L, FLAG)
        alpha = rr / pap
        s["x1"].assign([1.0, alpha], [s["x"], s["p"]], L, FLAG)
        s["r1"].assign([1.0, -alpha], [s["r"], s["ap"]], L, FLAG)
        rr1 = s["r1"].dot_global(s["r1"], L, FLAG)
        s["p1"].assign([1.0, rr1 / rr], [s["r1"], s["p"]], L, FLAG)
        for f, o in zip((s["x1"], s["r1"], s["p1"]), s["out"]):
            f.get_device(o.data_ptr(), L)
        return s["out"] + [rr, pap, rr1]
    if kind == "transfer":
        H.P1toP1LinearRestriction().restrict(s["r"], L, FLAG)
        H.P1toP1LinearProlongation().prolongate(s["e"], L - 1, FLAG)
        s["r"].get_device(s["out"][0].data_ptr(), L - 1)
        s["e"].get_device(s["out"][1].data_ptr(), L)
        return s["out"]
    ids = [s["server"].submit(r, keep_solution=True, num_dofs=n) for r, n in s["requests"]]
    s["server"].run()
    return [s["server"].solution(i) for i in ids] + [s["server"].result(i).cycles for i in ids]


# ---------------------------------------------------------------------------- necessary work
def _box_dofs(nx, ny, nz, level):
    return (nx * 2 ** level + 1) * (ny * 2 ** level + 1) * (nz * 2 ** level + 1)


def work(case):
    kind, L = case["kind"], case["level"]
    var = case["coefficient"] != "constant"
    if kind == "shell":
        nC = 60 * (case["nx"] - 1) ** 2 * (case["ny"] - 1)
        n = nC * 8 ** L / 6
        # apply and download; 690 flops per micro-tet row, 4 rows per micro-tet
        return {"bytes": 32 * n, "flops": 690 * 4 * nC * 8 ** L}
    if kind == "serve":
        one = [work(_case("solve", None, r.nx, r.ny, r.nz, r.level, r.precision,
                          "lognormal" if r.coefficient == H.COEFF_LOGNORMAL else "constant")) for r, _ in _requests(case, 0)]
        return {k: sum(w[k] for w in one) for k in ("bytes", "flops")}
    n, e = _box_dofs(case["nx"], case["ny"], case["nz"], L), case["precision"] / 8
    coef = e if var else 0.0  # the nodal coefficient is read with the stencil
    row = 250.0 if var else 30.0  # flops of one row of the operator
    if kind == "apply":
        return {"bytes": (4 * e + coef) * n, "flops": row * n}  # apply, then slab -> canonical order
    if kind == "smooth":
        sweeps = 6 if case["symmetric"] else 3
        return {"bytes": (sweeps * (3 * e + coef) + 4 * e) * n, "flops": sweeps * row * n}
    if kind == "cg_step":  # apply, three dots, three two-term assigns, three downloads
        return {"bytes": (2 + 4 + 9 + 6) * e * n, "flops": (row + 18) * n}
    if kind == "transfer":
        return {"bytes": (2 * (1 + 1 / 8) + 2 * (1 + 1 / 8)) * e * n, "flops": 6 * n}
    # one V(3,3) cycle: six sweeps, a residual, a restriction and a prolongation on every level
    c = case["precision"] / 8 if kind == "solve" else 8
    coef = c if var else 0.0
    cycle = 8 / 7 * ((6 * (3 * c + coef) + 3 * c + coef + 4.25 * c) * n)
    flops = 8 / 7 * (7 * row + 6) * n
    if kind == "cycle":
        return {"bytes": cycle + 16 * n, "flops": flops}
    cycles = 16 if var else 17
    norm = (16 + (8 if var else 0) + (24 if case["precision"] == 32 else 0)) * n  # FP64 residual norm, refinement update
    return {"bytes": cycles * (cycle + norm) + 16 * n, "flops": cycles * (flops + row * n)}


# ---------------------------------------------------------------------------- 64-bit results
_MICRO = (((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)), ((1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 0, 1)),
          ((1, 0, 0), (0, 1, 0), (1, 0, 1), (0, 0, 1)), ((1, 1, 0), (1, 1, 1), (0, 1, 1), (1, 0, 1)),
          ((1, 0, 1), (0, 1, 1), (0, 0, 1), (0, 1, 0)), ((0, 1, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1)))
_CUBE = ((4, 5, 7, 3), (0, 3, 1, 4), (4, 1, 5, 3), (5, 6, 7, 2), (1, 3, 2, 5), (7, 2, 3, 5))
_CORNER = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))


class _Grid:
    """The refined mesh of a box in plain torch: per macro-tet the canonical DoF of every
    micro-vertex, on an (N+1)^3 index grid (z, y, x) whose points outside the tet are masked."""

    def __init__(self, nx, ny, nz, level):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        vid = lambda i, j, k: (k * (ny + 1) + j) * (nx + 1) + i  # noqa: E731
        self.V = np.array([(i / nx, j / ny, k / nz) for k in range(nz + 1) for j in range(ny + 1) for i in range(nx + 1)])
        self.T = sorted({tuple(vid(i + _CORNER[m][0], j + _CORNER[m][1], k + _CORNER[m][2]) for m in t)
                         for k in range(nz) for j in range(ny) for i in range(nx) for t in _CUBE})
        N = self.N = 1 << level
        E = sorted({tuple(sorted(p)) for t in self.T for p in itertools.combinations(t, 2)})
        F = sorted({tuple(sorted(p)) for t in self.T for p in itertools.combinations(t, 3)})
        nf, nc = (N - 1) * (N - 2) // 2, (N - 1) * (N - 2) * (N - 3) // 6
        oE = len(self.V)
        oF = oE + len(E) * (N - 1)
        oC = oF + len(F) * nf
        self.n = oC + len(self.T) * nc
        eid, fid = {e: i for i, e in enumerate(E)}, {f: i for i, f in enumerate(F)}
        z, y, x = torch.meshgrid(*[torch.arange(N + 1, device=self.dev)] * 3, indexing="ij")
        b = torch.stack([N - x - y - z, x, y, z])
        self.inside = b[0] >= 0
        pos = b > 0
        self.ids = []
        for c, t in enumerate(self.T):
            ids = torch.full_like(x, -1)
            for k in range(4):
                ids[(b[k] == N) & self.inside] = t[k]
            for p in itertools.combinations(range(4), 2):
                p = sorted(p, key=lambda k: t[k])
                m = self.inside & pos[p[0]] & pos[p[1]] & (b[p[0]] + b[p[1]] == N)
                ids[m] = oE + eid[tuple(t[k] for k in p)] * (N - 1) + b[p[1]][m] - 1
            for p in itertools.combinations(range(4), 3):
                p = sorted(p, key=lambda k: t[k])
                m = self.inside & pos[p[0]] & pos[p[1]] & pos[p[2]] & (b[p[0]] + b[p[1]] + b[p[2]] == N)
                i, j = b[p[1]][m], b[p[2]][m]
                ids[m] = oF + fid[tuple(t[k] for k in p)] * nf + (j - 1) * (N - 1) - (j - 1) * j // 2 + i - 1
            m = self.inside & pos.all(0)
            ids[m] = oC + c * nc + torch.arange(nc, device=self.dev)  # x fastest, then y, then z
            self.ids.append(ids)
        P = self.positions()
        self.inner = ((P > 1e-12) & (P < 1 - 1e-12)).all(1)

    def positions(self):
        P = torch.zeros(self.n, 3, dtype=torch.float64, device=self.dev)
        z, y, x = torch.meshgrid(*[torch.arange(self.N + 1, device=self.dev, dtype=torch.float64)] * 3, indexing="ij")
        for t, ids in zip(self.T, self.ids):
            v = torch.as_tensor(self.V[list(t)], device=self.dev)
            X = v[0] + (x[..., None] * (v[1] - v[0]) + y[..., None] * (v[2] - v[0]) + z[..., None] * (v[3] - v[0])) / self.N
            P[ids[self.inside]] = X[self.inside]
        return P

    def _matrix(self, t, micro):
        X = self.V[t[0]] + np.array(micro) @ (self.V[list(t[1:])] - self.V[t[0]]) / self.N
        J = (X[1:] - X[0]).T
        g = np.linalg.inv(J)
        g = np.vstack([-g.sum(0), g])
        return abs(np.linalg.det(J)) / 6 * g @ g.T

    def apply(self, u, k=None):
        """The P1 stiffness matrix (element coefficient: mean of the nodal k) times u."""
        N, y = self.N, torch.zeros_like(u)
        for t, ids in zip(self.T, self.ids):
            at = ids.clamp(min=0)
            U, Y = u[at], torch.zeros(N + 1, N + 1, N + 1, dtype=u.dtype, device=self.dev)
            Kn = None if k is None else k[at]
            for micro in _MICRO:
                K, most = self._matrix(t, micro), max(sum(o) for o in micro)
                cut = lambda G, o: G[o[2]:N + o[2], o[1]:N + o[1], o[0]:N + o[0]]  # noqa: E731
                i = torch.arange(N, device=self.dev)
                w = ((i[:, None, None] + i[None, :, None] + i) <= N - most).to(u.dtype)
                if Kn is not None:
                    w = w * sum(cut(Kn, o) for o in micro) / 4
                for a in range(4):
                    cut(Y, micro[a]).add_(w * sum(float(K[a, b]) * cut(U, micro[b]) for b in range(4)))
            y.index_add_(0, ids[self.inside], Y[self.inside])
        return y

    def times_inner(self, u, k=None):
        return torch.where(self.inner, self.apply(u, k), torch.zeros_like(u))


def _interpolation(fine, coarse, c):
    """Coarse endpoints (weight 1/2 each) of every fine micro-vertex of macro-tet c."""
    N = fine.N
    z, y, x = torch.meshgrid(*[torch.arange(N + 1, device=fine.dev)] * 3, indexing="ij")
    px, py, pz = x & 1, y & 1, z & 1
    ox = torch.where(px == 1, torch.where((py | pz) == 1, -1, 1), 0)
    oy, oz = py.clone(), torch.where(pz == 1, torch.where((px & py) == 1, -1, 1), 0)
    oy = torch.where((py == 1) & (pz == 1) & (px == 0), -1, oy)
    m = fine.inside
    at = lambda s: coarse.ids[c][((z + s * oz) >> 1)[m], ((y + s * oy) >> 1)[m], ((x + s * ox) >> 1)[m]]  # noqa: E731
    return fine.ids[c][m], at(-1), at(1)


def exact(case, seed):
    kind, L = case["kind"], case["level"]
    if kind in ("cycle", "smooth", "shell", "serve"):
        return None  # defined by the solver's own sweep order, map or request mix
    n = _box_dofs(case["nx"], case["ny"], case["nz"], L)
    if kind == "solve" and n > 300000:
        return None
    g = _Grid(case["nx"], case["ny"], case["nz"], L)
    assert g.n == n
    td = torch.float64 if kind == "solve" else _dtype(case)[1]
    vec = lambda stream, m=n: torch.as_tensor(_uniform(seed, stream, m)).to(td).to(torch.float64).to(g.dev)  # noqa: E731
    inner = lambda v: torch.where(g.inner, v, torch.zeros_like(v))  # noqa: E731
    k = None
    if case["coefficient"] == "lognormal":
        w, ph = (torch.as_tensor(a, device=g.dev) for a in _field(seed))
        k = torch.cat([torch.exp(math.sqrt(2 / 64) * torch.cos(P @ w.T + ph).sum(1)) for P in g.positions().split(1 << 18)])
    if kind == "apply":
        return g.times_inner(vec(1), k)
    if kind == "cg_step":
        x, r, p = (inner(vec(i)) for i in (1, 2, 3))
        ap = g.times_inner(p)
        rr, pap = float(r @ r), float(p @ ap)
        x1, r1 = x + rr / pap * p, r - rr / pap * ap
        rr1 = float(r1 @ r1)
        return [x1, r1, r1 + rr1 / rr * p, rr, pap, rr1]
    if kind == "transfer":
        gc = _Grid(case["nx"], case["ny"], case["nz"], L - 1)
        r, e = vec(1), vec(2, gc.n)
        count = torch.zeros_like(r)
        rc, ef = torch.zeros_like(e), torch.zeros_like(r)
        maps = [_interpolation(g, gc, c) for c in range(len(g.T))]
        for f, _, _ in maps:
            count.index_add_(0, f, torch.ones_like(f, dtype=torch.float64))
        for f, a, b in maps:
            ef[f] = 0.5 * (e[a] + e[b])
            for end in (a, b):
                rc.index_add_(0, end, 0.5 * r[f] / count[f])
        return [torch.where(gc.inner, rc, torch.zeros_like(rc)), inner(ef)]
    b = inner(vec(1))  # solve: conjugate gradients on the unknowns, far below the case's tolerance
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), r @ r
    stop = 1e-26 * rr
    for _ in range(3000):
        ap = g.times_inner(p, k)
        a = rr / (p @ ap)
        x, r = x + a * p, r - a * ap
        new = r @ r
        if new <= stop:
            break
        p, rr = r + new / rr * p, new
    return {"x": x, "cycles": None}
