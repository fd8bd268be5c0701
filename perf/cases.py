"""What this framework is used for, as cases that can be timed.

A case is a dict of plain values. `prepare` makes what a program has in hand
before the call (the grid handle, K on the device, slips), from a seed;
`run` is one pass through the public entry points; `exact` is the same result
in 64 bits from plain torch and numpy; `work` is what the result cannot do
without. `listed` names the cases, `draw` gives more of the same ranges.

Grids are the BP8 ones (`bp8_grids`: h, L_fault, L_normal) or the reference
tests' cubes (`cube_grids`). The material is drawn around mu = 32.04 GPa,
nu = 0.25, so that grids of two seeds have different operators.
"""
import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@functools.lru_cache(maxsize=None)
def package():
    """The `earthquakediffinitive.jl_b200` directory, imported as `eqd_b200`."""
    if "eqd_b200" not in sys.modules:
        here = os.path.join(ROOT, "earthquakediffinitive.jl_b200")
        spec = importlib.util.spec_from_file_location("eqd_b200", os.path.join(here, "__init__.py"),
                                                      submodule_search_locations=[here])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["eqd_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["eqd_b200"]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def bp8(name, kind, h, L_normal, l_f, ncols=0, precision="mixed"):
    c = dict(kind=kind, n1=int(round(L_normal / h)) + 1, n23=int(round(1600 / h)) + 1, L_normal=float(L_normal),
             L_fault=800.0, l_f=float(l_f), ncols=int(ncols), precision=precision)
    return dict(c, name=name) if name else c


def cube(name, kind, n, nodes, ncols=0, precision="mixed"):
    """n^3 nodes a side on [-1, 1]^2, Omega_f the middle 2 * nodes + 1 nodes each way (n odd)."""
    c = dict(kind=kind, n1=n, n23=n, L_normal=1.0, L_fault=1.0, l_f=2.0 * nodes / (n - 1), ncols=int(ncols),
             precision=precision)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The time loop's K s with one slip vector on the smallest resident K (h = 100 m, whole fault plane).
        dict(name="ks_578_1", kind="ks", n=578, nvec=1),
        # K S for an ensemble of slips (64 vectors).
        dict(name="ks_4356_64", kind="ks", n=4356, nvec=64),
        # The time loop's K s on the K of h = 20 m (1.38 GB).
        dict(name="ks_13122_1", kind="ks", n=13122, nvec=1),
        # One right-hand side evaluation of the coupled time loop at h = 50 m (host state in, host state out).
        dict(name="rhs_1089", kind="rhs", side=33),
        # A small request of the serving mix: three columns on the h = 100 m grid.
        bp8("columns_h100_3", "columns", 100, 800, 800, 3),
        # The response to one slip distribution (`shear_traction`) at h = 50 m.
        bp8("traction_h50_1", "traction", 50, 400, 800, 1),
        # `build_model`'s default K: the ten Toeplitz solves at h = 50 m, l_f = 400 m, and their expansion.
        bp8("toeplitz_h50", "toeplitz", 50, 400, 400),
        # One explicit right-hand side, FP64 (`split_node_solve`), on an odd cube.
        cube("solve_cube25", "solve", 25, 6, 1, "fp64"),
        # The whole K at h = 100 m (578 columns).
        bp8("exact_h100", "exact", 100, 800, 800),
        # The whole K at h = 50 m (2,178 columns).
        bp8("exact_h50", "exact", 50, 400, 800),
        # A block of K's columns at h = 20 m (0.83 M DOF).
        bp8("columns_h20_96", "columns", 20, 400, 800, 96),
        # The near-diagonal solves at h = 25 m, L = 1600 / 800 m (3.3 M DOF a column).
        dict(name="columns_h25_10", kind="columns", n1=33, n23=129, L_normal=800.0, L_fault=1600.0, l_f=1600.0,
             ncols=10, precision="mixed"),
    ]


# Grids a drawn case may take: (h, L_normal) of the BP8 ones, L_fault = 800 m.
DRAWN_BP8 = [(100, 800), (80, 800), (50, 400), (50, 800), (40, 400), (40, 800), (32, 800), (25, 400), (20, 400)]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ks", "rhs", "columns", "columns", "columns", "traction", "toeplitz", "exact", "solve"])
    if kind == "ks":
        n = _log_uniform(rng, 300, 13122)
        return dict(kind="ks", n=n, nvec=_log_uniform(rng, 1, 64) if n < 6000 else rng.choice([1, 2, 3, 4]))
    if kind == "rhs":
        return dict(kind="rhs", side=rng.randrange(9, 60))
    if kind == "solve":
        return cube(None, "solve", 2 * rng.randrange(4, 15) + 1, 3, rng.choice([1, 1, 2, 3]), "fp64")
    if kind == "exact":
        n = 2 * rng.randrange(4, 10) + 1
        return cube(None, "exact", n, rng.randrange(2, (n - 1) // 2), 0, rng.choice(["mixed", "mixed", "fp64"]))
    h, L_normal = rng.choice(DRAWN_BP8)
    g = bp8(None, kind, h, L_normal, 800 if kind != "toeplitz" else 400 if 400 % h == 0 else 480 if h == 80 else 384)
    if kind == "toeplitz":
        return g
    # At most the column-iterations x DOF of 64 columns at h = 20 m.
    most = 64 * _cg_points(bp8(None, kind, 20, 400, 800)) / _cg_points(g)
    if kind == "traction":
        return dict(g, ncols=rng.choice([1, 1, 2, 4, 8]))
    fp64 = rng.random() < 0.3
    ncols = _log_uniform(rng, 1, max(1, min(512, 2 * g["n23"] ** 2, most / (4 if fp64 else 1))))
    return dict(g, ncols=ncols, precision="fp64" if fp64 else "mixed")


def _iterations(c):
    """About how many CG iterations a column takes at rtol 1e-10 (measured: 147 at n23 = 33, 320 at n23 = 81)."""
    return 60 + 3.2 * max(c["n1"], c["n23"])


def _cg_points(c):
    return 2.0 * c["n1"] * c["n23"] ** 2 * _iterations(c)


def _fault_nodes(c):
    h = 2 * c["L_fault"] / (c["n23"] - 1)
    return (2 * int(round(c["l_f"] / h)) + 1) ** 2


def _ncols(c):
    return {"exact": 2 * _fault_nodes(c), "toeplitz": 10}.get(c["kind"], c["ncols"])


def work(c):
    if c["kind"] == "ks":
        n, v = c["n"], c["nvec"]
        return {"bytes": 8.0 * n * n + 16.0 * n * v, "flops": 2.0 * n * n * v}
    if c["kind"] == "rhs":
        nf = c["side"] ** 2
        return {"bytes": 8.0 * (2 * nf) ** 2 + 64.0 * nf + 60.0 * nf, "flops": 2.0 * (2 * nf) ** 2 + 1000.0 * nf}
    nf, ncols = _fault_nodes(c), _ncols(c)
    dof = 6.0 * c["n1"] * c["n23"] ** 2
    io = {"solve": 16.0 * dof * ncols, "traction": 32.0 * nf * ncols, "toeplitz": 8.0 * (2 * nf) ** 2}
    # Per point and iteration: nine second and six first derivatives of 5 and 4 points, and the CG vectors.
    return {"bytes": io.get(c["kind"], 16.0 * nf * ncols), "flops": 150.0 * _cg_points(c) * ncols}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _material(c, seed):
    """(lambda, mu) of this seed: around 32.04 GPa and nu = 0.25, or the tests' 2 and 1 on the cubes."""
    r = np.random.default_rng([seed, 1])
    mu = (32.04e9 if c["L_fault"] > 10 else 1.0) * r.uniform(0.9, 1.1)
    nu = r.uniform(0.22, 0.28)
    return 2 * mu * nu / (1 - 2 * nu), mu


def _columns(c, seed):
    nf = _fault_nodes(c)
    return np.random.default_rng([seed, 2]).choice(2 * nf, size=min(c["ncols"], 2 * nf), replace=False).astype(np.int32)


def _slips(c, seed):
    """Smooth slip patches (a few Gaussians of random place, width and size), nf x ncols for x2 and x3."""
    r = np.random.default_rng([seed, 3])
    m = int(round(math.sqrt(_fault_nodes(c))))
    ax = np.linspace(-1, 1, m)
    x2, x3 = np.tile(ax, m), np.repeat(ax, m)
    out = np.zeros((2, m * m, c["ncols"]))
    for j in range(c["ncols"]):
        for d in range(2):
            for _ in range(3):
                a, b, w, s = r.uniform(-0.5, 0.5), r.uniform(-0.5, 0.5), r.uniform(0.2, 0.6), r.normal()
                out[d, :, j] += s * np.exp(-((x2 - a) ** 2 + (x3 - b) ** 2) / w ** 2)
    return out


def _stiffness_like(n, seed):
    """A dense n x n matrix with a negative dominant diagonal, Pa/m, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 11)
    K = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64).mul_(1e6)
    K.diagonal().sub_(4e8)
    return K


def _host(K):
    """The host's column-major copy of K, as Julia or `fault_stiffness` holds it."""
    return K.t().contiguous().cpu().numpy().T


def _rhs_inputs(c, seed):
    m = c["side"]
    nf = m * m
    r = np.random.default_rng([seed, 4])
    x = np.linspace(-800, 800, m)
    h2 = (x[1] - x[0]) ** 2
    X2, X3 = np.tile(x, m), np.repeat(x, m)
    # 0.05 m^2/s diffusion with zero-flux ends, five points.
    main = np.zeros(nf)
    rows, cols, vals = [], [], []
    idx = np.arange(nf).reshape(m, m)
    for a, b in ((idx[:, :-1], idx[:, 1:]), (idx[:-1], idx[1:])):
        a, b = a.ravel(), b.ravel()
        rows += [a, b]
        cols += [b, a]
        vals += [np.full(a.size, 0.05 / h2)] * 2
        np.add.at(main, a, -0.05 / h2)
        np.add.at(main, b, -0.05 / h2)
    rows, cols, vals = (np.concatenate(v) for v in (rows + [idx.ravel()], cols + [idx.ravel()], vals + [main]))
    u = np.concatenate([r.normal(size=2 * nf) * 1e-4,
                        math.log(1e4) + 0.3 * r.normal(size=nf),
                        1e6 * np.exp(-(X2 ** 2 + X3 ** 2) / 2e5) * (1 + 0.1 * r.normal(size=nf))])
    kw = dict(sigma0=25e6, sigma_min=1e5, eta=32.04e9 / (2 * 3464.0), tau0=(15e6, 1e5), q0=1.25e-6, beta=1e-8,
              phi=0.1, t_off=1e7)
    src = np.exp(-(X2 ** 2 + X3 ** 2) / (2 * 50.0 ** 2)) / (2 * np.pi * 50.0 ** 2)
    return (rows, cols, vals), u, kw, src, (0.016, 0.010, 0.5e-3, 1e-6, 0.6)


def _grid(c, seed):
    eqd = package()
    lam, mu = _material(c, seed)
    L = c["L_fault"]
    grids = eqd.GridPair(c["n1"], c["n23"], c["n23"], c["L_normal"], (-L, L), (-L, L))
    return eqd.FaultElasticity(grids, lam, mu, c["l_f"], precision=c["precision"])


def prepare(case, seed):
    eqd = package()
    kind = case["kind"]
    if kind == "ks":
        n, v = case["n"], case["nvec"]
        M = eqd.KMatrix(_host(_stiffness_like(n, seed)))
        g = torch.Generator(device="cuda").manual_seed(seed * 7 + 12)
        s = torch.randn((v, n), generator=g, device="cuda", dtype=torch.float64)
        return dict(case=case, M=M, s=s, y=torch.empty_like(s), stream=torch.cuda.current_stream())
    if kind == "rhs":
        import scipy.sparse as sp
        (rows, cols, vals), u, kw, src, fric = _rhs_inputs(case, seed)
        nf = case["side"] ** 2
        K = _host(_stiffness_like(2 * nf, seed))
        Ap = sp.csr_matrix((vals, (rows, cols)), shape=(nf, nf))
        return dict(case=case, rhs=eqd.BP8Rhs(K, Ap, eqd.FrictionParams(*fric), source=src, **kw), u=u)
    st = dict(case=case, fe=_grid(case, seed))
    if kind == "columns":
        st["cols"] = _columns(case, seed)
    elif kind == "traction":
        st["s2"], st["s3"] = _slips(case, seed)
    elif kind == "solve":
        chi = _chi(case, _slips(case, seed))
        st["b"] = eqd.apply_operator(st["fe"], chi.reshape(case["ncols"], -1).T, mode="HP_DSAT")
    return st


def run(state):
    eqd = package()
    kind = state["case"]["kind"]
    if kind == "ks":
        state["M"].gemv_device(state["s"], state["y"], stream=state["stream"])
        return state["y"]
    if kind == "rhs":
        return state["rhs"](state["u"], 1.0)
    fe = state["fe"]
    if kind == "columns":
        # (K columns; the iteration counts, which depend on how the FP32 sums round, stay out.)
        return eqd.stiffness_columns(fe, state["cols"])[0]
    if kind == "traction":
        return eqd.shear_traction(fe, state["s2"], state["s3"])
    if kind == "toeplitz":
        return eqd.fault_stiffness_toeplitz(fe)
    if kind == "exact":
        return eqd.fault_stiffness(fe)
    return eqd.split_node_solve(fe.rs, state["b"])


# ---------------------------------------------------------------------------
# The same results in 64 bits: dense 1D operators along each axis, plain CG
# ---------------------------------------------------------------------------
def _sbp(n, h):
    """Order-4 diagonal-norm SBP operators (Mattsson and Nordstrom 2004): weights, D1, D2, boundary derivative."""
    w, D1, D2 = np.ones(n), np.zeros((n, n)), np.zeros((n, n))
    w[:4] = np.array([17, 59, 43, 49]) / 48
    w[-4:] = w[3::-1]
    for i in range(4, n - 4):
        D1[i, i - 2:i + 3] = np.array([1, -8, 0, 8, -1]) / 12
        D2[i, i - 2:i + 3] = np.array([-1, 16, -30, 16, -1]) / 12
    c1 = [[-24 / 17, 59 / 34, -4 / 17, -3 / 34, 0, 0], [-1 / 2, 0, 1 / 2, 0, 0, 0],
          [4 / 43, -59 / 86, 0, 59 / 86, -4 / 43, 0], [3 / 98, 0, -59 / 98, 0, 32 / 49, -4 / 49]]
    c2 = [[2, -5, 4, -1, 0, 0], [1, -2, 1, 0, 0, 0], [-4 / 43, 59 / 43, -110 / 43, 59 / 43, -4 / 43, 0],
          [-1 / 49, 0, 59 / 49, -118 / 49, 64 / 49, -4 / 49]]
    for r in range(4):
        D1[r, :6], D2[r, :6] = c1[r], c2[r]
        D1[n - 1 - r, n - 6:] = -np.array(c1[r])[::-1]
        D2[n - 1 - r, n - 6:] = np.array(c2[r])[::-1]
    d = np.zeros(n)
    d[:4] = np.array([-11, 18, -9, 2]) / 6
    return w * h, D1 / h, D2 / h ** 2, d / h


class _Exact:
    """-H P (D + SAT) P on fields [column, side, component, x3, x2, x1], FP64 torch."""

    def __init__(self, c, seed):
        self.c, self.n = c, (c["n1"], c["n23"], c["n23"])
        self.lam, self.mu = _material(c, seed)
        h = (c["L_normal"] / (c["n1"] - 1),) + (2 * c["L_fault"] / (c["n23"] - 1),) * 2
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        ops = [_sbp(n, s) for n, s in zip(self.n, h)]
        self.D1, self.D2 = [t(o[1]) for o in ops], [t(o[2]) for o in ops]
        w = [t(o[0]) for o in ops]
        self.H = w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]
        self.sat = 0.5 / float(ops[0][0][0])
        self.d = t(ops[0][3])
        k = torch.ones(2, self.n[2], self.n[1], self.n[0], dtype=torch.float64, device=dev)
        k[:, 0], k[:, -1], k[:, :, 0], k[:, :, -1] = 0, 0, 0, 0
        k[0, :, :, 0], k[1, :, :, -1] = 0, 0
        self.keep, self.dev = k[:, None], dev
        self.m = int(round(math.sqrt(_fault_nodes(c))))
        self.o = (c["n23"] - self.m) // 2

    def along(self, M, v, a):
        if a == 0:
            return v @ M.T
        if a == 1:
            return M @ v
        return (M @ v.reshape(*v.shape[:-2], -1)).reshape(v.shape)

    def d1(self, v, a):
        return self.along(self.D1[a], v, a)

    def traction(self, v):
        """tau[column, side, component, x3, x2] on the fault, fixed +x1 axis."""
        f = torch.stack([v[:, 0, ..., -1], v[:, 1, ..., 0]], 1)
        dn = torch.stack([-(v[:, 0].flip(-1) @ self.d), v[:, 1] @ self.d], 1)
        g1 = torch.stack([v[:, 0, 0] @ self.D1[0][-1], v[:, 1, 0] @ self.D1[0][0]], 1)
        D2, D3 = self.D1[1], self.D1[2]
        t1 = self.lam * (g1 + f[:, :, 1] @ D2.T + D3 @ f[:, :, 2]) + 2 * self.mu * dn[:, :, 0]
        t2 = self.mu * (f[:, :, 0] @ D2.T + dn[:, :, 1])
        t3 = self.mu * (D3 @ f[:, :, 0] + dn[:, :, 2])
        return torch.stack([t1, t2, t3], 2)

    def P(self, v):
        v = v * self.keep
        a = 0.5 * (v[:, 0, ..., -1] + v[:, 1, ..., 0])
        v[:, 0, ..., -1] = a
        v[:, 1, ..., 0] = a
        return v

    def HPD(self, v):
        G = [self.d1(v[:, :, k], k) for k in range(3)]
        S = (self.lam + self.mu) * (G[0] + G[1] + G[2])
        w = torch.empty_like(v)
        for j in range(3):
            y = self.d1(S - self.mu * G[j], j)
            for a in range(3):
                y += self.along(self.D2[a], v[:, :, j], a) * (self.mu * (2 if a == j else 1))
            w[:, :, j] = y
        t = self.traction(v)
        s = self.sat * (t[:, 1] - t[:, 0])
        w[:, 0, ..., -1] += s
        w[:, 1, ..., 0] += s
        return self.P(w) * self.H

    def chi(self, s2, s3):
        """Fields of slips [column, nf]."""
        n1, n2, n3 = self.n
        v = torch.zeros(s2.shape[0], 2, 3, n3, n2, n1, dtype=torch.float64, device=self.dev)
        b = slice(self.o, self.o + self.m)
        for k, s in ((1, s2), (2, s3)):
            f = s.reshape(-1, self.m, self.m) / 2
            v[:, 0, k, b, b, -1] = -f
            v[:, 1, k, b, b, 0] = f
        return v

    def solve(self, b):
        """CG from zero to a relative residual of 1e-13."""
        dot = lambda x, y: (x * y).flatten(1).sum(1)  # noqa: E731
        x, r, p = torch.zeros_like(b), b.clone(), b.clone()
        rr = dot(r, r)
        stop, col = rr * 1e-26, (slice(None),) + (None,) * 5
        for _ in range(3000):
            if bool((rr <= stop).all()):
                break
            q = -self.HPD(p)
            al = torch.where(rr > stop, rr / dot(p, q), torch.zeros_like(rr))
            al = torch.nan_to_num(al)
            x += al[col] * p
            r -= al[col] * q
            new = dot(r, r)
            be = torch.nan_to_num(new / rr)
            rr = new
            p = r + be[col] * p
        return x

    def response(self, s2, s3):
        """Fault-averaged shear traction of the slips, [column, 2 nf]."""
        out = []
        per = max(1, int(4e8 / (6 * self.n[0] * self.n[1] * self.n[2])))
        for k in range(0, s2.shape[0], per):
            chi = self.chi(s2[k:k + per], s3[k:k + per])
            t = self.traction(self.solve(self.HPD(chi)) + chi).mean(1)
            f = slice(self.o, self.o + self.m)
            out.append(t[:, 1:, f, f].flatten(1))
        return torch.cat(out)

    def unit(self, cols):
        nf = self.m * self.m
        e = torch.zeros(len(cols), 2 * nf, dtype=torch.float64, device=self.dev)
        e[torch.arange(len(cols)), torch.as_tensor(np.asarray(cols), dtype=torch.long)] = 1.0
        return self.response(e[:, :nf], e[:, nf:]).T


def _chi(c, slips):
    """Reference-layout vectors [column, DOF] that hold -+ s / 2 at the fault nodes of Omega_f."""
    n1, n, m = c["n1"], c["n23"], int(round(math.sqrt(_fault_nodes(c))))
    v = np.zeros((slips.shape[2], 2, 3, n, n, n1))
    b = slice((n - m) // 2, (n - m) // 2 + m)
    for k in (0, 1):
        f = slips[k].T.reshape(-1, m, m) / 2
        v[:, 0, k + 1, b, b, -1] = -f
        v[:, 1, k + 1, b, b, 0] = f
    return v


def _exact_toeplitz(E):
    m, nf = E.m, E.m * E.m
    mid = (m + 1) // 2 - 1
    src = [(mid, mid), (0, 0), (m - 1, 0), (0, m - 1), (m - 1, m - 1)]
    R = E.unit([c for a, b in src for c in (b * m + a, nf + b * m + a)]).cpu().numpy()
    K = np.zeros((2 * nf, 2 * nf))
    a, b = np.tile(np.arange(m), m), np.repeat(np.arange(m), m)
    da, db = a[:, None] - a[None, :], b[:, None] - b[None, :]
    todo = np.ones((nf, nf), bool)
    for s, (sa, sb) in enumerate(src):
        ia, ib = sa + da, sb + db
        hit = todo & (ia >= 0) & (ia < m) & (ib >= 0) & (ib < m)
        node = (ib * m + ia)[hit]
        i, j = np.nonzero(hit)
        for d in range(2):
            K[i, d * nf + j] = R[node, 2 * s + d]
            K[nf + i, d * nf + j] = R[nf + node, 2 * s + d]
        todo &= ~hit
    return K


def _exact_rhs(c, seed):
    (rows, cols, vals), u, kw, src, (a, b, Dc, Vs, fs) = _rhs_inputs(c, seed)
    nf = c["side"] ** 2
    K = _stiffness_like(2 * nf, seed)
    dt = (K @ torch.tensor(u[:2 * nf], device="cuda")).cpu().numpy()
    phi, p = u[2 * nf:3 * nf], u[3 * nf:]
    T2, T3 = kw["tau0"][0] + dt[:nf], kw["tau0"][1] + dt[nf:]
    T, sig = np.hypot(T2, T3), np.maximum(kw["sigma0"] - p, kw["sigma_min"])
    C = np.exp((fs + b * np.log(Vs * np.exp(phi) / Dc)) / a)
    x = np.full(nf, math.log(1e-9))
    for _ in range(200):  # Newton in ln V for T = eta V + sigma a asinh(V C / (2 V*))
        V = np.exp(x)
        w = V / (2 * Vs) * C
        g = kw["eta"] * V + sig * a * np.arcsinh(w) - T
        x -= np.clip(g / (kw["eta"] * V + sig * a * w / np.sqrt(1 + w * w)), -5, 5)
    V = np.exp(x)
    dp = np.zeros(nf)
    np.add.at(dp, rows, vals * p[cols])
    dp += kw["q0"] / (kw["beta"] * kw["phi"]) * src
    return np.concatenate([V * T2 / T, V * T3 / T, np.exp(-phi) - V / Dc, dp])


def exact(case, seed):
    kind = case["kind"]
    if kind == "ks":
        g = torch.Generator(device="cuda").manual_seed(seed * 7 + 12)
        s = torch.randn((case["nvec"], case["n"]), generator=g, device="cuda", dtype=torch.float64)
        return s @ _stiffness_like(case["n"], seed).T
    if kind == "rhs":
        return _exact_rhs(case, seed)
    E = _Exact(case, seed)
    if kind == "toeplitz":
        return _exact_toeplitz(E)
    if kind == "exact":
        return E.unit(range(2 * E.m * E.m)).cpu().numpy()
    if kind == "columns":
        return E.unit(_columns(case, seed)).cpu().numpy()
    if kind == "traction":
        s = torch.tensor(_slips(case, seed), device=E.dev)
        t = E.response(s[0].T.contiguous(), s[1].T.contiguous()).T.cpu().numpy()
        nf = E.m * E.m
        return t[:nf], t[nf:]
    chi = torch.tensor(_chi(case, _slips(case, seed)), device=E.dev)
    return E.solve(E.HPD(chi)).flatten(1).T.cpu().numpy()
