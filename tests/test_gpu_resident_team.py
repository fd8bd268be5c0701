"""The resident CG of FP64 grids beyond 13 points a line: columns on one cluster
(15 to 19 points), and on a team of CTAs that meets through global memory (17
points, and a few explicit right-hand sides up to 29), against the oracle (rtol
1e-13); and explicit right-hand sides outside the range of P, which stay on the
streamed path.

Tolerance: solved to rtol 1e-10, within the K bar of 1e-8 of the oracle's; the
residual of an explicit solve is twice rtol at most (CG's own residual, summed
anew each iteration, ends below rtol)."""
import numpy as np
import pytest

from oracle.cref import CRefStiffness
from oracle.fault import FaultElasticity as OracleFE
from oracle.operators import Grid3

pytestmark = pytest.mark.gpu

K_TOL = 1e-8
STREAMED = 0
# (n1, n2, n3, half-width x2, half-width x3, l_f)
CASES = [
    (15, 13, 21, 1.2, 2.0, 0.4),
    (17, 17, 15, 1.6, 1.4, 0.4),
    (17, 33, 19, 3.2, 1.8, 0.4),   # 17 points: no cluster holds it
    (19, 11, 13, 1.0, 1.2, 0.4),
    (21, 15, 21, 1.4, 2.0, 0.4),  # uneven tiles
    (23, 11, 19, 1.0, 1.8, 0.4),  # 23, 27 and 29 points: the last part of a line is shorter
    (25, 15, 13, 1.4, 1.2, 0.2),
    (27, 14, 12, 1.3, 1.1, 0.3),
    (29, 15, 11, 1.4, 1.0, 0.2),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}x{c[2]}")
def test_fp64_resident(eqd, case):
    n1, n2, n3, L2, L3, l_f = case
    gm = Grid3((-1.0, -L2, -L3), (0.0, L2, L3), (n1, n2, n3))
    gp = Grid3((0.0, -L2, -L3), (1.0, L2, L3), (n1, n2, n3))
    g = eqd.GridPair(n1, n2, n3, 1.0, (-L2, L2), (-L3, L3))
    ofe = OracleFE(gm, gp, 2.0, 1.0, l_f=l_f)
    fe = eqd.FaultElasticity(g, 2.0, 1.0, l_f, precision="fp64")
    cols = np.unique(np.linspace(0, 2 * ofe.nf - 1, 5).astype(int))
    K_ref, _, ok = CRefStiffness(ofe).columns(cols, rtol=1e-13)
    assert ok.all()
    K, it, st = eqd.stiffness_columns(fe, cols)
    assert (st == 1).all()
    assert np.linalg.norm(K - K_ref) / np.linalg.norm(K_ref) < K_TOL
    K1, it1, _ = eqd.stiffness_columns(fe, [cols[-1]])
    assert np.array_equal(K1[:, 0], K[:, -1]) and it1[0] == it[-1]

    rng = np.random.default_rng(n1)
    chi = rng.standard_normal((fe.Ntot, 2))
    b = eqd.apply_operator(fe, chi, mode="HP_DSAT")
    u = eqd.split_node_solve(fe.rs, b)
    for j in range(2):
        res = np.linalg.norm(eqd.apply_operator(fe, u[:, j]) - b[:, j]) / np.linalg.norm(b[:, j])
        assert res < 2e-10, (j, res)
    assert np.array_equal(eqd.split_node_solve(fe.rs, b[:, 0]), u[:, 0])

    # Outside the range of P by one fault node: the streamed path, bit for bit.
    c = b[:, 0].copy()
    node = (n3 // 2 * n2 + n2 // 2) * n1
    c[node + n1 - 1] += 1e-3 * np.abs(b).max()
    solver = eqd.CGSolver(fe, precision="fp64", itmax=12)
    u0 = eqd.split_node_solve(solver, c)
    eqd.set_stencil_variant(fe, STREAMED)
    assert np.array_equal(u0, eqd.split_node_solve(solver, c))
    # In its range: the streamed path ends within the same bar.
    us = eqd.split_node_solve(fe.rs, b)
    assert np.linalg.norm(us - u) / np.linalg.norm(us) < 2 * K_TOL
