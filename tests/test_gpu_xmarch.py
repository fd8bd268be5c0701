"""The x1-march FP32 apply and the streamed iteration on x2-fastest vectors
(csrc/xmarch.cuh, launch variant 12) against the oracle: the operator on grids
whose tiles meet every case (one tile, narrower last tiles, several tiles both
ways, the shortest and even axes, odd row padding), K, and batch independence.

The operator's bound is the one of the other FP32 variants, 2e-5 of |A||x|;
K's is the K bar, 1e-8."""
import numpy as np
import pytest

from oracle.cref import CRefStiffness
from oracle.fault import FaultElasticity as OracleFE, cube_grids
from oracle.operators import Grid3, SplitNodeSystem

pytestmark = pytest.mark.gpu

XMARCH = 12
MU = 32.04e9
CASES = [
    (9, 17, 21, 0.8, (-1.6, 1.6), (-2.0, 2.0), 1.5, 0.7, 0.0),
    (12, 10, 9, 1.0, (-1, 1), (-1, 1), 2.0, 1.0, 1.0),
    (21, 33, 13, 2.0, (-1, 1), (-1, 1), 2.0, 1.0, 0.5),
    (33, 17, 13, 800.0, (-400, 400), (-300, 300), MU, MU, 200.0),
    (9, 41, 33, 1.0, (-1, 1), (-1, 1), 2.0, 1.0, 0.5),
    (10, 38, 27, 1.0, (-1, 1), (-1, 1), 2.0, 1.0, 1.0),
]


@pytest.mark.parametrize("c", CASES, ids=lambda c: f"{c[0]}x{c[1]}x{c[2]}")
def test_xmarch_operator_matches_oracle(eqd, c):
    n1, n2, n3, L1, x2, x3, lam, mu, l_f = c
    S = SplitNodeSystem(Grid3((-L1, x2[0], x3[0]), (0.0, x2[1], x3[1]), (n1, n2, n3)),
                        Grid3((0.0, x2[0], x3[0]), (L1, x2[1], x3[1]), (n1, n2, n3)), lam, mu)
    fe = eqd.FaultElasticity(eqd.GridPair(n1, n2, n3, L1, x2, x3), lam, mu, l_f)
    eqd.set_stencil_variant(fe, XMARCH)
    X = S.P @ np.random.default_rng(5).standard_normal((S.Ntot, 3))
    Y = eqd.apply_operator(fe, X, mode="A_rangeP", precision="mixed")
    for j in range(3):
        err = abs(Y[:, j] - S.A @ X[:, j]).max() / abs(S.A).dot(abs(X[:, j])).max()
        assert err < 2e-5, (j, err)
    assert abs(S.P @ Y - Y).max() == 0.0
    y1 = eqd.apply_operator(fe, X[:, 1], mode="A_rangeP", precision="mixed")
    assert np.array_equal(Y[:, 1], y1)


@pytest.mark.parametrize("n, l_f", [(11, 0.4), (13, 0.5), (25, 0.25)])
def test_xmarch_K_matches_oracle(eqd, n, l_f):
    gm, gp = cube_grids(n)
    ofe = OracleFE(gm, gp, 2.0, 1.0, l_f=l_f)
    cols = np.unique(np.linspace(0, 2 * ofe.nf - 1, 9).astype(int))
    K_ref, _, ok = CRefStiffness(ofe).columns(cols, rtol=1e-13)
    assert ok.all()
    fe = eqd.FaultElasticity(eqd.cube_grids(n), 2.0, 1.0, l_f)
    eqd.set_stencil_variant(fe, XMARCH)
    K, it, st = eqd.stiffness_columns(fe, cols)
    assert (st == 1).all()
    assert np.linalg.norm(K - K_ref) / np.linalg.norm(K_ref) < 1e-8
    assert abs(K - K_ref).max() / abs(K_ref).max() < 1e-8
    # alone, and with fewer slots than columns: the same bits
    K1, it1, _ = eqd.stiffness_columns(fe, [cols[3]])
    assert np.array_equal(K1[:, 0], K[:, 3]) and it1[0] == it[3]
    Kf, itf, _ = eqd.stiffness_columns(fe, cols, solver=eqd.CGSolver(fe, chunk=4))
    assert np.array_equal(Kf, K) and np.array_equal(itf, it)


def test_xmarch_split_equals_one_chain(eqd):
    """Two halves on two streams (64 columns and more) against one chain."""
    fe = eqd.FaultElasticity(eqd.cube_grids(13, L=1.2), 2.0, 1.0, 0.6)
    eqd.set_stencil_variant(fe, XMARCH)
    cols = np.arange(2 * fe.nf)
    Ks, its, _ = eqd.stiffness_columns(fe, cols)
    K1, it1, _ = eqd.stiffness_columns(fe, cols, solver=eqd.CGSolver(fe, split=False))
    assert len(cols) >= 64 and np.array_equal(Ks, K1) and np.array_equal(its, it1)
