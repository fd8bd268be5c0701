"""The resident CG (csrc/resident_cg.cuh), which runs a column's iterations on
one cluster of CTAs: K columns against the oracle (rtol 1e-13) on grids whose
tiles meet every case of the plan (one CTA, one row of tiles, both axes split,
tiles of three lines at the ends, lines of 9 to 25 points), mixed precision and
FP64, and a column alone against the same column in a batch, bit for bit.

Tolerance: the columns are solved to rtol 1e-10, and K's relative error stays
within the K bar of 1e-8 (the streamed engine measures 1e-11 to 4e-10)."""
import numpy as np
import pytest

from oracle.cref import CRefStiffness
from oracle.fault import FaultElasticity as OracleFE
from oracle.operators import Grid3

pytestmark = pytest.mark.gpu

K_TOL = 1e-8
RESIDENT = 11   # its index in the launch variants
# (n1, n2, n3, x1_extent, x2 half-width, x3 half-width, l_f, precisions)
CASES = [
    (9, 9, 9, 1.0, 1.0, 1.0, 0.5, ("mixed", "fp64")),          # one CTA
    (9, 10, 18, 0.8, 0.9, 1.7, 0.3, ("mixed", "fp64")),        # even axes, one of them split
    (9, 33, 17, 1.0, 1.6, 0.8, 0.3, ("mixed", "fp64")),        # more tiles along x2 than x3
    (11, 13, 21, 1.0, 1.2, 2.0, 0.4, ("mixed", "fp64")),
    (13, 15, 11, 1.0, 1.4, 1.0, 0.6, ("mixed", "fp64")),
    (15, 15, 13, 1.0, 1.4, 1.2, 0.4, ("mixed",)),
    (17, 17, 19, 1.0, 1.6, 1.8, 0.4, ("mixed",)),
    (21, 11, 13, 1.0, 1.0, 1.2, 0.4, ("mixed",)),
    (25, 15, 15, 1.0, 1.4, 1.4, 0.4, ("mixed",)),
]


def grids(eqd, c):
    n1, n2, n3, L1, L2, L3, l_f, _ = c
    gm = Grid3((-L1, -L2, -L3), (0.0, L2, L3), (n1, n2, n3))
    gp = Grid3((0.0, -L2, -L3), (L1, L2, L3), (n1, n2, n3))
    return gm, gp, eqd.GridPair(n1, n2, n3, L1, (-L2, L2), (-L3, L3))


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}x{c[2]}")
def test_resident_columns_match_oracle(eqd, case):
    l_f = case[6]
    gm, gp, g = grids(eqd, case)
    ofe = OracleFE(gm, gp, 2.0, 1.0, l_f=l_f)
    cols = np.unique(np.linspace(0, 2 * ofe.nf - 1, 7).astype(int))
    K_ref, _, ok = CRefStiffness(ofe).columns(cols, rtol=1e-13)
    assert ok.all()
    for precision in case[7]:
        fe = eqd.FaultElasticity(g, 2.0, 1.0, l_f, precision=precision)
        eqd.set_stencil_variant(fe, RESIDENT)
        K, it, st = eqd.stiffness_columns(fe, cols)
        assert (st == 1).all() and (it > 0).all()
        assert np.linalg.norm(K - K_ref) / np.linalg.norm(K_ref) < K_TOL, precision
        assert abs(K - K_ref).max() / abs(K_ref).max() < K_TOL, precision
        for j in (0, len(cols) - 1):
            K1, it1, _ = eqd.stiffness_columns(fe, [cols[j]])
            assert np.array_equal(K1[:, 0], K[:, j]) and it1[0] == it[j]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_resident_itmax_and_zero_slip(eqd, precision):
    """itmax ends the columns inside a launch; a zero slip needs no iteration."""
    fe = eqd.FaultElasticity(eqd.cube_grids(11), 2.0, 1.0, 0.4, precision=precision)
    eqd.set_stencil_variant(fe, RESIDENT)
    K, it, st = eqd.stiffness_columns(fe, [0, 7], solver=eqd.CGSolver(fe, precision=precision, itmax=5))
    assert (it == 5).all() and (st == eqd._abi.COL_MAXITER).all()
    z2, z3 = eqd.shear_traction(fe, np.zeros(fe.nf), np.zeros(fe.nf))
    assert (z2 == 0).all() and (z3 == 0).all()
