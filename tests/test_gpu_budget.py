"""What a slot costs of an HBM budget: 24 bytes a stored element in mixed precision (x in
FP64, d, r, p, q in FP32), 32 in FP64, whichever kernel runs the iterations, and 16
bytes a fault node and 1 KB beside them. A budget of exactly n such slots has room
for n; where the x1 march's padded lines would overdraw it, the grid streams
x1-fastest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K_TOL = 1e-8
ON_CHIP, STREAMED = (11, 11, 11), (10, 13, 11)    # no on-chip plan for lines of 10 points


def slot(n, nf, precision):
    n1, n2, n3 = n
    stored = 6 * n3 * ((n1 * n2 + 3) // 4 * 4)
    return stored * (24 if precision == "mixed" else 32) + 16 * nf + 1024


CASES = [(n, p, c, v) for n in (ON_CHIP, STREAMED) for p, c, v in (
    ("mixed", "none", 0), ("mixed", "jacobi", 0), ("mixed", "none", 2), ("fp64", "none", 0))]


@pytest.mark.parametrize("n,precision,precond,variant", CASES, ids=str)
def test_budget_of_one_slot(eqd, n, precision, precond, variant):
    fe = eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-1.0, 1.0), (-1.0, 1.0)), 2.0, 1.0, 1.0)
    kw = dict(precision=precision, precond=precond, variant=variant)
    cols = [0, fe.nf // 2, 2 * fe.nf - 1]
    K = eqd.stiffness_columns(fe, cols, solver=eqd.CGSolver(fe, **kw))[0]
    one = slot(n, fe.nf, precision)
    K1, _, st = eqd.stiffness_columns(fe, cols, solver=eqd.CGSolver(fe, hbm_budget_bytes=one, **kw))
    assert (st == 1).all()
    assert np.linalg.norm(K1 - K) <= 2 * K_TOL * np.linalg.norm(K)
    with pytest.raises(eqd.EqdError):
        eqd.stiffness_columns(fe, cols, solver=eqd.CGSolver(fe, hbm_budget_bytes=one - 1, **kw))


@pytest.mark.parametrize("n,precision,precond", [c[:3] for c in CASES if c[3] == 0], ids=str)
def test_server_budget(eqd, n, precision, precond):
    def grid():
        return eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-1.0, 1.0), (-1.0, 1.0)), 2.0, 1.0, 1.0)
    fe, ref = grid(), grid()
    seven = 7 * slot(n, fe.nf, precision)
    with eqd.Server(hbm_budget_bytes=seven, precision=precision, precond=precond) as srv:
        with pytest.raises(eqd.EqdError):
            srv.add(fe, slots=8)
        srv.add(fe, slots=7)
        K = srv.submit(fe, np.arange(10)).result(timeout=120)
    K0 = eqd.stiffness_columns(ref, np.arange(10), solver=eqd.CGSolver(ref, precision=precision, precond=precond))[0]
    assert np.linalg.norm(K - K0) <= 2 * K_TOL * np.linalg.norm(K0)
