"""Explicit right-hand sides (`split_node_solve`) take the on-chip CG or the streamed
one each for itself: whether one is in the range of P decides for that one only,
and the width that memory or `chunk` allows decides nothing. A solution is the
same bits alone and in company."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(eqd, n, l_f):
    L = [(k - 1) * 0.1 for k in n[1:]]
    return eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-L[0], L[0]), (-L[1], L[1])), 2.0, 1.0, l_f, precision="fp64")


def in_range(eqd, fe, m, seed):
    x = np.random.default_rng(seed).standard_normal((fe.Ntot, m))
    return eqd.apply_operator(fe, x, mode="HP_DSAT")


@pytest.mark.parametrize("n,l_f", [((11, 11, 11), 0.4), ((25, 15, 13), 0.2)], ids=["cluster", "team"])
def test_company_out_of_range(eqd, n, l_f):
    fe = grid(eqd, n, l_f)
    b = in_range(eqd, fe, 3, 1)
    n1, n2, n3 = n
    out = b[:, 1].copy()
    out[(n3 // 2 * n2 + n2 // 2) * n1 + n1 - 1] += 1e-3 * np.abs(b).max()   # one side of a fault node
    B = np.column_stack([b[:, 0], out, b[:, 1], b[:, 2]])
    solver = eqd.CGSolver(fe, precision="fp64", itmax=12)
    U = eqd.split_node_solve(solver, B)
    assert solver.stats.solves == 4 and solver.stats.iterations == 48 and solver.stats.unconverged == 4
    for j in range(4):
        assert np.array_equal(U[:, j], eqd.split_node_solve(solver, B[:, j])), j


def test_team_limit_is_the_calls(eqd):
    """25 x 15 x 13: 13 and 11 lines in tiles of at most 4 (no bound at rows 5 and n - 5, three rows
    at least at the ends): four by four CTAs, so 148 // 16 = 9 teams and 36 right-hand sides."""
    fe = grid(eqd, (25, 15, 13), 0.2)
    b = in_range(eqd, fe, 37, 2)
    solver = eqd.CGSolver(fe, precision="fp64", itmax=12)
    streamed = eqd.CGSolver(fe, precision="fp64", itmax=12, variant=1)
    narrow = eqd.CGSolver(fe, precision="fp64", itmax=12, chunk=5)
    u36, u37 = eqd.split_node_solve(solver, b[:, :36]), eqd.split_node_solve(solver, b)
    s37 = eqd.split_node_solve(streamed, b)
    assert np.array_equal(u37, s37) and not np.array_equal(u36, s37[:, :36])
    for j in (0, 17, 35):
        assert np.array_equal(u36[:, j], eqd.split_node_solve(solver, b[:, j]))
    assert np.array_equal(u36, eqd.split_node_solve(narrow, b[:, :36]))
    assert np.array_equal(u37, eqd.split_node_solve(narrow, b))
