"""The request server on the kernels that grids take when nothing is pinned: the
on-chip CG (a cluster to a column; FP64 at 17 points a line, a team of CTAs that takes
several columns in turn) and the x1 march. Fewer slots than columns, so that slots
refill while others are in flight, and requests of two grids at once: every K column
is the same bits, after the same iterations, as built alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = {
    "cluster": ((11, 11, 11), 0.8, 8),
    "cluster_tall": ((13, 17, 13), 0.5, 16),
    "x1_march": ((10, 21, 11), 0.8, 6),
    "x1_march_halves": ((12, 17, 17), 1.0, 64),     # from 64 slots on, two halves
    "team": ((17, 33, 33), 0.5, 13),                # FP64: 4 teams of 36 CTAs
}


def make(eqd, name, precision):
    n, l_f, slots = GRIDS[name]
    return eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-1.0, 1.0), (-1.0, 1.0)), 2.0, 1.0, l_f,
                               precision=precision), slots


@pytest.mark.parametrize("names,precision", [
    (("cluster", "x1_march"), "mixed"), (("cluster_tall", "x1_march_halves"), "mixed"),
    (("cluster", "cluster_tall"), "fp64"), (("team", "cluster"), "fp64")], ids=lambda v: "-".join(v) if isinstance(v, tuple) else v)
def test_default_paths_in_the_mix_equal_alone(eqd, names, precision):
    refs = [make(eqd, k, precision)[0] for k in names]
    rng = np.random.default_rng(7)
    with eqd.Server(hbm_budget_bytes=4 << 30, precision=precision) as srv:
        served = []
        for k in names:
            fe, slots = make(eqd, k, precision)
            srv.add(fe, slots=slots)
            served.append(fe)
        reqs = []
        for j in range(10):
            i = int(j % 3 == 0)
            n = int(rng.integers(1, min(2 * refs[i].nf, 70)))
            cols = rng.choice(2 * refs[i].nf, size=n, replace=False)
            reqs.append((srv.submit(served[i], cols), refs[i], cols))
        got = [r.result(timeout=300) for r, _, _ in reqs]
        infos = [r.info() for r, _, _ in reqs]
    for K, inf, (_, ref, cols) in zip(got, infos, reqs):
        alone = [eqd.stiffness_columns(ref, [c]) for c in cols[:3]]
        for j, (K1, _, _) in enumerate(alone):
            assert np.array_equal(K[:, j], K1[:, 0])
        K_all, it, _ = eqd.stiffness_columns(ref, cols)
        assert np.array_equal(K, K_all)
        assert inf["unconverged"] == 0 and inf["iterations"] == int(it.sum())


def test_teams_take_columns_in_turn(eqd):
    """More columns than teams, of unequal iteration counts: the halo and the sums that a team
    keeps are those of its current column."""
    fe, _ = make(eqd, "team", "fp64")
    cols = np.unique(np.linspace(0, 2 * fe.nf - 1, 19).astype(int))
    K, it, st = eqd.stiffness_columns(fe, cols)
    assert (st == 1).all() and len(set(it.tolist())) > 1
    for j, c in enumerate(cols):
        K1, it1, _ = eqd.stiffness_columns(fe, [c])
        assert np.array_equal(K1[:, 0], K[:, j]) and it1[0] == it[j]


@pytest.mark.parametrize("n,team", [((17, 33, 33), True), ((17, 49, 17), False), ((17, 65, 33), False)],
                         ids=["fills", "too_few_lines", "too_few_teams"])
def test_columns_take_teams_that_fill_the_device(eqd, n, team):
    """`team_fills`: 25 own lines an SM in four teams at least. Other grids stream their columns,
    and their explicit right-hand sides keep the team."""
    L = [(k - 1) / 16 for k in n[1:]]
    fe = eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-L[0], L[0]), (-L[1], L[1])), 2.0, 1.0, 0.5, precision="fp64")
    short, streamed = (eqd.CGSolver(fe, precision="fp64", itmax=20, variant=v) for v in (0, 1))
    cols = [fe.nf // 2, fe.nf + 3]
    K, Ks = (eqd.stiffness_columns(fe, cols, solver=s)[0] for s in (short, streamed))
    assert np.array_equal(K, Ks) == (not team)
    b = eqd.apply_operator(fe, np.random.default_rng(1).standard_normal(fe.Ntot), mode="HP_DSAT")
    assert not np.array_equal(eqd.split_node_solve(short, b), eqd.split_node_solve(streamed, b))
