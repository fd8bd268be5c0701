"""`autotune` times mixed precision and chooses for mixed precision: FP64 solves of the
grid keep their kernel, where it is the on-chip one too (lines of 19 points have an
FP64 plan and no FP32 one, so the tuner's choice is a streamed variant). A variant
that the caller pins holds for both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_autotune_leaves_fp64_alone(eqd):
    fe = eqd.FaultElasticity(eqd.GridPair(19, 11, 13, 1.0, (-1.0, 1.0), (-1.2, 1.2)), 2.0, 1.0, 0.4)
    fp64 = eqd.CGSolver(fe, precision="fp64")
    cols = [0, 7, 2 * fe.nf - 1]
    K, it, _ = eqd.stiffness_columns(fe, cols, solver=fp64)
    b = eqd.apply_operator(fe, np.random.default_rng(3).standard_normal(fe.Ntot), mode="HP_DSAT")
    u = eqd.split_node_solve(fp64, b)
    assert eqd.autotune(fe, 16)[0] != 11
    K2, it2, _ = eqd.stiffness_columns(fe, cols, solver=fp64)
    assert np.array_equal(K2, K) and np.array_equal(it2, it)
    assert np.array_equal(eqd.split_node_solve(fp64, b), u)
    eqd.set_stencil_variant(fe, 0)
    assert not np.array_equal(eqd.stiffness_columns(fe, cols, solver=fp64)[0], K)
