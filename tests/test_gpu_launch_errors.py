"""An error of a launch that is recorded into the graph of CG iterations ends the
call (a graph without that kernel would leave its columns where they are, and the
host waiting for them), and the next call on the grid runs normally. The error is
made on the host (`eqd_test_inject_failure`). So does an error while a grid's plan
is made, and the next call makes the plan: the grid does not change to another
kernel for its later calls."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EQD_FAIL_CG_LAUNCH = 1
EQD_FAIL_PLAN = 2
ON_CHIP = (11, 11, 11)
STREAMED = (10, 11, 11)     # no on-chip plan for lines of 10 points


@pytest.mark.parametrize("ncols", [4, 64])     # 64: recorded as two halves on two streams
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [ON_CHIP, STREAMED], ids=["on_chip", "streamed"])
def test_failed_launch_ends_the_call(eqd, n, precision, ncols):
    def grid():
        return eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-1.0, 1.0), (-1.0, 1.0)), 2.0, 1.0, 0.6,
                                   precision=precision)
    cols = np.arange(ncols)
    fe = grid()
    lib = eqd._abi.lib()
    eqd._abi.check(lib.eqd_test_inject_failure(fe.handle, C.c_int32(EQD_FAIL_CG_LAUNCH)))
    with pytest.raises(eqd.EqdError) as e:
        eqd.stiffness_columns(fe, cols)
    assert e.value.code == eqd._abi.EQD_ERR_CUDA and "recording" in str(e.value)
    K, it, st = eqd.stiffness_columns(fe, cols)
    assert (st == 1).all()
    K0, it0, _ = eqd.stiffness_columns(grid(), cols)
    assert np.array_equal(K, K0) and np.array_equal(it, it0)


@pytest.mark.parametrize("n,precision", [
    (ON_CHIP, "mixed"), (ON_CHIP, "fp64"), ((17, 33, 19), "mixed"), ((17, 33, 19), "fp64"), (STREAMED, "mixed")],
    ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_failed_plan_is_made_again(eqd, n, precision):
    def grid():
        return eqd.FaultElasticity(eqd.GridPair(*n, 1.0, (-1.0, 1.0), (-1.0, 1.0)), 2.0, 1.0, 1.0,
                                   precision=precision)
    cols = np.arange(5)
    fe = grid()
    eqd._abi.check(eqd._abi.lib().eqd_test_inject_failure(fe.handle, C.c_int32(EQD_FAIL_PLAN)))
    with pytest.raises(eqd.EqdError):
        eqd.stiffness_columns(fe, cols)
    K, it, st = eqd.stiffness_columns(fe, cols)
    assert (st == 1).all()
    other = grid()
    K0, it0, _ = eqd.stiffness_columns(other, cols)
    assert np.array_equal(K, K0) and np.array_equal(it, it0)
    if precision == "mixed":
        assert eqd.autotune(fe, 0)[0] == eqd.autotune(other, 0)[0] == (12 if n == STREAMED else 11)


def test_rejects_unknown_failures(eqd):
    fe = eqd.FaultElasticity(eqd.cube_grids(9), 2.0, 1.0, 0.5)
    assert eqd._abi.lib().eqd_test_inject_failure(fe.handle, C.c_int32(0)) == eqd._abi.EQD_ERR_ARG
