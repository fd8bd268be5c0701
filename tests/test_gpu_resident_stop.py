"""Where the resident FP64 CG stops. An iteration that cuts the residual by eight
or nine digits leaves its norm below the rounding of |r|^2 - 2 a r.q + a^2 q.q, so
the decision must come from the new residual itself: right-hand sides within 1e-9
of the operator's largest eigenvector, solved to rtol 1e-10, on one CTA, on a
cluster and on a team that meets through global memory.

Tolerance: CG's residual ends at or below 1e-10 |b|; it differs from b - A u by a
few rounding errors of |A| |u|, which a right-hand side this close to the largest
eigenvector keeps below 1e-13 |b|."""
import numpy as np
import pytest
import scipy.sparse.linalg as sl

from oracle.fault import FaultElasticity as OracleFE
from oracle.operators import Grid3

pytestmark = pytest.mark.gpu


def project(b, n1, n2, n3):
    """b in the range of P exactly: zero far field, equal sides of the fault."""
    v = b.reshape(2, 3, n3, n2, n1).copy()
    v[:, :, 0] = v[:, :, -1] = 0.0
    v[:, :, :, 0] = v[:, :, :, -1] = 0.0
    v[0, ..., 0] = v[1, ..., -1] = 0.0
    v[0, ..., -1] = v[1, ..., 0] = 0.5 * (v[0, ..., -1] + v[1, ..., 0])
    return v.reshape(-1)


@pytest.mark.parametrize("n1,n2,n3,l_f", [(9, 9, 9, 0.5), (11, 11, 11, 0.4), (19, 11, 13, 0.4), (25, 15, 13, 0.2)],
                         ids=lambda v: str(v))
def test_first_step_cuts_the_residual_by_1e9(eqd, n1, n2, n3, l_f):
    L2, L3 = (n2 - 1) * 0.1, (n3 - 1) * 0.1
    if n1 == 9:
        L2 = L3 = 1.0
    gm = Grid3((-1.0, -L2, -L3), (0.0, L2, L3), (n1, n2, n3))
    gp = Grid3((0.0, -L2, -L3), (1.0, L2, L3), (n1, n2, n3))
    A = OracleFE(gm, gp, 2.0, 1.0, l_f=l_f).sys.A
    rng = np.random.default_rng(1)
    w, v = sl.eigsh(A, k=1, which="LM", v0=rng.standard_normal(A.shape[0]))
    v = project(v[:, 0], n1, n2, n3)
    v /= np.linalg.norm(v)
    B = np.empty((A.shape[0], 8))
    for j in range(8):
        x = project(rng.standard_normal(A.shape[0]), n1, n2, n3)
        B[:, j] = v + 1e-9 * x / np.linalg.norm(x)
    fe = eqd.FaultElasticity(eqd.GridPair(n1, n2, n3, 1.0, (-L2, L2), (-L3, L3)), 2.0, 1.0, l_f, precision="fp64")
    U = eqd.split_node_solve(fe.rs, B)
    for j in range(8):
        r1 = B[:, j] - A @ B[:, j] / w[0]
        assert 1e-10 < np.linalg.norm(r1) < 2e-9      # what one iteration leaves
        res = np.linalg.norm(A @ U[:, j] - B[:, j]) / np.linalg.norm(B[:, j])
        assert res < 1.01e-10, (j, res)
    assert fe.rs.stats.unconverged == 0
