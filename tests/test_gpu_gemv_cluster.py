"""The one-pass GEMV (`gemv_kernel`): a cluster of eight CTAs to 64, 128 or 256 rows,
whose sums meet in shared memory. Edges of the row tiles and of the column
shares, fewer columns than CTAs, the changes of tile at n = 7,104 and 14,208, 8-byte loads
(odd n, K at an 8-byte offset), groups of 1, 2 and 4 vectors, more groups than
one grid dimension holds, and y in the place of s.

Tolerance: a row is a sum of n products whose terms are added in some order, so
its error is at most (n + 1) 2^-53 sum |K| |s| on each side of the comparison."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gemv_static(eqd, n, K, S, Y):
    import torch
    eqd._abi.check(eqd._abi.lib().eqd_kmat_gemv_static(
        C.c_int32(0), C.c_int32(n), C.c_void_p(K.data_ptr()), C.c_void_p(S.data_ptr()), C.c_void_p(Y.data_ptr()),
        C.c_int32(S.shape[0]), C.c_void_p(torch.cuda.current_stream().cuda_stream)))


@pytest.mark.parametrize("n,nvec,offset", [
    (1, 1, 0), (2, 3, 0), (7, 2, 0), (63, 1, 0), (64, 5, 0), (65, 2, 0), (129, 4, 1), (130, 1, 1), (578, 1, 0),
    (1090, 2, 0), (7103, 1, 0), (7104, 2, 0), (7105, 1, 0), (7106, 3, 0),
    (7234, 1, 1), (14210, 1, 0), (2, 262144, 0)])
def test_gemv_sizes(eqd, n, nvec, offset):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    buf = torch.randn(n * n + offset, generator=g, device="cuda", dtype=torch.float64)
    K = buf[offset:].view(n, n)       # row c is column c of the column-major matrix
    S = torch.randn(nvec, n, generator=g, device="cuda", dtype=torch.float64)
    Y = torch.full_like(S, float("nan"))
    gemv_static(eqd, n, K, S, Y)
    ref = S @ K
    bound = 2 * (n + 1) * 2.0 ** -53 * (S.abs() @ K.abs())
    assert bool(((Y - ref).abs() <= bound).all())
    one = torch.empty_like(S[-1:])
    gemv_static(eqd, n, K, S[-1:].clone(), one)
    assert torch.equal(one[0], Y[-1])
    T = S.clone()
    gemv_static(eqd, n, K, T, T)
    assert torch.equal(T, Y)


def test_gemv_nonfinite_stays_in_its_rows(eqd):
    import torch
    n = 200
    K = torch.ones(n, n, device="cuda", dtype=torch.float64)
    K[3, 77] = float("inf")
    K[5, 130] = float("nan")
    S = torch.ones(1, n, device="cuda", dtype=torch.float64)
    Y = torch.empty_like(S)
    gemv_static(eqd, n, K, S, Y)
    y = Y[0].cpu().numpy()
    assert np.isposinf(y[77]) and np.isnan(y[130])
    assert (np.delete(y, [77, 130]) == n).all()


@pytest.mark.parametrize("nvec", [1, 2])
def test_kmat_gemv_in_place(eqd, nvec):
    import torch
    n = 333
    rng = np.random.default_rng(0)
    K = rng.standard_normal((n, n))
    M = eqd.KMatrix(K)
    S = torch.from_numpy(rng.standard_normal((nvec, n))).cuda()
    Y = torch.empty_like(S)
    M.gemv_device(S, Y)
    torch.cuda.synchronize()
    M.gemv_device(S, S)
    torch.cuda.synchronize()
    assert torch.equal(S, Y)
    M.close()
