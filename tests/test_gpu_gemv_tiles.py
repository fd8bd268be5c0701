"""The lines between the GEMV's row tiles (n = 6,656 and 13,312: 104 clusters of 64 and
of 128 rows) and between the GEMV and the blocked K S (`gemv_better`: 71 clusters
of groups of four vectors, odd n from 3,201 on, short waves up to n = 1,000 and
1,280).

Tolerance: as a row is a sum of n products in some order, (n + 1) 2^-53 sum |K| |s|
on each side of the comparison."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nvec", [
    (6655, 1), (6656, 2), (6657, 1), (6658, 2), (13312, 1), (13314, 2),
    (4544, 4), (4546, 3), (3199, 4), (3201, 3), (1136, 16), (1152, 16), (1000, 40), (1000, 41), (999, 20), (999, 24),
    (1280, 20), (1282, 20), (1280, 21)])
def test_products_on_both_sides(eqd, n, nvec):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + nvec)
    K = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)    # row c is column c of K
    S = torch.randn(nvec, n, generator=g, device="cuda", dtype=torch.float64)
    M = eqd.KMatrix(K.cpu().numpy().T)
    Y = torch.full_like(S, float("nan"))
    M.gemv_device(S, Y)
    torch.cuda.synchronize()
    bound = 2 * (n + 1) * 2.0 ** -53 * (S.abs() @ K.abs())
    assert bool(((Y - S @ K).abs() <= bound).all())
    T = S.clone()
    M.gemv_device(T, T)
    torch.cuda.synchronize()
    assert torch.equal(T, Y)
    M.close()
