"""`KMatrix.gemv_device` under stream capture: the first call with a given n * nvec may
allocate its scratch, so after one the same product is captured, also with y in the
place of s, which goes through that scratch. The replayed product is the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nvec", [(333, 1), (333, 2), (578, 64), (6000, 4)])
def test_capture_after_a_call_out_of_place(eqd, n, nvec):
    import torch
    rng = np.random.default_rng(n + nvec)
    M = eqd.KMatrix(rng.standard_normal((n, n)))
    S = torch.from_numpy(rng.standard_normal((nvec, n))).cuda()
    Y, T = torch.empty_like(S), S.clone()
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    M.gemv_device(S, Y, stream=st)
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        M.gemv_device(T, T, stream=st)
    T.copy_(S)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(T, Y)
    del g
    M.close()
