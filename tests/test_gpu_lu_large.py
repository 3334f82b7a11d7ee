"""LU beyond the one-launch solve and the portable cluster size: the blocked
triangular solves (above N = 1562 with more than eight right-hand sides), panels of
more than 2048 rows (clusters of sixteen CTAs), and the same orders with the few
right-hand sides that keep the one-launch solve.

Tolerance 1e-10 of the largest solution value, as the other LU tests."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs,batch", [(1563, 9, 2), (1601, 33, 2), (1601, 8, 1), (2049, 1, 1),
                                          (2085, 40, 2), (31, 9, 3), (64, 12, 1)])
def test_factor_and_solve(cuda, n, nrhs, batch):
    import torch
    from euvlitho_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(n)
    s = torch.cuda.current_stream().cuda_stream
    A = torch.randn(batch, n, n, dtype=torch.complex128, device="cuda", generator=g)
    X = torch.randn(batch, nrhs, n, dtype=torch.complex128, device="cuda", generator=g)
    ref = torch.linalg.solve(A.transpose(1, 2), X.transpose(1, 2)).transpose(1, 2)
    W = A.clone()
    piv = torch.empty(batch * n, dtype=torch.int32, device="cuda")
    info = torch.empty(batch, dtype=torch.int32, device="cuda")
    L.call("euv_lu_factor", n, W.data_ptr(), n, n * n, piv.data_ptr(), info.data_ptr(), batch, s)
    L.call("euv_lu_solve", n, nrhs, W.data_ptr(), n, n * n, piv.data_ptr(), X.data_ptr(), n, n * nrhs,
           batch, s)
    assert int(info.abs().max()) == 0
    assert float((X - ref).abs().max() / ref.abs().max()) < 1e-10
