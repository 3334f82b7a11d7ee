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


def _factor(A, s):
    import torch
    from euvlitho_b200 import _lib as L
    batch, n, _ = A.shape
    W = A.clone()
    piv = torch.empty(batch * n, dtype=torch.int32, device="cuda")
    info = torch.empty(batch, dtype=torch.int32, device="cuda")

    def run(stream):
        L.call("euv_lu_factor", n, W.data_ptr(), n, n * n, piv.data_ptr(), info.data_ptr(), batch,
               stream)
    run(s)
    return W, piv.view(batch, n), info, run


@pytest.mark.parametrize("n", [33, 64, 97, 300, 450])
def test_factor_alone_and_in_a_batch(cuda, n):
    """Trailing updates of one wave run before the next panel, larger ones beside it:
    one matrix takes the first form, twenty-four of them the second (from n = 97 on);
    the operations on each element are the same."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    s = torch.cuda.current_stream().cuda_stream
    A = torch.randn(24, n, n, dtype=torch.complex128, device="cuda", generator=g)
    W, piv, info, _ = _factor(A, s)
    assert int(info.abs().max()) == 0
    for b in (0, 23):
        w1, p1, _, _ = _factor(A[b:b + 1], s)
        assert torch.equal(p1[0], piv[b]) and torch.equal(w1[0], W[b])


@pytest.mark.parametrize("n,batch", [(300, 1), (450, 24)])
def test_factor_under_capture(cuda, n, batch):
    """Both forms recorded in a CUDA graph and replayed."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(batch, n, n, dtype=torch.complex128, device="cuda", generator=g)
    W, piv, info, run = _factor(A, torch.cuda.current_stream().cuda_stream)
    ref, rp = W.clone(), piv.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        W.copy_(A)
        piv.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert int(info.abs().max()) == 0
        assert torch.equal(W, ref) and torch.equal(piv, rp)
