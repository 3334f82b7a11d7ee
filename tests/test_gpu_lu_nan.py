"""Pivots of a matrix with NaN entries: a NaN is no pivot beside a number, in panels of every
cluster size and in those beyond; with nothing else in a column the factorisation goes on with
its first row.  Pivots are compared, so there is no tolerance."""
import pytest

pytestmark = pytest.mark.gpu


def _pivots(A):
    import torch
    from euvlitho_b200 import _lib as L
    n = A.shape[-1]
    W = A.clone()
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.empty(1, dtype=torch.int32, device="cuda")
    L.call("euv_lu_factor", n, W.data_ptr(), n, n * n, piv.data_ptr(), info.data_ptr(), 1,
           torch.cuda.current_stream().cuda_stream)
    return piv.cpu()


@pytest.mark.parametrize("n", [1, 7, 40, 256, 300, 900, 1700, 3000, 4100])
@pytest.mark.parametrize("part", ["re", "im", "both"])
def test_nan_is_no_pivot(cuda, n, part):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g)  # column-major
    rows = sorted({0, n // 3, n - 1})[:max(1, min(3, n - 1))]
    nan, one = float("nan"), 1.0
    value = {"re": complex(nan, one), "im": complex(one, nan), "both": complex(nan, nan)}[part]
    for r in rows:
        A[0, r] = value
    size = A[0].real.abs() + A[0].imag.abs()
    want = int(torch.where(size.isnan(), torch.zeros_like(size), size).argmax()) if n > 1 else 0
    assert int(_pivots(A)[0]) == want


@pytest.mark.parametrize("n", [40, 900, 3000])
def test_column_of_nan(cuda, n):
    import torch
    A = torch.full((n, n), float("nan"), dtype=torch.complex128, device="cuda")
    p = _pivots(A)
    assert bool((p == torch.arange(n, dtype=torch.int32)).all())
