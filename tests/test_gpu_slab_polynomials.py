"""The slab polynomials of ampS (degree, blocks and double-angle steps chosen from
the configuration) at the ends of their range: slices of no thickness, one block,
several blocks, double-angle steps, orders near grazing, a single order, strong
and vanishing absorber contrast, one to three slices.

Tolerance: FP64 1e-8 relative as the other parity tests (the polynomials are
truncated below 1e-16); mixed 5e-4, the bar of the mixed amplitudes."""
import numpy as np
import pytest

from euvlitho_b200.config import SimConfig, preset
from oracle import euv_oracle as O
from tests.helpers import flat_bits, packed, random_mask, rel_err, to_oracle

pytestmark = pytest.mark.gpu

TA = complex(0.95, 0.031) ** 2
DENSE = complex(0.87, 0.08) ** 2


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-8), ("mixed", 5e-4)])
@pytest.mark.parametrize("period,box,eabs,dabs,refresh,pol", [
    (256, 5, (TA,), (0.0,), False, "X"),            # c = 1, s = 0
    (256, 5, (TA,), (1.0,), False, "Y"),            # one block
    (256, 0, (TA,), (60.0,), False, "X"),           # a single order
    (128, 4, (TA,), (60.0,), False, "Y"),           # near grazing, a wide ellipse
    (256, 5, (DENSE,), (90.0,), False, "X"),        # strong contrast
    (128, 4, (DENSE,), (150.0,), False, "X"),       # double-angle steps
    (256, 5, (complex(1.0, 1e-9),), (60.0,), False, "X"),  # no contrast
    (256, 5, (TA, DENSE), (30.0, 2.0), False, "Y"),  # slices of different degree
    (256, 5, (TA, DENSE, TA), (20.0, 45.0, 7.5), True, "X"),
    (256, 5, (DENSE, TA), (40.0, 12.0), True, "Y"),
])
def test_amp_over_the_polynomials_range(cuda, precision, tol, period, box, eabs, dabs, refresh, pol):
    import torch
    from euvlitho_b200.engine import Plan
    cfg = preset("small").with_(ndivx=period, ndivy=period, lbox=box, mbox=box, eabs=eabs, dabs=dabs,
                                refresh_sigma=refresh)
    plan = Plan(cfg, device=cuda, precision=precision, pols=(pol,))
    m = random_mask(period, period, seed=11)
    ax, srcs = plan.amp(torch.from_numpy(packed(m)[None]), polar=pol)  # raises on a flagged unit
    ax = ax.cpu().numpy()
    oc = to_oracle(cfg)
    L, M = cfg.order_limits()
    ref = O.amp_s(pol, flat_bits(m), oc, plan.orders.lidx, plan.orders.midx, L, M, oc.kx0, oc.ky0)
    seen = 0
    for s, key in enumerate(srcs):
        if plan.pos.get(key) is not None:
            assert rel_err(ax[0, s], ref[key]) < tol, (key, rel_err(ax[0, s], ref[key]))
            seen += 1
    assert seen > 0


@pytest.mark.parametrize("n", [121, 257, 289, 300])
def test_mixed_gemm_block_order(cuda, n):
    """Sums of more than eight k-blocks run in the tile's own order (its columns'
    and rows' blocks last in the two accumulator sets): every block must enter
    once, for tile counts around the block and tile edges.  Bound as for the other
    mixed GEMM tests, 3e-8 K + 1e-6 of max |C|."""
    import torch
    from euvlitho_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(2, n, n, dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn(2, n, n, dtype=torch.complex128, device="cuda", generator=g)
    C = torch.empty_like(A)
    wb = L.lib().euv_zgemm_mixed_workspace_bytes(n, n, n, 2)
    ws = torch.empty(wb, dtype=torch.uint8, device="cuda")
    L.call("euv_zgemm_mixed", n, n, n, L.c64(1, 0), None, A.data_ptr(), n, n * n, B.data_ptr(), n,
           n * n, L.c64(0, 0), C.data_ptr(), n, n * n, L.c64(0, 0), 2, None, 0, ws.data_ptr(), wb,
           None, torch.cuda.current_stream().cuda_stream)
    # column-major operands: the tensors hold the transposes
    ref = torch.matmul(B, A)
    assert float((C - ref).abs().max() / ref.abs().max()) < 3e-8 * n + 1e-6
