"""Amplitudes of one slab at bars a few times what the form is good to, so that a dropped
block, a degree too few or a stale operand shows: thicknesses from one block to several and
to double-angle steps, square and wide order boxes above 128 orders (split planes in the mixed
form) and below.

FP64 against the slab equations with scipy's block exponential, 1e-11 of the largest amplitude
(two thousand terms of 2^-53, carried through up to 12 products and a solve with a condition
below 1000).  Mixed against the FP64 form, 2e-5 (2^-24 of a running sum at each of up to 20
steps, through the same), and M3D parameters of a clip, 3e-5 of the largest."""
import numpy as np
import pytest

from euvlitho_b200.config import preset
from tests.helpers import packed, random_mask, rel_err
from tests.test_gpu_amp_spectra import _reference

pytestmark = pytest.mark.gpu

TA = complex(0.95, 0.031) ** 2
DENSE = complex(0.87, 0.08) ** 2


@pytest.mark.parametrize("nx,ny,box", [(256, 256, 5), (320, 320, 6), (640, 272, 7)])
@pytest.mark.parametrize("eps,thick,pol", [
    (TA, (0.5,), "X"), (TA, (3.0,), "Y"), (TA, (7.5,), "X"), (TA, (15.0,), "Y"), (TA, (25.0,), "X"),
    (TA, (45.0,), "Y"), (TA, (60.0,), "X"), (TA, (60.0,), "Y"), (TA, (100.0,), "X"),
    (DENSE, (60.0,), "Y"), (TA, (7.5, 30.0, 20.0), "X"),
])
def test_one_slab(cuda, nx, ny, box, eps, thick, pol):
    import torch
    from euvlitho_b200.engine import Plan
    n = len(thick)
    cfg = preset("small").with_(ndivx=nx, ndivy=ny, lbox=box, mbox=box, eabs=(eps,) * n, dabs=thick,
                                refresh_sigma=n > 1)
    L, M = cfg.order_limits()
    mask = packed(random_mask(nx, ny, seed=5))
    got = {}
    for precision in ("fp64", "mixed"):
        plan = Plan(cfg, device=cuda, precision=precision, pols=(pol,))
        spec = plan.spectra(plan.as_mask_tensor(torch.from_numpy(mask[None])), 2 * L, 2 * M)
        hold = []
        kz = 2 * np.sqrt(cfg.k ** 2 - cfg.kx0 ** 2 - cfg.ky0 ** 2)
        d = plan.amp_desc(plan.orders, plan._t_l, plan._t_m, plan._f64([cfg.kx0]),
                          plan._f64([cfg.ky0]), plan._i32([0 if pol == "X" else 1]), plan._i32([0]),
                          plan._i32([[plan.pos[(0, 0)]]]), plan._f64([[kz]]), hold)
        ax = torch.empty((1, 1, plan.orders.n), dtype=torch.complex128, device=cuda)
        plan.run_amp(d, spec, ax)
        plan.check()
        got[precision] = ax[0, 0].cpu().numpy()
    F = spec.cpu().numpy().reshape(n, 4 * M + 1, 4 * L + 1).transpose(0, 2, 1)
    assert rel_err(got["fp64"], _reference(cfg, plan, pol, F, L, M)) < 1e-11
    assert rel_err(got["mixed"], got["fp64"]) < 2e-5


@pytest.mark.parametrize("nx,ny", [(400, 400), (512, 512)])
def test_mixed_m3d_parameters(cuda, nx, ny):
    import torch
    from euvlitho_b200.config import SimConfig
    from euvlitho_b200.engine import Plan
    cfg = SimConfig(ndivx=nx, ndivy=ny)
    masks = torch.from_numpy(np.stack([packed(random_mask(nx, ny, seed=s)) for s in range(2)]))
    r = {p: Plan(cfg, device=cuda, precision=p).m3d(masks) for p in ("fp64", "mixed")}
    top = float(torch.as_tensor(r["fp64"]["a0"]).abs().max())
    for key in ("a0", "ax", "ay"):
        d = torch.as_tensor(r["mixed"][key]) - torch.as_tensor(r["fp64"][key])
        assert float(d.abs().max()) / top < 3e-5, key
