"""Mixed-precision images of clips whose order box is wide against a period: the powers of
the slab operator cancel there, so that the split products' rounding is multiplied unless
the slab takes double-angle steps and keeps the diagonals apart.

Bounds.  Image, root mean square of a mask's pixels relative to the FP64 form: 5e-6 (the
split products' running sums lose 2^-24 of themselves at each of up to 40 steps, about 1e-6,
carried through 7 to 11 products that do not amplify it).  The FP64 form itself against the
eigen-based oracle: 1e-11 of the largest amplitude (products of 1000 terms of 2^-53, and a
condition number below 100).  A unit's result next to units of another period: 1e-13."""
import ctypes as C

import numpy as np
import pytest

from euvlitho_b200.config import preset
from oracle import euv_oracle as O
from tests.helpers import flat_bits, packed, random_mask, rel_err, to_oracle

pytestmark = pytest.mark.gpu

TA = complex(0.95, 0.031) ** 2


def _config(nx, ny, box, slices, refresh=False):
    return preset("small").with_(ndivx=nx, ndivy=ny, lbox=box, mbox=box, max_sources=40,
                                 eabs=(TA,) * slices, dabs=(60.0 / slices,) * slices,
                                 refresh_sigma=refresh)


@pytest.mark.parametrize("nx,ny,box,slices,refresh", [
    (1088, 272, 12, 1, False),   # four blocks, two steps, both polarisations' units unlike
    (272, 1088, 12, 1, False),
    (1104, 296, 12, 1, False),
    (700, 256, 9, 1, False),
    (256, 256, 9, 1, False),     # near grazing
    (800, 264, 9, 2, True),      # three blocks, no step
    (800, 264, 9, 3, True),
    (640, 640, 8, 1, False),     # two blocks
    (312, 312, 6, 1, False),     # N = 169
])
def test_mixed_image_of_wide_boxes(cuda, nx, ny, box, slices, refresh):
    import torch
    from euvlitho_b200.engine import Plan
    cfg = _config(nx, ny, box, slices, refresh)
    masks = torch.from_numpy(np.stack([packed(random_mask(nx, ny, seed=s)) for s in range(8)]))
    img = {}
    for p in ("fp64", "mixed"):
        img[p] = Plan(cfg, device=cuda, precision=p, pols=("X", "Y")).intensity(masks)
    d = (img["mixed"] - img["fp64"]).flatten(2).norm(dim=2) / img["fp64"].flatten(2).norm(dim=2)
    assert float(d.max()) < 5e-6, d


@pytest.mark.parametrize("pol", ["X", "Y"])
@pytest.mark.parametrize("nx,ny,box", [(560, 256, 7), (256, 256, 8)])
def test_fp64_amplitudes_of_wide_boxes(cuda, pol, nx, ny, box):
    import torch
    from euvlitho_b200.engine import Plan
    cfg = _config(nx, ny, box, 1)
    plan = Plan(cfg, device=cuda, pols=(pol,))
    m = random_mask(nx, ny, seed=3)
    ax, srcs = plan.amp(torch.from_numpy(packed(m)[None]), polar=pol)
    ax = ax.cpu().numpy()
    oc = to_oracle(cfg)
    L, M = cfg.order_limits()
    ref = O.amp_s(pol, flat_bits(m), oc, plan.orders.lidx, plan.orders.midx, L, M, oc.kx0, oc.ky0)
    seen = [rel_err(ax[0, s], ref[k]) for s, k in enumerate(srcs) if plan.pos.get(k) is not None]
    assert seen and max(seen) < 1e-11, max(seen)


def test_wide_and_narrow_units_in_one_launch(cuda):
    """Units of 256 nm (wide: steps, diagonals apart) and 720 nm (neither) with one order
    set: each as it is alone."""
    import torch
    from euvlitho_b200 import _lib as L
    from euvlitho_b200.engine import Plan
    plans, spectra = [], []
    for i, p in enumerate((256, 720)):
        plan = Plan(_config(p, p, 8, 1), device=cuda, precision="mixed")
        m = plan.as_mask_tensor(torch.from_numpy(packed(random_mask(p, p, seed=i))[None]))
        spectra.append(plan.spectra(m, 2 * plan.orders.lmax, 2 * plan.orders.mmax)[0])
        plans.append(plan)
    spec = torch.stack(spectra).contiguous()
    plan = plans[0]
    centre = plan.pos[(0, 0)]

    def run(units):
        n = len(units)
        keep = []
        dx = plan._f64([float(plans[u].cfg.dx) for u in units])
        d = plan.amp_desc(plan.orders, plan._t_l, plan._t_m, plan._f64([plan.cfg.kx0] * n),
                          plan._f64([plan.cfg.ky0] * n), plan._i32([u % 2 for u in units]),
                          plan._i32(units), plan._i32(np.full((n, 1), centre)),
                          plan._f64(np.full((n, 1), 1.0)), keep)
        d.dx = d.dy = min(plans[u].cfg.dx for u in units)
        d.d_dx = d.d_dy = dx.data_ptr()
        ax = torch.empty((n, 1, plan.orders.n), dtype=torch.complex128, device=cuda)
        plan.run_amp(d, spec, ax)
        plan.check()
        return ax

    both = run([0, 1])
    for u in (0, 1):
        one = run([u])[0]
        assert float((both[u] - one).abs().max() / one.abs().max()) < 1e-13, u
