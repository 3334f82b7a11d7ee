"""ampS with empty source slots (order -1) anywhere in the table: the filled columns are those
of a table without gaps, the empty ones zero, for the one-launch solve, the blocked one (above
1562 orders) and more slots than stand behind the matrix.  Tolerance 1e-13 of the largest
amplitude: a column's operations do not depend on its neighbours."""
import numpy as np
import pytest

from euvlitho_b200.config import preset
from tests.helpers import packed, random_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("period,box,slots,keep", [
    (256, 5, 40, "head"),
    (256, 5, 40, "every third"),
    (256, 5, 200, "tail"),
    (256, 5, 300, "every third"),   # more than 2 N: solved apart
    (1024, 12, 200, "head"),
    (1024, 12, 130, "every third"),
    (2048, 20, 130, "head"),        # blocked backward pass
    (2048, 20, 70, "tail"),
    (256, 5, 70, "none"),
])
def test_empty_slots(cuda, precision, period, box, slots, keep):
    import torch
    from euvlitho_b200.engine import Plan
    cfg = preset("small").with_(ndivx=period, ndivy=period, lbox=box, mbox=box)
    plan = Plan(cfg, device=cuda, precision=precision)
    m = plan.as_mask_tensor(torch.from_numpy(packed(random_mask(period, period, seed=4))[None]))
    spec = plan.spectra(m, 2 * plan.orders.lmax, 2 * plan.orders.mmax)
    n, units = plan.orders.n, 2
    rng = np.random.default_rng(slots)
    full = rng.integers(0, n, (units, slots)).astype(np.int32)
    on = {"head": np.arange(slots) < 9, "tail": np.arange(slots) >= slots - 5,
          "every third": np.arange(slots) % 3 == 1, "none": np.zeros(slots, bool)}[keep]
    on = np.stack([on, np.roll(on, 1) & on])  # the units differ

    def run(order):
        hold = []
        d = plan.amp_desc(plan.orders, plan._t_l, plan._t_m, plan._f64([cfg.kx0] * units),
                          plan._f64([cfg.ky0] * units), plan._i32([0, 1]), plan._i32([0] * units),
                          plan._i32(order), plan._f64(np.full(order.shape, 0.9)), hold)
        ax = torch.full((units, slots, n), 7.0, dtype=torch.complex128, device=cuda)
        plan.run_amp(d, spec, ax)
        plan.check()
        return ax

    want = run(full)
    got = run(np.where(on, full, -1).astype(np.int32))
    t = torch.from_numpy(on).cuda()
    assert float(got[~t].abs().sum()) == 0.0
    if on.any():
        assert float((got[t] - want[t]).abs().max() / want.abs().max()) < 1e-13
