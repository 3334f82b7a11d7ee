"""ampS for spectra that belong to no pattern with values in [0, 1] (scaled, sign-flipped,
offset, complex or skew): the slab polynomials' ellipse is not theirs, and the operator takes
the spectrum's own bound and more double-angle steps.  Against the slab equations with the
block exponential of scipy, which asks for no eigenvectors.

Tolerance, of the largest amplitude: FP64 1e-9 (up to 12 steps, each doubling an error of
1e-15 a few times, and a condition number below 100); mixed 2e-3 (the same from 1e-7)."""
import numpy as np
import pytest

from euvlitho_b200.config import preset
from oracle import euv_oracle as O
from tests.helpers import packed, random_mask, rel_err, to_oracle

pytestmark = pytest.mark.gpu

TA = complex(0.95, 0.031) ** 2


def _reference(cfg, plan, pol, F, L, M):
    """Reflected amplitudes of a unit wave in order (0, 0), F[slice] the absorber's spectra:
    X1 = c Z - i s Y2, Y1 = -i D s Z + c Y2, Z = G1^-1 G2 X2, from the cap to the top."""
    from scipy.linalg import expm
    l, m = np.asarray(plan.orders.lidx), np.asarray(plan.orders.midx)
    k, n = cfg.k, l.size
    kx, ky = cfg.kx0 + 2 * np.pi / cfg.dx * l, cfg.ky0 + 2 * np.pi / cfg.dy * m
    kp = kx if pol == "X" else ky
    kxy2 = kx ** 2 + ky ** 2
    st = to_oracle(cfg).stack
    u, v = O.multilayer_s(pol, k, kx, ky, kxy2, st)
    eru = st.n_ru ** 2
    dl, dm = l[:, None] - l[None, :], m[:, None] - m[None, :]
    eye = np.eye(n)
    X = Y = Gup = None
    for i in range(cfg.nabs - 1, -1, -1):
        e, d = complex(cfg.eabs[i]), cfg.dabs[i]
        f = F[i][dl + 2 * L, dm + 2 * M]
        one = (dl == 0) & (dm == 0)
        grad = 2 * np.pi / cfg.dx * dl * kx[None, :] if pol == "X" else 2 * np.pi / cfg.dy * dm * ky[None, :]
        D = k * k * ((e - 1) * f + one) + grad * np.log(e) * f - np.diag(kxy2)
        G = 1j * (k * eye - kp[:, None] / k * ((1 / e - 1) * f + one) * kp[None, :])
        if X is None:
            Z = np.linalg.solve(G, np.diag((1j * k - 1j / k / eru * kp ** 2) * (u + v)))
            Y = np.diag(np.sqrt(k * k * eru - kxy2 + 0j) * (u - v))
        else:
            Z = np.linalg.solve(G, Gup @ X) if cfg.refresh_sigma else X
        full = expm(d * np.block([[0 * eye, eye], [-D, 0 * eye]]))
        c, s = full[:n, :n], full[:n, n:]
        X, Y, Gup = c @ Z - 1j * s @ Y, c @ Y - 1j * D @ (s @ Z), G
    klm = np.sqrt(k * k - kxy2)
    o = plan.pos[(0, 0)]
    rhs = 2 * klm * (np.arange(n) == o)
    a = -(Y @ np.linalg.solve(klm[:, None] * X + Y, rhs)) / klm
    a[o] += 1.0
    return a


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 2e-3)])
@pytest.mark.parametrize("period,box,slices,pol,change", [
    (256, 5, 1, "X", lambda F, z: 3.0 * F),
    (256, 5, 1, "Y", lambda F, z: -F),
    (256, 5, 1, "X", lambda F, z: 8.0 * F),
    (320, 6, 1, "X", lambda F, z: (1.5 - 2.0j) * F),
    (256, 5, 2, "X", lambda F, z: 4.0 * F - 1.0 * z),
    (320, 6, 2, "Y", lambda F, z: np.triu(F) * 2.0),
    (256, 5, 2, "Y", lambda F, z: F),                 # a pattern's, as ever
])
def test_amp_takes_any_spectrum(cuda, precision, tol, period, box, slices, pol, change):
    import torch
    from euvlitho_b200.engine import Plan
    cfg = preset("small").with_(ndivx=period, ndivy=period, lbox=box, mbox=box, eabs=(TA,) * slices,
                                dabs=(60.0 / slices,) * slices, refresh_sigma=slices > 1)
    plan = Plan(cfg, device=cuda, precision=precision, pols=(pol,))
    m = random_mask(period, period, seed=7)
    L, M = cfg.order_limits()
    tm = plan.as_mask_tensor(torch.from_numpy(packed(m)[None]))
    spec = plan.spectra(tm, 2 * L, 2 * M)
    F0 = spec.cpu().numpy().reshape(slices, 4 * M + 1, 4 * L + 1).transpose(0, 2, 1)
    zero = np.zeros_like(F0[0])
    zero[2 * L, 2 * M] = 1.0
    # the last slice is changed, the others are the mask's
    F = F0.copy()
    F[-1] = change(F0[-1], zero)
    spec = torch.from_numpy(np.ascontiguousarray(F.transpose(0, 2, 1)).reshape(1, slices, -1)).cuda()
    centre = plan.pos[(0, 0)]
    keep = []
    d = plan.amp_desc(plan.orders, plan._t_l, plan._t_m, plan._f64([cfg.kx0]), plan._f64([cfg.ky0]),
                      plan._i32([0 if pol == "X" else 1]), plan._i32([0]), plan._i32([[centre]]),
                      plan._f64([[2 * np.sqrt(cfg.k ** 2 - cfg.kx0 ** 2 - cfg.ky0 ** 2)]]), keep)
    ax = torch.empty((1, 1, plan.orders.n), dtype=torch.complex128, device=cuda)
    plan.run_amp(d, spec.contiguous(), ax)
    plan.check()  # no status bit: the steps were there
    ref = _reference(cfg, plan, pol, F, L, M)
    assert rel_err(ax[0, 0].cpu().numpy(), ref) < tol


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e9])
def test_amp_flags_spectra_without_bound(cuda, value):
    import torch
    from euvlitho_b200 import _lib
    from euvlitho_b200.engine import Plan
    plan = Plan(preset("small"), device=cuda)
    m = plan.as_mask_tensor(torch.from_numpy(packed(random_mask(256, 256, seed=7))[None]))
    spec = plan.spectra(m, 2 * plan.orders.lmax, 2 * plan.orders.mmax)
    spec[0, 0, 3] = value
    centre = plan.pos[(0, 0)]
    keep = []
    cfg = plan.cfg
    d = plan.amp_desc(plan.orders, plan._t_l, plan._t_m, plan._f64([cfg.kx0]), plan._f64([cfg.ky0]),
                      plan._i32([0]), plan._i32([0]), plan._i32([[centre]]), plan._f64([[0.9]]), keep)
    ax = torch.empty((1, 1, plan.orders.n), dtype=torch.complex128, device=cuda)
    plan.run_amp(d, spec, ax)
    with pytest.raises(_lib.EuvError):
        plan.check()
