"""euv_abbe with source slots beyond a unit's sources (padded tables): the band-limited form
gives the image of the exact tables, and a unit without a source leaves its image alone.
Tolerance 1e-13 of the largest value: the order of the FP64 sums over sources."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sources", [1, 8, 9, 12, 50, 199])
def test_padded_slots(cuda, precision, sources):
    import torch
    from euvlitho_b200 import _lib as L
    lpx, lpy, xdiv, ydiv, padded = 12, 6, 576, 1536, 200
    assert xdiv * ydiv * (2 * lpx + 1) >= 2e7  # the band form's side of the rule, one source
    rng = np.random.default_rng(sources)
    px, py = [a.ravel().astype(np.int32) for a in np.meshgrid(
        np.arange(-lpx, lpx + 1), np.arange(-lpy, lpy + 1), indexing="ij")]
    ncut, n_order = px.size, 30
    nidx = np.full((padded, ncut), -1, np.int32)
    for s in range(sources):
        w = rng.integers(1, 2 * lpx + 1)
        ok = (px <= -lpx + w) & (np.abs(py) <= rng.integers(1, lpy + 1))
        nidx[s, ok] = rng.integers(0, n_order, ok.sum())
    cplx = lambda *sh: rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    coef, ax = cplx(padded, ncut, 3), cplx(3, padded, n_order)
    t = {k: dev(v) for k, v in dict(px=px, py=py, w=np.ones(3), tab=np.zeros(3, np.int32),
                                    rs=np.searchsorted(px, np.arange(-lpx, lpx + 2)).astype(np.int32),
                                    img=np.arange(3, dtype=np.int32),
                                    nsrc=np.array([sources, 0, sources], np.int32)).items()}

    def run(slots):
        c, n, a = dev(coef[:slots]), dev(nidx[:slots]), dev(ax[:, :slots])
        d = L.AbbeDesc()
        d.xdiv, d.ydiv, d.lpx, d.lpy = xdiv, ydiv, lpx, lpy
        d.ncut, d.n_units, d.n_src, d.n_order, d.n_images = ncut, 3, slots, n_order, 3
        d.d_coef, d.d_nidx = c.data_ptr(), n.data_ptr()
        d.d_px, d.d_py, d.d_row_start = t["px"].data_ptr(), t["py"].data_ptr(), t["rs"].data_ptr()
        d.d_tab_of_unit, d.d_img_of_unit = t["tab"].data_ptr(), t["img"].data_ptr()
        d.d_nsrc_of_unit, d.d_inv_weight = t["nsrc"].data_ptr(), t["w"].data_ptr()
        d.precision = precision
        image = torch.full((3, xdiv, ydiv), -0.0, dtype=torch.float64, device="cuda")
        L.call("euv_abbe", C.byref(d), a.data_ptr(), image.data_ptr(),
               torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return image

    exact, wide = run(sources), run(padded)
    for u in (0, 2):
        assert float((exact[u] - wide[u]).abs().max() / exact[u].abs().max()) < 1e-13
    for image in (exact, wide):  # not even the sign of a zero
        assert bool((image[1] == 0).all()) and bool(torch.signbit(image[1]).all())
