"""The band-limited form of euv_abbe (samples of each source's |E|^2 on the coarse grid
its support needs, interpolated once) against the sum written out in torch FP64:
ragged image sizes, supports as narrow as one order and as wide as the pupil box
(several passes over rows), sources without a point, empty source slots, images that
already hold something, several units per image.

Tolerance, of the largest value: FP64 1e-13 (sums of at most 10^4 terms of rounding
2^-53, carried through two interpolations of norm below 10); FP32 fields 2e-5 (sums of
up to 2 x 41 x 41 terms of rounding 2^-24)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(0, 1e-13), (1, 2e-5)])
@pytest.mark.parametrize("lpx,lpy,xdiv,ydiv,units,n_src,width", [
    (4, 4, 130, 90, 6, 200, 4),      # image sizes that are no multiples of four or eight
    (4, 2, 256, 61, 5, 150, 8),      # supports as wide as the box
    (20, 10, 255, 128, 4, 15, 20),   # fewer sources than two per CTA
    (20, 20, 96, 96, 3, 60, 40),     # wide supports: several passes over rows
    (3, 1, 512, 256, 8, 24, 0),      # a single order per source
    (41, 20, 128, 64, 2, 30, 41),    # coarse grid finer than the image along x
])
def test_band_form_matches_the_sum(cuda, precision, tol, lpx, lpy, xdiv, ydiv, units, n_src, width):
    import torch
    from euvlitho_b200 import _lib as L
    rng = np.random.default_rng(lpx * 1000 + xdiv + width)
    px, py = [a.ravel() for a in np.meshgrid(np.arange(-lpx, lpx + 1), np.arange(-lpy, lpy + 1),
                                             indexing="ij")]
    keep = rng.random(px.size) < 0.9
    keep[[0, -1]] = True
    px, py = px[keep], py[keep]
    ncut, n_order, n_tab, n_img = px.size, 57, 2, 2
    # supports: boxes of the given width somewhere in the pupil box; one source empty
    nidx = np.full((n_tab, n_src, ncut), -1, np.int32)
    for t in range(n_tab):
        for s in range(n_src):
            wy = min(width, 2 * lpy)
            x0 = rng.integers(-lpx, 2 * lpx - min(width, 2 * lpx) + 1 - lpx)
            y0 = rng.integers(-lpy, 2 * lpy - wy + 1 - lpy)
            ok = (px >= x0) & (px <= x0 + width) & (py >= y0) & (py <= y0 + wy)
            nidx[t, s, ok] = rng.integers(0, n_order, ok.sum())
    nidx[0, n_src // 2] = -1
    cplx = lambda *sh: rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
    coef = cplx(n_tab, n_src, ncut, 3)
    ax = cplx(units, n_src, n_order)
    tab = rng.integers(0, n_tab, units).astype(np.int32)
    img = (np.arange(units) % n_img).astype(np.int32)
    nsrc = rng.integers(0, n_src + 1, units).astype(np.int32)
    nsrc[0] = n_src
    weight = 1.0 / rng.integers(1, 90, n_img)
    start = rng.standard_normal((n_img, xdiv, ydiv))
    assert n_src * xdiv * ydiv * (2 * lpx + 1) >= 2e7  # the band form's side of the rule

    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rs = np.searchsorted(px, np.arange(-lpx, lpx + 2)).astype(np.int32)
    t = {k: dev(v) for k, v in dict(coef=coef, nidx=nidx, px=px.astype(np.int32),
                                    py=py.astype(np.int32), rs=rs, tab=tab, img=img, nsrc=nsrc,
                                    w=weight, ax=ax).items()}
    d = L.AbbeDesc()
    d.xdiv, d.ydiv, d.lpx, d.lpy = xdiv, ydiv, lpx, lpy
    d.ncut, d.n_units, d.n_src, d.n_order, d.n_images = ncut, units, n_src, n_order, n_img
    d.d_coef, d.d_nidx = t["coef"].data_ptr(), t["nidx"].data_ptr()
    d.d_px, d.d_py, d.d_row_start = t["px"].data_ptr(), t["py"].data_ptr(), t["rs"].data_ptr()
    d.d_tab_of_unit, d.d_img_of_unit = t["tab"].data_ptr(), t["img"].data_ptr()
    d.d_nsrc_of_unit, d.d_inv_weight = t["nsrc"].data_ptr(), t["w"].data_ptr()
    d.precision = precision
    image = dev(start)
    L.call("euv_abbe", C.byref(d), t["ax"].data_ptr(), image.data_ptr(),
           torch.cuda.current_stream().cuda_stream)

    wx = torch.exp(2j * np.pi / xdiv * dev(np.outer(np.arange(xdiv), px) % xdiv).to(torch.complex128))
    wy = torch.exp(2j * np.pi / ydiv * dev(np.outer(py, np.arange(ydiv)) % ydiv).to(torch.complex128))
    ref = dev(start).clone()
    for u in range(units):
        for s in range(nsrc[u]):
            n = nidx[tab[u], s]
            ok = np.nonzero(n >= 0)[0]
            if ok.size == 0:
                continue
            e = dev(coef[tab[u], s, ok] * ax[u, s, n[ok]][:, None])
            f = torch.einsum("xi,ic,iy->cxy", wx[:, ok], e, wy[ok])
            ref[img[u]] += float(weight[img[u]]) * (f.real ** 2 + f.imag ** 2).sum(0)
    err = float((image - ref).abs().max() / ref.abs().max())
    assert err < tol, err


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("lpx,lpy,xdiv,ydiv,n_src", [
    (12, 6, 256, 128, 67),    # band-limited in both precisions
    (8, 8, 128, 128, 30),     # FP32: below the rule for one unit, so for twelve too
])
def test_a_unit_alone_and_among_others(cuda, precision, lpx, lpy, xdiv, ydiv, n_src):
    """Supports of many widths: neither the form nor a source's coarse grid may depend
    on how many units share the launch.  1e-13: only the order of the FP64 sums over
    sources does."""
    import torch
    from euvlitho_b200 import _lib as L
    units = 12
    rng = np.random.default_rng(n_src)
    px, py = [a.ravel().astype(np.int32) for a in np.meshgrid(
        np.arange(-lpx, lpx + 1), np.arange(-lpy, lpy + 1), indexing="ij")]
    ncut, n_order = px.size, 40
    nidx = np.full((1, n_src, ncut), -1, np.int32)
    for s in range(n_src):
        w = rng.integers(1, 2 * lpx + 1)
        ok = (px >= -lpx) & (px <= -lpx + w) & (np.abs(py) <= rng.integers(1, lpy + 1))
        nidx[0, s, ok] = rng.integers(0, n_order, ok.sum())
    cplx = lambda *sh: rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    t = {k: dev(v) for k, v in dict(
        coef=cplx(1, n_src, ncut, 3), nidx=nidx, px=px, py=py, ax=cplx(units, n_src, n_order),
        rs=np.searchsorted(px, np.arange(-lpx, lpx + 2)).astype(np.int32),
        tab=np.zeros(units, np.int32), img=np.arange(units, dtype=np.int32),
        nsrc=np.full(units, n_src, np.int32), w=np.ones(units)).items()}

    def run(first, count):
        d = L.AbbeDesc()
        d.xdiv, d.ydiv, d.lpx, d.lpy = xdiv, ydiv, lpx, lpy
        d.ncut, d.n_units, d.n_src, d.n_order, d.n_images = ncut, count, n_src, n_order, count
        d.d_coef, d.d_nidx = t["coef"].data_ptr(), t["nidx"].data_ptr()
        d.d_px, d.d_py, d.d_row_start = t["px"].data_ptr(), t["py"].data_ptr(), t["rs"].data_ptr()
        d.d_tab_of_unit, d.d_img_of_unit = t["tab"].data_ptr(), t["img"].data_ptr()
        d.d_nsrc_of_unit, d.d_inv_weight = t["nsrc"].data_ptr(), t["w"].data_ptr()
        d.precision = precision
        image = torch.zeros(count, xdiv, ydiv, dtype=torch.float64, device="cuda")
        L.call("euv_abbe", C.byref(d), t["ax"][first:].data_ptr(), image.data_ptr(),
               torch.cuda.current_stream().cuda_stream)
        return image

    many = run(0, units)
    for u in (0, 7):
        one = run(u, 1)[0]
        assert float((one - many[u]).abs().max() / one.abs().max()) < 1e-13, u
