"""The mask spectrum from the packed bits on the FP64 tensor path: rows that start inside
a byte, sizes that are no multiples of the tiles (128 rows, 32 pixels, 8 clusters'
shares, 8 columns), refined grids, the y offset, one frequency and more column tiles
than one, groups of masks that do not fit the workspace at once.

Tolerance 1e-14 of the largest value, as the other spectrum test (sums of at most
10^6 terms of size 1 / (fx fy), accumulated in blocks)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vacuum", [0, 1])
@pytest.mark.parametrize("nx,ny,mesh,lh,mh,yoff,masks", [
    (64, 64, 1, 5, 3, 0, 1),
    (250, 252, 1, 20, 31, 1, 3),     # rows start inside bytes
    (36, 2, 1, 0, 0, 0, 2),          # one frequency, two rows
    (72, 130, 2, 40, 9, 0, 2),       # refined grid, 82 columns in two tiles
    (520, 136, 1, 75, 30, 0, 2),     # three column tiles, a ragged last row block
    (8, 400, 3, 11, 70, 1, 5),       # fewer pixels than the clusters' shares
])
def test_spectrum_matches_fft(cuda, vacuum, nx, ny, mesh, lh, mh, yoff, masks):
    import torch
    from euvlitho_b200 import _lib as L
    rng = np.random.default_rng(nx * ny + lh)
    m = (rng.random((masks, ny, nx)) < 0.6).astype(np.uint8)
    bits = np.stack([np.packbits(x.reshape(-1), bitorder="big") for x in m])
    fx, fy = mesh * nx, mesh * ny
    d = torch.from_numpy(bits).cuda()
    out = torch.empty((masks, (2 * mh + 1), (2 * lh + 1)), dtype=torch.complex128, device="cuda")
    one = L.lib().euv_mask_spectrum_workspace_bytes(1, nx, ny, fx, fy, lh, mh)
    full = L.lib().euv_mask_spectrum_workspace_bytes(masks, nx, ny, fx, fy, lh, mh)
    jj = ny - 1 - np.arange(fy) // mesh + yoff
    inside = (jj >= 0) & (jj < ny)
    pat = np.where(inside[:, None], m[:, np.clip(jj, 0, ny - 1)][:, :, np.arange(fx) // mesh], 0)
    pat = pat if vacuum else 1 - pat                               # [mask][y][x]
    F = np.fft.fft2(pat.astype(float)) / (fx * fy)
    ref = F[:, np.arange(-mh, mh + 1) % fy][:, :, np.arange(-lh, lh + 1) % fx]
    for nbytes in (full, one):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        out.zero_()
        L.call("euv_mask_spectrum", d.data_ptr(), masks, nx, ny, fx, fy, lh, mh, vacuum, yoff,
               out.data_ptr(), ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)
        assert np.max(np.abs(out.cpu().numpy() - ref)) < 1e-14 * np.max(np.abs(ref))


@pytest.mark.parametrize("vacuum", [0, 1])
@pytest.mark.parametrize("nx,ny,mesh", [(672, 280, 1), (584, 424, 1), (250, 252, 2), (8, 400, 3)])
def test_mean_is_exact(cuda, vacuum, nx, ny, mesh):
    """F(0, 0) is a whole number of cells over all of them, rounded once (twice for the
    absorber's 1 - F); an all-vacuum mask has exactly 1 and 0."""
    import torch
    from euvlitho_b200 import _lib as L
    rng = np.random.default_rng(nx)
    m = np.stack([np.ones((ny, nx), np.uint8), (rng.random((ny, nx)) < 0.6).astype(np.uint8)])
    d = torch.from_numpy(np.stack([np.packbits(x.reshape(-1)) for x in m])).cuda()
    fx, fy, lh, mh = mesh * nx, mesh * ny, 3, 2
    out = torch.empty((2, 2 * mh + 1, 2 * lh + 1), dtype=torch.complex128, device="cuda")
    n = L.lib().euv_mask_spectrum_workspace_bytes(2, nx, ny, fx, fy, lh, mh)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    L.call("euv_mask_spectrum", d.data_ptr(), 2, nx, ny, fx, fy, lh, mh, vacuum, 0, out.data_ptr(),
           ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    got = out[:, mh, lh].cpu().numpy()
    f = np.array([float(x.sum()) * mesh * mesh / (fx * fy) for x in m])
    np.testing.assert_array_equal(got.real, f if vacuum else 1.0 - f)
