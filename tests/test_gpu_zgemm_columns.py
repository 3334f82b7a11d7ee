"""FP64 products of more than 65535 column tiles: euv_zgemm itself, and the mask spectra of
many masks, whose second stage has a column per mask and frequency.

Tolerance: 1e-13 of the largest value for two products of 3 terms; the spectra equal those of
smaller calls (a column's operations do not depend on the others)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(3, 65535 * 32), (3, 65535 * 32 + 1), (70, 2500003)])
def test_zgemm_of_many_columns(cuda, m, n):
    import torch
    from euvlitho_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(n)
    # column-major operands: the tensors hold the transposes
    A = torch.randn(3, m, dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn(n, 3, dtype=torch.complex128, device="cuda", generator=g)
    C = torch.empty(n, m, dtype=torch.complex128, device="cuda")
    L.call("euv_zgemm", m, n, 3, L.c64(1, 0), None, A.data_ptr(), m, 0, B.data_ptr(), 3, 0,
           L.c64(0, 0), C.data_ptr(), m, 0, L.c64(0, 0), 1, None, 0,
           torch.cuda.current_stream().cuda_stream)
    ref = (B[:, :, None] * A[None]).sum(1)
    assert float((C - ref).abs().max() / ref.abs().max()) < 1e-13


def test_spectra_of_many_masks(cuda):
    import torch
    from euvlitho_b200 import _lib as L
    n, nx, ny, lh, mh = 21000, 256, 8, 100, 1  # 21000 x 101 columns
    rng = np.random.default_rng(1)
    masks = torch.from_numpy(rng.integers(0, 256, (n, nx * ny // 8)).astype(np.uint8)).cuda()

    def spectra(part):
        k = part.shape[0]
        out = torch.empty((k, (2 * lh + 1) * (2 * mh + 1)), dtype=torch.complex128, device="cuda")
        wb = L.lib().euv_mask_spectrum_workspace_bytes(k, nx, ny, nx, ny, lh, mh)
        ws = torch.empty(wb, dtype=torch.uint8, device="cuda")
        L.call("euv_mask_spectrum", part.data_ptr(), k, nx, ny, nx, ny, lh, mh, 0, 0,
               out.data_ptr(), ws.data_ptr(), wb, torch.cuda.current_stream().cuda_stream)
        return out

    whole = spectra(masks)
    parts = torch.cat([spectra(masks[i:i + 7000]) for i in range(0, n, 7000)])
    assert torch.equal(whole, parts)
