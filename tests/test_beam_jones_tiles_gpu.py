"""Jones tables from beam images at the edges of the kernel's tiles: one
component and one more than a CTA holds, one plane and the most, the narrowest
and widest interpolation, blanked and off-grid positions, against the FP64
oracle within the bound of the other beam-image tests (2e-5 absolute)."""
import numpy as np
import pytest

import oracle
from obit_b200.beam import BeamImages, jones_from_images

pytestmark = pytest.mark.gpu
FBLANK = -3.0e38


@pytest.mark.parametrize("ncomp, ntype, nplane, hwidth", [(1, 1, 1, 1), (33, 2, 1, 4), (9, 1, 8, 2), (65, 3, 3, 3),
                                                          (5, 1, 64, 2), (130, 2, 17, 4)])
def test_jones_tiles(ncomp, ntype, nplane, hwidth):
    torch = pytest.importorskip("torch")
    r = np.random.default_rng(ncomp + nplane)
    n = 41
    y, x = (np.mgrid[0:n, 0:n] - n // 2) / (n // 2)
    px = 0.05 + 0.02 * r.uniform(-1, 1, (ntype, 8, nplane, 1, 1)) * (x + y)
    px[:, [0, 2]] += 0.9 * np.exp(-0.3 * (x * x + y * y))
    px = px.astype(np.float32)
    px[:, :, :, 5:9, 30:33] = FBLANK
    im = BeamImages(px, np.linspace(1.2e9, 1.6e9, nplane), crpix=(n // 2 + 1, n // 2 + 1), cdelt=(0.05, 0.05),
                    hwidth=hwidth, fblank=FBLANK, refSizeFact=3.0e-10)
    pos = r.uniform(-1.2, 1.2, (ncomp, 2)).astype(np.float32)
    d_px, d_pos = torch.from_numpy(px).cuda(), torch.from_numpy(pos).cuda()
    d_j = torch.zeros((ntype, ncomp, nplane, 8), dtype=torch.float32, device="cuda")
    jones_from_images(im, d_px.data_ptr(), d_pos.data_ptr(), ncomp, 0.37, d_j.data_ptr())
    want = oracle.beam_jones_fp64(im, pos, 0.37)
    assert np.abs(d_j.cpu().numpy() - want).max() < 2e-5
