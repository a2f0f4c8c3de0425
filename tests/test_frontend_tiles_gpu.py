"""Front end at the edges of its tiles (62 rows x 30 columns of a frame) and over
kernel sizes, looped and unrolled: the filter within the rounding bound of an
FP32 sum of the kernel's terms, and maxima, order, coordinates and ROIs equal to
the restatement's on the GPU's own filtered frames, with and without the
filtered output."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,H,W,k,s,mirror,dog", [
    (1, 3, 3, 3, 1, False, False), (2, 62, 30, 4, 7, False, False), (2, 63, 31, 5, 7, True, True),
    (3, 61, 29, 6, 9, False, True), (2, 64, 32, 7, 51, False, False), (2, 125, 91, 8, 13, True, True),
    (1, 200, 333, 13, 15, False, False), (2, 65, 200, 14, 11, False, True), (1, 130, 64, 31, 21, True, False),
    (5, 40, 37, 1, 5, False, False), (2, 128, 62, 2, 5, False, True), (2, 96, 61, 11, 3, False, False)])
def test_tiles_match_restatement(bsfit_mod, F, H, W, k, s, mirror, dog):
    import torch
    from oracle import frontend as FE
    rng = np.random.default_rng(H * W + k)
    fr = rng.poisson(20, (F, W, H)).astype(np.float32) * 2 + 100
    fr[:, ::7, ::5] += rng.uniform(0, 400, fr[:, ::7, ::5].shape).astype(np.float32)
    h = rng.uniform(-0.2, 1, (k, k)).astype(np.float32)
    ph = FE.imphot(fr, 100.0, 0.5)
    d = torch.from_numpy(fr).cuda()
    for cut in (-1e39, 25.3):
        rois, coords, filt = bsfit_mod.find_rois_torch(d, 100.0, 0.5, h, dog, cut, s, mirror=mirror,
                                                       filtered=True)
        filt = filt.cpu().numpy()
        for f in range(F):
            x = ph[f] - (ph[f][0].min() if dog else 0.0)
            ref = FE.filter2_same(h.astype(np.float64), x)
            size = FE.filter2_same(np.abs(h).astype(np.float64), np.abs(x))
            # k^2 FMAs and the pixel's own rounding, each at most 2^-24 of the sum
            # of the absolute terms
            assert np.all(np.abs(filt[f] - ref) <= (k * k + 2) * 2.0 ** -24 * size + 1e-30)
        R, C, _ = FE.find_rois(fr, 100.0, 0.5, None, dog, cut, s, mirror=mirror, impf=filt)
        assert np.array_equal(coords.cpu().numpy(), C.astype(np.float32))
        assert np.array_equal(rois.cpu().numpy(), R)
        r2, c2 = bsfit_mod.find_rois_torch(d, 100.0, 0.5, h, dog, cut, s, mirror=mirror)
        assert torch.equal(r2, rois) and torch.equal(c2, coords)
