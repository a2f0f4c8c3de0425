"""Front end, every kernel size: the filter within the rounding bound of an FP32 sum of the
kernel's terms, and a large kernel on a small movie in the time of its multiply-adds."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", range(1, 32))
def test_filter_of_every_size(bsfit_mod, k):
    import torch
    from oracle import frontend as FE
    rng = np.random.default_rng(k)
    fr = rng.poisson(20, (2, 45, 77)).astype(np.float32) * 2 + 100
    h = rng.uniform(-0.2, 1, (k, k)).astype(np.float32)
    rois, coords, filt = bsfit_mod.find_rois_torch(torch.from_numpy(fr).cuda(), 100.0, 0.5, h, True, 0.0, 5,
                                                   filtered=True)
    filt = filt.cpu().numpy()
    ph = FE.imphot(fr, 100.0, 0.5)
    for f in range(2):
        x = ph[f] - ph[f][0].min()
        size = FE.filter2_same(np.abs(h).astype(np.float64), np.abs(x))
        # k^2 FMAs and the pixel's own rounding, each at most 2^-24 of the sum of the
        # absolute terms
        assert np.all(np.abs(filt[f] - FE.filter2_same(h.astype(np.float64), x)) <= (k * k + 2) * 2.0 ** -24 * size)
    R, C, _ = FE.find_rois(fr, 100.0, 0.5, None, True, 0.0, 5, impf=filt)
    assert np.array_equal(coords.cpu().numpy(), C.astype(np.float32)) and np.array_equal(rois.cpu().numpy(), R)


def test_large_kernel_on_a_small_movie(bsfit_mod):
    import torch
    d = torch.full((30, 100, 100), 140.0, device="cuda")

    def best(k):
        h = np.full((k, k), 1.0 / k ** 2, np.float32)
        ts = []
        for _ in range(12):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            bsfit_mod.find_rois_torch(d, 100.0, 0.5, h, False, 1e6, 13, capacity=100)
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return min(ts)

    # most of the call is the same at any size; a loop over the terms made it 2.7 times as long
    assert best(31) <= 2.0 * best(13)
