"""Front end, dense maxima: the cut-out of a tile column's ROIs shared among blocks gives the
restatement's list, whole and cut off by the capacity, and a single frame does not take
the time of a movie."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


def _frames(F, H, W):
    return np.random.default_rng(F * H + W).poisson(20, (F, W, H)).astype(np.float32) * 2 + 100


@pytest.mark.parametrize("F,H,W", [(1, 700, 29), (1, 63, 31), (3, 130, 95), (1, 64, 8), (40, 40, 40)])
def test_shares_match_restatement(bsfit_mod, F, H, W):
    import torch
    from oracle import frontend as FE
    fr = _frames(F, H, W)
    h = np.full((3, 3), 1.0 / 9.0, np.float32)
    d = torch.from_numpy(fr).cuda()
    rois, coords, filt = bsfit_mod.find_rois_torch(d, 100.0, 0.5, h, False, 0.0, 5, filtered=True)
    R, C, _ = FE.find_rois(fr, 100.0, 0.5, None, False, 0.0, 5, impf=filt.cpu().numpy())
    assert np.array_equal(coords.cpu().numpy(), C.astype(np.float32)) and np.array_equal(rois.cpu().numpy(), R)
    n = len(C)
    for cap in sorted({1, 7, 8, 9, n // 3, n - 1}):
        if not 0 < cap < n:
            continue
        r, c = bsfit_mod.find_rois_torch(d, 100.0, 0.5, h, False, 0.0, 5, capacity=cap)
        assert torch.equal(r, rois[:cap]) and torch.equal(c, coords[:cap]), cap


def test_one_frame_in_less_time_than_many(bsfit_mod):
    import torch
    h = np.full((7, 7), 1.0 / 49.0, np.float32)
    d = torch.from_numpy(_frames(1, 2048, 1024)).cuda()
    many = d.expand(12, -1, -1).contiguous()

    def best(x):
        ts = []
        for _ in range(8):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            bsfit_mod.find_rois_torch(x, 100.0, 0.5, h, False, 0.0, 13, capacity=x.numel() // 50)
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return min(ts)

    # a tile column's ROIs by one block: the frame's columns all at once, as long as the movie's
    assert best(d) <= 0.5 * best(many)
