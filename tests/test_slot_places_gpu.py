"""Where several ROIs per warp are taken: not where their shared memory costs 4D and 5D
calls resident warps or the L1 of the 5D gathers. Either way the bits are those of one ROI
per warp."""
import numpy as np
import pytest

from kernel_names import captured
from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fittype,s,slots", [
    (6, 13, True), (6, 21, True), (6, 33, True), (7, 13, True), (7, 21, True), (7, 24, False), (7, 27, False),
    (8, 13, True), (8, 14, True), (8, 15, False), (8, 16, False), (8, 17, True), (8, 19, False), (8, 25, False)])
def test_place(bsfit_mod, fittype, s, slots):
    import torch
    from bsfit import workloads as W
    few, many = 40, {6: 152 * 85, 7: 152 * 52, 8: 152 * 38}[fittype]
    w = (W.workload_3d(few, s=s, stream=980 + s) if fittype == 6 else
         W.workload_4d(few, sizes=(s,), stream=980 + s)[0] if fittype == 7 else W.workload_5d(few, s=s, stream=980 + s))
    rois = w.rois.copy()
    rois[1] = 0.0
    rois[2, 0, 0] = np.nan
    m = bsfit_mod.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    idx = np.random.default_rng(s).integers(0, few, many)
    r = torch.from_numpy(rois).cuda()
    lots = r[torch.from_numpy(idx).cuda()].contiguous()
    for a, b in zip(m.fit_torch(lots, 5), m.fit_torch(r, 5)):
        assert np.array_equal(a.cpu().numpy(), np.take(b.cpu().numpy(), idx, axis=-1), equal_nan=True)
    names = captured(lambda: m.fit_torch(lots, 5))[1]
    assert any("slot_kernel" in k for k in names) == slots, names
    m.close()


@pytest.mark.parametrize("fittype,per_sm,segments,slots", [
    (7, 56, 1, True), (7, 80, 2, False), (7, 80, 4, False), (7, 140, 2, True), (8, 42, 1, True), (8, 60, 2, False),
    (8, 110, 3, True), (6, 120, 2, False), (6, 320, 2, True)])
def test_batches_by_segments(bsfit_mod, fittype, per_sm, segments, slots):
    import torch
    from bsfit import workloads as W
    few, n = 30, 152 * per_sm // segments
    w = (W.workload_3d(few, s=13, stream=991) if fittype == 6 else
         W.workload_4d(few, sizes=(13,), stream=992)[0] if fittype == 7 else W.workload_5d(few, s=13, stream=993))
    m = bsfit_mod.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    idx = np.random.default_rng(9).integers(0, few, n)
    r = torch.from_numpy(w.rois).cuda()
    lots = r[torch.from_numpy(idx).cuda()].contiguous()
    b = bsfit_mod.Batch([(m, lots, 4)] * segments)
    ref = m.fit_torch(r, 4)
    for out in b.run():
        for x, y in zip(out, ref):
            assert np.array_equal(x.cpu().numpy(), np.take(y.cpu().numpy(), idx, axis=-1), equal_nan=True)
    names = captured(lambda: b.run())[1]
    assert any("slot_batch_kernel" in k for k in names) == slots, names
    m.close()
