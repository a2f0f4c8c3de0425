"""The double-float fit's blocks: calls whose ROIs are fitted by blocks of every
width, in step and on their own, bit-identical to one large call whose warps claim
several ROIs each."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fittype,s,its", [(6, 5, 30), (6, 13, 0), (6, 13, 30), (6, 21, 10), (6, 51, 3),
                                           (7, 13, 20), (7, 33, 2), (8, 13, 5), (8, 17, 1)])
def test_blocks_equal_one_large_call(bsfit_mod, fittype, s, its):
    import torch
    from bsfit import workloads as W
    n = 60
    if fittype == 6:
        w = W.workload_3d(n, s=s, stream=700 + s)
    elif fittype == 7:
        w = W.workload_4d(n, sizes=(s,), stream=720 + s)[0]
    else:
        w = W.workload_5d(n, s=s, stream=740 + s)
    rois = np.array(w.rois)
    rois[1] = 0.0
    rois[2, 0, 0] = np.nan
    rois[3] *= -1.0
    rois[4] = 7.0
    model = bsfit_mod.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    big = 5000 if fittype == 6 and s < 51 else 1300
    r = torch.from_numpy(rois[np.resize(np.arange(n), big)]).cuda()
    ref = [x.cpu().numpy() for x in model.fit_torch(r, its, precision="parity")]
    for m in (1, 153, 610, 1064, 1065, 1220, 2433):
        if m < big:
            out = model.fit_torch(r[:m].contiguous(), its, precision="parity")
            for a, b in zip(out, ref):
                assert np.array_equal(a.cpu().numpy(), b[..., :m], equal_nan=True), m
    for k in range(n, big, n):  # each repetition of the same ROIs
        m = min(n, big - k)
        for b in ref:
            assert np.array_equal(b[..., k:k + m], b[..., :m], equal_nan=True), k
    model.close()
