"""Which double-float calls are fitted on their own and which in step, and that a call that
the in-step warps hold takes one wave; the bits of both are those of one large call."""
import numpy as np
import pytest

from kernel_names import launches
from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu

SM = 152


# (fit type, size, ROIs, in step, warps per block in step)
@pytest.mark.parametrize("fittype,s,n,step,warps", [
    (6, 7, 8 * SM, False, 0), (6, 7, 8 * SM + 1, False, 0), (6, 9, 9 * SM + SM // 2 + 1, True, 10),
    (6, 13, 8 * SM, False, 0), (6, 13, 8 * SM + 1, True, 9), (6, 19, 10 * SM, True, 10), (6, 19, 30 * SM, True, 8),
    (6, 23, 20 * SM, False, 0), (7, 9, 4 * SM, False, 0), (7, 9, 4 * SM + 1, True, 5), (7, 13, 40 * SM, True, 12),
    (8, 13, 2 * SM, True, 2),
    (8, 17, SM, True, 1), (8, 17, SM + 1, False, 0), (8, 17, 3 * SM, False, 0), (8, 17, 3 * SM + 1, True, 4)])
def test_place(bsfit_mod, fittype, s, n, step, warps):
    import torch
    from bsfit import workloads as W
    few = 40
    w = (W.workload_3d(few, s=s, stream=760 + s) if fittype == 6 else
         W.workload_4d(few, sizes=(s,), stream=770 + s)[0] if fittype == 7 else W.workload_5d(few, s=s, stream=780 + s))
    rois = w.rois.copy()
    rois[1] = 0.0
    rois[2, 0, 0] = np.nan
    rois[3] *= -1.0
    m = bsfit_mod.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    r = torch.from_numpy(rois[np.resize(np.arange(few), max(n, 45 * SM))]).cuda()
    fit = lambda k: m.fit_torch(r[:k], 3, precision="parity", exact_steps=0)  # noqa: E731
    ref = [x.cpu().numpy() for x in fit(len(r))]
    for a, b in zip(fit(n), ref):
        assert np.array_equal(a.cpu().numpy(), b[..., :n], equal_nan=True)
    for b in ref:
        assert np.array_equal(b[..., few:2 * few], b[..., :few], equal_nan=True)
    got = [x for x in launches(lambda: fit(n)) if x[1] and "fitdd_kernel" in x[1]]
    assert len(got) == 1 and f"fitdd_kernelILi{fittype}ELb{int(step)}E" in got[0][1], got
    if step:
        assert got[0][3] == 32 * warps, got
    m.close()
