"""The double-precision fit's variances and log-likelihoods at ROI sizes around the 128
pixels that a block evaluates at once: where the parameters are the FP64 oracle's, the
variances are its bits, and the log-likelihoods agree to the rounding of log()."""
import os

import numpy as np
import pytest

from test_fit64_blocks_gpu import _workload
from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fittype,s,n,its", [(6, 11, 40, 20), (6, 12, 40, 20), (6, 23, 20, 20), (7, 11, 20, 15),
                                             (7, 17, 12, 15), (8, 11, 10, 6), (8, 12, 10, 6), (8, 17, 6, 6)])
def test_variances_and_log_likelihoods(bsfit_mod, oracle, fittype, s, n, its):
    import torch
    wl = _workload(fittype, s, n)
    m = bsfit_mod.Model(fittype, wl.coeff, coeff3=wl.coeff3, init_p=wl.init_p)
    P, C, L = (x.cpu().numpy().T for x in m.fit_f64_torch(torch.from_numpy(wl.rois).cuda(), its))
    R, RC, RL = oracle.fit(wl.rois, fittype, its, wl.coeff, precision="f64", init_p=wl.init_p,
                           coeff3=wl.coeff3, threads=os.cpu_count() or 1)
    same = np.all((P == R) | (np.isnan(P) & np.isnan(R)), axis=1)
    assert (~same).sum() <= 1, np.where(~same)[0]  # one ROI of slack for a log() rounding flip
    assert np.array_equal(C[same], RC[same], equal_nan=True)
    # A pixel's term is d log(m) - m - d log(d) + d, of at most 4 top (1 + log(top)) with
    # d, m <= top; every log and every one of the s^2 + 8 operations behind it may round
    # by one unit of that.
    top = 2.0 * float(wl.rois.max()) + float(np.nanmax(np.abs(R[same][:, 2:4]), initial=1.0))
    tol = np.finfo(float).eps * (s * s + 8) * s * s * 4.0 * top * (1.0 + np.log(top))
    a, b = np.ravel(L)[same], np.ravel(RL)[same]
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.nanmax(np.abs(a - b), initial=0.0) <= tol
    m.close()
