"""Fused multi-start 4Pi calls with one warp per ROI: the kept results are those of a loop over
single-start calls, NaN and flat ROIs among them, and two starts take the time of two
single-start calls."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401
from test_multistart_gpu import _np, compose

pytestmark = pytest.mark.gpu


def _call(b, s, n):
    import torch
    from bsfit import workloads as W
    w = W.workload_4pi(500, s=s, stream=910 + s)
    rois = w.rois.copy()
    rois[:, 1] = 0.0
    rois[:, 2, 0, 0] = np.nan
    rois[:, 3] = 7.0
    idx = torch.arange(n, device="cuda") % 500
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()[idx].contiguous()  # noqa: E731
    r = torch.from_numpy(rois).cuda()[:, idx].contiguous()
    return b.Model4Pi(w.coeff, w.extra["phase_shift"]), r, cu(w.extra["init_z"]), cu(w.extra["init_phi"]), \
        cu(w.extra["dT"])


@pytest.mark.parametrize("s,n,strict", [(4, 1500, False), (11, 1500, True), (16, 3000, False), (24, 1400, True)])
def test_starts_match_loop(bsfit_mod, s, n, strict):
    import torch
    m, r, z, phi, dT = _call(bsfit_mod, s, n)
    zs = torch.stack([z, z + 3, z])
    phis = torch.stack([phi, phi + 5, phi + 9])
    fused = _np(m.fit_multistart_torch(r, 40, zs, phis, dT=dT, strict=strict))
    singles = [_np(m.fit_torch(r, 40, zs[k].contiguous(), phis[k].contiguous(), dT=dT)) for k in range(3)]
    for a, b in zip(fused, compose(singles, strict)):
        assert np.array_equal(a, b, equal_nan=True)
    m.close()


def test_two_starts_in_twice_the_time(bsfit_mod):
    import torch
    m, r, z, phi, dT = _call(bsfit_mod, 12, 1500)
    zs, phis = torch.stack([z, z]), torch.stack([phi, phi])

    def best(call):
        ts = []
        for _ in range(8):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return min(ts)

    one = best(lambda: m.fit_torch(r, 100, z, phi, dT=dT))
    two = best(lambda: m.fit_multistart_torch(r, 100, zs, phis, dT=dT))
    # the kernel of several starts spilled registers in the evaluation: 2.3 times
    assert two <= 2.15 * one
    m.close()
