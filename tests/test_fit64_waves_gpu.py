"""The double-precision fit's blocks of four, two and one warp: calls of few iterations take
the widest that holds them in one wave, calls of many iterations always four, and all give
the same bits."""
import numpy as np
import pytest

from kernel_names import captured
from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


def _calls(b, fittype):
    """fit(n, iterations) over ROIs that repeat after `base` of them."""
    import torch
    from bsfit import workloads as W
    base, most = 90, 152 * 14
    idx = torch.arange(most, device="cuda") % base
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    if fittype == 9:
        w = W.workload_4pi(base, s=9, stream=951)
        rois = w.rois.copy()
        rois[:, 1] = 0.0
        rois[:, 2, 0, 0] = np.nan
        m = b.Model4Pi(w.coeff, w.extra["phase_shift"])
        r, z, p, d = cu(rois)[:, idx].contiguous(), cu(w.extra["init_z"])[idx], cu(w.extra["init_phi"])[idx], \
            cu(w.extra["dT"])[idx]
        return base, m, lambda n, its: m.fit_f64_torch(r[:, :n].contiguous(), its, z[:n].contiguous(),
                                                       p[:n].contiguous(), d[:n].contiguous())
    w = (W.workload_3d(base, s=12, stream=952) if fittype == 6 else
         W.workload_4d(base, sizes=(9,), stream=953)[0] if fittype == 7 else W.workload_5d(base, s=9, stream=954))
    rois = w.rois.copy()
    rois[1] = 0.0
    rois[2, 0, 0] = np.nan
    rois[3] = 7.0
    m = b.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    r = cu(rois)[idx]
    return base, m, lambda n, its: m.fit_f64_torch(r[:n].contiguous(), its)


@pytest.mark.parametrize("fittype,warps", [(6, (4, 4, 2, 2, 4)), (7, (4, 4, 2, 1, 4)), (8, (4, 2, 4, 4, 4)),
                                           (9, (4, 2, 2, 1, 4))])
def test_blocks_by_count(bsfit_mod, fittype, warps):
    base, m, fit = _calls(bsfit_mod, fittype)
    ref = [x.cpu().numpy() for x in fit(base, 3)]
    for per_sm, w in zip((2, 3.5, 5, 8, 13) if fittype == 6 else (2, 3.5, 5, 9, 13) if fittype == 7 else
                         (2, 2.6, 6, 8, 9) if fittype == 8 else (3, 3.5, 8, 10, 13), warps):
        n = int(152 * per_sm)
        out = [x.cpu().numpy() for x in fit(n, 3)]
        for a, b in zip(out, ref):
            assert np.array_equal(a, np.take(b, np.arange(n) % base, axis=-1), equal_nan=True), per_sm
        name = captured(lambda: fit(n, 3))[1][-1]
        assert f"fit64_kernelILi{fittype}ELi{w}E" in name, (per_sm, name)
        name = captured(lambda: fit(n, 100))[1][-1]
        assert f"fit64_kernelILi{fittype}ELi4E" in name, (per_sm, name)
    m.close()
