"""One-ROI-per-block fits of large ROIs, whose shared memory leaves an SM fewer blocks than
the form of that count is compiled for: the sparser form that fits runs (warps, blocks), and
gives the bits of the one-warp form."""
import numpy as np
import pytest

from kernel_names import captured
from test_fit_gpu import bsfit_mod  # noqa: F401
from test_team_gpu import BIG, _call, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fittype,s,n,form", [
    (6, 27, 700, (4, 6)), (6, 33, 700, (8, 2)), (6, 51, 900, (8, 2)), (7, 33, 500, (8, 2)), (7, 41, 700, (8, 2)),
    (8, 21, 690, (4, 4)), (8, 25, 700, (4, 3)), (8, 27, 760, (4, 3)), (8, 33, 700, (8, 2)), (8, 51, 300, None),
    (9, 18, 1200, (8, 2)), (9, 24, 150, (16, 1)), (9, 24, 1000, (16, 1)), (9, 24, 1200, None)])
def test_form_that_fits(bsfit_mod, fittype, s, n, form):
    rois, model, extra = _setup(bsfit_mod, fittype, s)
    axis = 1 if fittype == 9 else 0
    rois = np.moveaxis(rois, axis, 0).copy()
    rois[1] = 0.0
    rois[2, ..., 0, 0] = np.nan
    many = np.resize(np.arange(len(rois)), BIG)

    def call(k):
        idx = many[:k]
        e = tuple(x[idx] for x in extra) if fittype == 9 else extra
        return _call(bsfit_mod, fittype, np.moveaxis(rois[idx], 0, axis), 4, model, e, "plain")

    import torch
    out, ref = [x.cpu().numpy() for x in call(n)], [x.cpu().numpy() for x in call(BIG)]
    for a, b in zip(out, ref):
        assert np.array_equal(a, b[..., :n], equal_nan=True)
    r = torch.from_numpy(np.ascontiguousarray(np.moveaxis(rois[many[:n]], 0, axis))).cuda()
    e = [torch.from_numpy(np.ascontiguousarray(x[many[:n]])).cuda() for x in extra] if fittype == 9 else []
    name = captured(lambda: model.fit_torch(r, 4, *e))[1][-1]
    if form:
        assert f"team_kernelILi{fittype}ELb0ELb0ELi{form[0]}ELi{form[1]}E" in name, name
    else:
        assert "fit_kernel" in name, name
    model.close()
