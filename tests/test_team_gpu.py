"""One-ROI-per-block fits (calls of few ROIs): bit-identical to the one-warp form
that larger calls take, at the block sizes' limits, window and ROI remainders,
iteration caps, malformed ROIs, with several starts and with sCMOS variances."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu

BIG = 1600  # more ROIs than any block form takes
SIZES = {6: (5, 7, 11, 13, 16, 21, 33, 51), 7: (5, 9, 13, 16, 33), 8: (5, 13, 17, 33), 9: (5, 12, 16, 25)}


def _call(b, fittype, rois, its, model, extra, kind):
    import torch
    r = torch.from_numpy(np.ascontiguousarray(rois)).cuda()
    if fittype == 9:
        z0, p0, dT = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in extra)
        if kind == "starts":
            return model.fit_multistart_torch(r, its, torch.stack([z0, z0 + 1]), torch.stack([p0, 0.5 * p0]), dT)
        return model.fit_torch(r, its, z0, p0, dT)
    if kind == "starts":
        return model.fit_multistart_torch(r, its, extra)
    if kind == "scmos":
        return model.fit_scmos_torch(r, torch.from_numpy(np.abs(np.sin(1.0 + rois)) + 0.5).cuda(), its)
    return model.fit_torch(r, its)


def _setup(b, fittype, s):
    from bsfit import workloads as W
    n = 60  # distinct ROIs, repeated to fill the large call
    if fittype == 6:
        rois, _ = W.rois3d(n, s, np.random.default_rng(s))
        return rois, b.Model(6, W.coeff3d()), None
    if fittype == 7:
        w = W.workload_4d(n, sizes=(s,), stream=70 + s)[0]
        return w.rois, b.Model(7, w.coeff, init_p=w.init_p), [(21.0, 3.5), (31.0, 3.5), (41.0, 2.5)]
    if fittype == 8:
        w = W.workload_5d(n, s=s, stream=80 + s)
        other = w.init_p.copy()
        other[1] = 6.0
        return w.rois, b.Model(8, w.coeff, coeff3=w.coeff3, init_p=w.init_p), [w.init_p, other]
    w = W.workload_4pi(n, s=s, stream=90 + s)
    dT = np.random.default_rng(s).uniform(-0.4, 0.4, (n, 4, 6)).astype(np.float32)
    return w.rois, b.Model4Pi(w.coeff, w.extra["phase_shift"]), (w.extra["init_z"], w.extra["init_phi"], dT)


@pytest.mark.parametrize("fittype,s", [(f, s) for f, v in SIZES.items() for s in v])
def test_block_form_is_bit_identical(bsfit_mod, fittype, s):
    rois, model, extra = _setup(bsfit_mod, fittype, s)
    axis = 1 if fittype == 9 else 0
    rois = np.moveaxis(rois, axis, 0).copy()
    rois[1] = 0.0
    rois[2, ..., 0, 0] = np.nan
    rois[3] *= -1.0
    rois[4] = 7.0
    rois[5, ..., 1, 1] = np.inf
    many = np.resize(np.arange(len(rois)), BIG)

    def pick(idx):
        e = tuple(x[idx] for x in extra) if fittype == 9 else extra
        return np.moveaxis(rois[idx], 0, axis), e

    kinds = ["plain"] + (["starts"] if fittype != 6 else []) + (["scmos"] if fittype != 9 else [])
    for kind in kinds:
        for its in ((0, 1, 30) if kind == "plain" else (12,)):
            r, e = pick(many)
            ref = [x.cpu().numpy()[..., :] for x in _call(bsfit_mod, fittype, r, its, model, e, kind)]
            for n in (1, 150, 300, 400, 600, 740, 900):
                r, e = pick(many[:n])
                out = [x.cpu().numpy() for x in _call(bsfit_mod, fittype, r, its, model, e, kind)]
                for a, b in zip(out, ref):
                    assert np.array_equal(a, b[..., :n], equal_nan=True), (kind, its, n)
    model.close()


def test_ill_conditioned_solve_rounds_alike(bsfit_mod):
    """5D fits of 5 px ROIs: the refinement of their nearly singular steps is large
    enough that a contracted sum would show."""
    import torch
    from bsfit import workloads as W
    w = W.workload_5d(24000, s=5, stream=5)
    model = bsfit_mod.Model(8, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    r = torch.from_numpy(np.ascontiguousarray(w.rois)).cuda()
    ref = [x.cpu().numpy() for x in model.fit_torch(r, 3)]
    for n in (150, 300, 450, 600, 750):
        parts = [model.fit_torch(r[i:i + n].contiguous(), 3) for i in range(0, len(r) - n + 1, n)]
        for k, b in enumerate(ref):
            a = np.concatenate([p[k].cpu().numpy() for p in parts], axis=-1)
            assert np.array_equal(a, b[..., :a.shape[-1]], equal_nan=True), (n, k)
    model.close()
