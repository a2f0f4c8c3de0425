"""Several ROIs in flight per warp (large calls): bit-identical to the small-call
forms, for every fit type, over ROI sizes (with room for four slots, two, none),
iteration caps, malformed ROIs, several starts, sCMOS variances, and batches whose
segments end inside a warp's slots."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu

BIG = 13000  # three ROIs for each of the most warps that stay resident, and more
CASES = [(6, 5), (6, 13), (6, 17), (6, 21), (6, 33), (7, 5), (7, 13), (7, 17), (7, 33), (8, 5), (8, 13), (8, 17)]


def _setup(b, fittype, s, n=40):
    from bsfit import workloads as W
    if fittype == 6:
        rois, _ = W.rois3d(n, s, np.random.default_rng(100 + s))
        return rois, b.Model(6, W.coeff3d()), None
    if fittype == 7:
        w = W.workload_4d(n, sizes=(s,), stream=170 + s)[0]
        return w.rois, b.Model(7, w.coeff, init_p=w.init_p), [(21.0, 3.5), (31.0, 3.5), (41.0, 2.5)]
    w = W.workload_5d(n, s=s, stream=180 + s)
    other = w.init_p.copy()
    other[1] = 6.0
    return w.rois, b.Model(8, w.coeff, coeff3=w.coeff3, init_p=w.init_p), [w.init_p, other]


def _spoil(rois):
    rois = rois.copy()
    rois[1] = 0.0
    rois[2, 0, 0] = np.nan
    rois[3] *= -1.0
    rois[4] = 7.0
    rois[5, 1, 1] = np.inf
    return rois


def _same(out, ref, n, many):
    for a, b in zip(out, ref):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.array_equal(a, np.take(b[..., :n], many, axis=-1), equal_nan=True)


@pytest.mark.parametrize("fittype,s", CASES)
def test_many_rois_equal_few(bsfit_mod, fittype, s):
    import torch
    rois, model, starts = _setup(bsfit_mod, fittype, s)
    rois = _spoil(rois)
    n = len(rois)
    big = 40000 if fittype == 6 else 9000 if fittype == 7 else 6000
    many = np.random.default_rng(s).integers(0, n, big)
    few = torch.from_numpy(rois).cuda()
    lots = few[torch.from_numpy(many).cuda()].contiguous()
    for its in (0, 1, 30):
        _same(model.fit_torch(lots, its), model.fit_torch(few, its), n, many)
    var = torch.from_numpy(np.random.default_rng(s).uniform(0.5, 4.0, rois.shape).astype(np.float32)).cuda()
    vlots = var[torch.from_numpy(many).cuda()].contiguous()
    _same(model.fit_scmos_torch(lots, vlots, 12), model.fit_scmos_torch(few, var, 12), n, many)
    if starts:
        for strict in (False, True):
            _same(model.fit_multistart_torch(lots, 12, starts, strict=strict),
                  model.fit_multistart_torch(few, 12, starts, strict=strict), n, many)
    model.close()


@pytest.mark.parametrize("fittype,sizes", [(6, (11, 13, 17)), (7, (9, 15)), (8, (13, 17))])
@pytest.mark.parametrize("several", [False, True])
def test_batches_equal_few(bsfit_mod, fittype, sizes, several):
    import torch
    if several and fittype == 6:
        pytest.skip("fit type 6 has one start")
    parts, entries, first = [], [], None
    big = 40000 if fittype == 6 else 9000 if fittype == 7 else 6000
    for k, s in enumerate(sizes + sizes[:1]):
        rois, model, starts = _setup(bsfit_mod, fittype, s)
        first = first or starts
        count = big if k == 0 else (big // 2 if k == 1 else 7 + k)  # the last segments are tiny
        many = np.random.default_rng(k).integers(0, len(rois), count)
        few = torch.from_numpy(_spoil(rois)).cuda()
        lots = few[torch.from_numpy(many).cuda()].contiguous()
        parts.append((model, few, len(rois), many))
        entries.append((model, lots, 12 + k))
    st = [first if k % 2 == 0 else None for k in range(len(entries))] if several else None
    batch = bsfit_mod.Batch(entries, starts=st)
    outs = batch.run()
    torch.cuda.synchronize()
    claimed, done = batch.counters()
    for k, ((model, few, n, many), out) in enumerate(zip(parts, outs)):
        assert done[k] == len(many) and claimed[k] >= len(many)
        if st and st[k]:
            ref = model.fit_multistart_torch(few, 12 + k, st[k])
        else:
            ref = model.fit_torch(few, 12 + k)
        _same(out, ref, n, many)
