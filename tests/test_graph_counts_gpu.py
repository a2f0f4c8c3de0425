"""CUDA graphs at other counts than the warm-up call's: a capture of another form of
the fit replays with the results of the direct call, and the double-precision fit's
capture records its launch alone at every count."""
import numpy as np
import pytest

from kernel_names import KERNEL, captured
from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


def _model(b, fittype, n):
    import torch
    from bsfit import workloads as W
    if fittype == 6:
        w = W.workload_3d(min(n, 500), s=13, stream=1060)
    elif fittype == 7:
        w = W.workload_4d(min(n, 200), sizes=(13,), stream=1061)[0]
    else:
        w = W.workload_5d(min(n, 60), s=13, stream=1062)
    r = torch.from_numpy(np.resize(w.rois, (n,) + w.rois.shape[1:])).cuda()
    return b.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p), r


def _replays(call):
    import torch
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        out = call()
    g.replay()
    torch.cuda.synchronize()
    got = [x.cpu().numpy().copy() for x in out]
    ref = [x.cpu().numpy() for x in call()]
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got, ref))


@pytest.mark.parametrize("fittype,warm,counts", [(6, 20000, (1, 300, 600, 3000, 60000)), (7, 12000, (1, 300, 700, 2000)),
                                                 (8, 6000, (1, 300, 600, 1500))])
def test_capture_at_other_counts(bsfit_mod, fittype, warm, counts):
    m, r = _model(bsfit_mod, fittype, max(counts + (warm,)))
    m.fit_torch(r[:warm], 5)
    for n in counts:
        _replays(lambda: m.fit_torch(r[:n], 5))
    m.close()


def test_capture_of_a_large_batch(bsfit_mod):
    m, r = _model(bsfit_mod, 6, 60000)
    b = bsfit_mod.Batch([(m, r[:300], 5)])
    b.run()
    many = bsfit_mod.Batch([(m, r, 5)])
    _replays(lambda: many.run()[0])
    assert any("slot_batch_kernel" in k for k in captured(lambda: many.run())[1])
    m.close()


@pytest.mark.parametrize("fittype,counts", [(6, (50, 700, 1300, 2000)), (7, (20, 700, 1400)), (8, (10, 400))])
def test_fp64_capture_is_the_launch_alone(bsfit_mod, fittype, counts):
    m, r = _model(bsfit_mod, fittype, max(counts))
    m.fit_f64_torch(r[:10], 2)  # the model's double tables
    for n in counts:
        types, names = captured(lambda: m.fit_f64_torch(r[:n], 2))
        assert types == [KERNEL] and "fit64_kernel" in names[0], (n, types)
        _replays(lambda: m.fit_f64_torch(r[:n], 2))
    m.close()
