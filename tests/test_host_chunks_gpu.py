"""The drop-in call's chunks: at the sizes where the last chunk is joined to the one
before, outputs bit-identical to one device call."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16384, 16385, 24575, 24576, 49152, 65535, 65536])
def test_chunks_equal_device_call(bsfit_mod, n):
    import torch
    from bsfit import workloads as W
    rois, _ = W.rois3d(500, 7, np.random.default_rng(4))
    rois = rois[np.resize(np.arange(500), n)]
    coeff = W.coeff3d()
    P, C, L = bsfit_mod.GPUmleFit_LM_multiD(rois, 6, 10, coeff)
    model = bsfit_mod.Model(6, coeff)
    ref = [x.cpu().numpy() for x in model.fit_torch(torch.from_numpy(rois).cuda(), 10)]
    model.close()
    for a, b in zip((P, C, L), ref):
        a = np.asarray(a)
        assert np.array_equal(a if a.shape == b.shape else a.T, b, equal_nan=True)
