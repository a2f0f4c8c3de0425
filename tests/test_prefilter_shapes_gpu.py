"""Coefficient builder over its forms: planes in shared memory and too large for
it, lines in shared memory and too long for it, axes of one and two samples, one
to five axes, each against the numpy restatement of bsarray (bounds as
test_prefilter_gpu.py)."""
import numpy as np
import pytest

from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [(1,), (2,), (300,), (9000,), (1, 9), (9, 1), (33, 31), (300, 300), (3, 9000), (9000, 3),
          (61, 26, 26), (2, 3, 4), (5, 1, 1, 7, 8), (1, 1, 1), (3, 2, 2, 2, 2), (900, 33, 31),
          (2000, 5, 4), (6, 900, 3, 3), (5, 9, 20, 17, 16)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_shapes_match_restatement(bsfit_mod, shape):
    import torch
    from bsfit import prefilter
    x = np.random.default_rng(sum(shape)).random(shape)
    ref = prefilter.bsarray_coeffs(x)
    d = torch.from_numpy(x).cuda()
    c32, c64 = bsfit_mod.bsarray_coeffs_torch(d, out64=True)
    only32 = bsfit_mod.bsarray_coeffs_torch(d)
    torch.cuda.synchronize()
    scale = np.abs(ref).max()
    assert np.abs(c64.cpu().numpy() - ref).max() <= 1e-13 * scale
    assert torch.equal(c32, c64.float()) and torch.equal(only32, c32)
    assert torch.equal(d.cpu(), torch.from_numpy(x))  # the samples are only read
