"""A tuned configuration holds for the calls of the form that it was measured in: after
tuning on a sample, calls of fewer and of more ROIs run the kernels that they ran before,
and so they do with the choice restored from a cache file. A configuration that the caller
sets holds for every count; sCMOS and multi-start calls have none."""
import numpy as np
import pytest

from kernel_names import captured
from test_fit_gpu import bsfit_mod  # noqa: F401

pytestmark = pytest.mark.gpu

# counts fitted with one block, one warp and several ROIs per warp
COUNTS = {6: (1, 300, 3000, 60000), 7: (1, 300, 2000, 20000), 8: (1, 150, 1500, 12000)}
MID = 2  # index of the one-warp count


@pytest.fixture
def fits(bsfit_mod, request):
    import torch
    from bsfit import tuning as T
    from bsfit import workloads as W
    fittype = request.param
    w = (W.workload_3d(200, s=13, stream=930) if fittype == 6 else
         W.workload_4d(100, sizes=(13,), stream=931)[0] if fittype == 7 else W.workload_5d(40, s=13, stream=932))
    m = bsfit_mod.Model(fittype, w.coeff, coeff3=w.coeff3, init_p=w.init_p)
    r = torch.from_numpy(np.resize(w.rois, (max(COUNTS[fittype]),) + w.rois.shape[1:])).cuda()

    def kernels(n):
        return captured(lambda: m.fit_torch(r[:n], 4))[1]

    T._set(fittype, 13, -1, 0)
    yield m, r, kernels, fittype
    T._set(fittype, 13, -1, 0)
    m.close()


@pytest.mark.parametrize("fits", [6, 7, 8], indirect=True)
def test_other_counts_keep_their_form(bsfit_mod, fits, tmp_path):
    from bsfit import tuning as T
    m, r, kernels, fittype = fits
    counts = COUNTS[fittype]
    before = [kernels(n) for n in counts]
    assert all("team_kernel" in k[0] for k in before[:MID]) and "10fit_kernel" in before[MID][0]
    assert any("slot_kernel" in k for k in before[-1])
    cache = str(tmp_path / "tune.json")
    for at in range(len(counts)):
        ch = T.autotune(m, r[:counts[at]], 4, reps=1, cache=cache)
        assert T.current(fittype, 13) == (ch["variant"], ch["warps_per_block"])
        # the counts of other forms (the two smallest share theirs)
        others = [i for i in range(len(counts)) if i != at and max(i, at) >= MID]
        assert [kernels(counts[i]) for i in others] == [before[i] for i in others]
        T._set(fittype, 13, -1, 0)
        assert T.apply_cache(cache, T.device_name()) == 1
        assert T.current(fittype, 13) == (ch["variant"], ch["warps_per_block"])
        assert [kernels(counts[i]) for i in others] == [before[i] for i in others]
        T._set(fittype, 13, -1, 0)
    assert [kernels(n) for n in counts] == before


@pytest.mark.parametrize("fits", [6, 7, 8], indirect=True)
def test_restored_where_it_was_measured(bsfit_mod, fits):
    from bsfit import tuning as T
    m, r, kernels, fittype = fits
    counts = COUNTS[fittype]
    before = [kernels(n) for n in counts]
    T._set(fittype, 13, 1, 4)  # the caller's choice: every count
    chosen = [kernels(n) for n in counts]
    assert all("10fit_kernel" in k[-1] for k in chosen)
    assert chosen[-1][-1] == chosen[0][-1] != before[MID][0]
    for rois, at in ((0, MID), (counts[MID], MID), (counts[-1], len(counts) - 1)):
        T._set(fittype, 13, -1, 0)
        T._restore(fittype, 13, 1, 4, rois)  # rois 0: a file from before counts were kept
        now = [kernels(n) for n in counts]
        assert now == [chosen[i] if i == at else before[i] for i in range(len(counts))], rois


def test_batches_take_the_form_of_their_count(bsfit_mod):
    import torch
    from bsfit import tuning as T
    from bsfit import workloads as W
    w = W.workload_3d(200, s=13, stream=930)
    m = bsfit_mod.Model(6, w.coeff)
    r = torch.from_numpy(np.resize(w.rois, (60000, 13, 13))).cuda()
    few, many = bsfit_mod.Batch([(m, r[:4000], 4)]), bsfit_mod.Batch([(m, r, 4)])
    names = lambda b: captured(lambda: b.run())[1]  # noqa: E731
    T._set(6, 13, -1, 0)
    before = names(few), names(many)
    assert "slot_batch_kernel" in before[1][-1] and "slot" not in before[0][-1]
    try:
        T._restore(6, 13, 1, 4, 0)
        assert names(many) == before[1] and names(few) != before[0]
        T._set(6, 13, -1, 0)
        T._restore(6, 13, 1, 4, 60000)
        assert names(few) == before[0] and names(many) != before[1]
    finally:
        T._set(6, 13, -1, 0)
    m.close()


def test_scmos_and_multistart_have_no_configuration(bsfit_mod):
    import torch
    from bsfit import tuning as T
    from bsfit import workloads as W
    w = W.workload_4d(100, sizes=(13,), stream=931)[0]
    m = bsfit_mod.Model(7, w.coeff, init_p=w.init_p)
    r = torch.from_numpy(w.rois).cuda()
    var = torch.ones_like(r)
    calls = [lambda: m.fit_scmos_torch(r, var, 4), lambda: m.fit_multistart_torch(r, 4, [(21.0, 3.5), (31.0, 3.5)])]
    T._set(7, 13, -1, 0)
    before = [captured(c)[1][-1] for c in calls]
    try:
        T._set(7, 13, 0, 4)
        assert [captured(c)[1][-1] for c in calls] == before and all("team_kernel" in k for k in before)
    finally:
        T._set(7, 13, -1, 0)
    m.close()
