"""The NUFFT form has nothing to tune: a reconstruction does not time it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [1, 3])
def test_reconstruction_times_nothing_in_the_nufft_form(L, method):
    rng = np.random.default_rng(1)
    data = [(rng.random((4, 11, 13), dtype=np.float32), rng.uniform(0, 6, 4).astype(np.float32), np.float32(0.4))]
    par = L.ReconParams(maxIters=2, op_kind="nufft", autotune=1)
    {1: L.MBIR1, 3: L.MBIR3}[method](data, (11, 5, 10 + method), par)
    assert L.mbir_phases()["tune_s"] == 0.0


def test_autotune_times_a_warm_operator(L):
    """The time of objective 'normal' is that of a repeated operator; building the
    tables first takes as long again (2.5 for 1.2 ms at this size)."""
    import torch
    rng = np.random.default_rng(7)
    dims = (180, 16, 180)
    pgs = [L.PolarGrid(rng.uniform(0, 6, 91).astype(np.float32), 309, 309, np.float32(g)) for g in (0.0, 0.7)]
    plan = L.NufftPlan(dims)
    _, ms = plan.autotune(pgs, "normal")
    x = torch.zeros((3,) + dims, device="cuda")
    times = []
    for _ in range(10):
        e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e[0].record()
        L.sysmat(x, pgs, plan=plan)
        e[1].record()
        e[1].synchronize()
        times.append(e[0].elapsed_time(e[1]))
    assert 0 < ms < 1.5 * sorted(times)[5]
