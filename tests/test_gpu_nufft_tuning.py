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
