"""What a call leaves in the library's pool goes back to the device on request."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def test_trim_gives_the_pool_back(L):
    """A reconstruction leaves its buffers (some 100 MB here) in the pool; after trim()
    they are free again, and the next call works.  16 MB for what the first call
    loads for good (modules, cuFFT's own tables)."""
    import torch
    rng = np.random.default_rng(0)
    data = [(rng.random((40, 96, 96), dtype=np.float32), rng.uniform(0, 6, 40).astype(np.float32), np.float32(0.3))]
    par = L.ReconParams(maxIters=1)
    want = L.MBIR1(data, (96, 12, 96), par)
    torch.cuda.synchronize()
    L.trim()
    before, _ = torch.cuda.mem_get_info()
    L.MBIR1(data, (96, 12, 96), par)
    torch.cuda.synchronize()
    kept, _ = torch.cuda.mem_get_info()
    assert kept < before - (64 << 20)
    L.trim()
    after, _ = torch.cuda.mem_get_info()
    assert after > before - (16 << 20)
    # (the setup adjoint adds rows by atomics: two runs agree to the bar of the batched form)
    assert rel(L.MBIR1(data, (96, 12, 96), par), want) < 1e-5
