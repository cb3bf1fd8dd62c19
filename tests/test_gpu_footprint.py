"""The memory estimate that admits requests, against what a request takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,kind,dets,ndata", [(3, "toeplitz", (192, 192), 2), (3, "toeplitz", (192, 192), 6),
                                                    (3, "mixed", (64, 64), 3), (3, "toeplitz_fp16", (192, 100), 2),
                                                    (3, "nufft", (192, 192), 2), (2, "toeplitz", (192, 192), 2),
                                                    (1, "toeplitz", (192, 192), 2)])
def test_footprint_covers_a_request_without_waste(L, method, kind, dets, ndata):
    """Not less than the largest number of bytes in use, and not more than 2.5 times that:
    a quarter is the estimate's own slack, and of the setup and the solve, whose peaks
    it adds up part by part, only one has its maximum at a time."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    drv = pytest.importorskip("cuda.bindings.driver")
    import torch
    torch.zeros(1, device="cuda")
    rng = np.random.default_rng(0)
    recon = (128, 16, 128)
    data = [(rng.random((30,) + dets, dtype=np.float32), rng.uniform(0, 6, 30).astype(np.float32), np.float32(0.3 * i))
            for i in range(ndata)]
    par = L.ReconParams(maxIters=1, innerIters=2, op_kind=kind)
    fp = L.mbir_footprint(method, [d[0].shape for d in data], recon, par)
    high = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    _, pool = rt.cudaDeviceGetDefaultMemPool(0)
    torch.cuda.synchronize()
    rt.cudaMemPoolSetAttribute(pool, high, drv.cuuint64_t(0))
    if method == 3:
        L.mbir3_batch([(data, recon, par)], threads=1)
    else:
        with L.ReconServer(budget_bytes=10**11, slots=1) as srv:
            srv.wait(srv.submit(method, data, recon, par))
    used = int(rt.cudaMemPoolGetAttribute(pool, high)[1])
    assert used <= fp < 2.5 * used + (64 << 20)
