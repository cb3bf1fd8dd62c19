"""Toeplitz operators over detectors narrower than the volume: the voxel distances
along the detector reach its period, where the kernel's quotient is 0 / 0."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrows,ncols", [(11, 13), (12, 7), (10, 16), (49, 9)])
@pytest.mark.parametrize("gammas", [(0.0,), (np.pi, 0.6), (np.pi / 2, 0.0)])
@pytest.mark.parametrize("dims", [(15, 4, 33), (60, 5, 14)])
def test_toeplitz_detector_narrower_than_the_volume(L, O, dims, gammas, nrows, ncols):
    """Against the sum of the datasets' A^H A; 1e-5 as for every operator.  The angles
    0 and pi / 2 put the other detector axis on integers as well."""
    rng = np.random.default_rng(9)
    pgs, opgs = [], []
    for g in gammas:
        th = np.concatenate([[0.0, np.pi / 2], rng.uniform(0, 2 * np.pi, 4)]).astype(np.float32)
        pgs.append(L.PolarGrid(th, nrows, ncols, np.float32(g)))
        opgs.append(O.PolarGrid(th, nrows, ncols, np.float32(g)))
    x = rng.standard_normal((3,) + dims).astype(np.float32)
    want = O.normal(x, opgs, [p.gamma for p in opgs], O.NufftPlan(dims, eps=1e-12))
    assert rel(L.ToeplitzNormal(pgs, dims)(x), want) < 1e-5


@pytest.mark.parametrize("method", [1, 2, 3])
def test_reconstruction_detector_narrower_than_the_volume(L, O, method):
    """The drivers' sums, whole and per dataset; 1e-4 as for the other reconstructions."""
    recon = (14, 5, 15)
    rng = np.random.default_rng(4)
    data = [(rng.random((5, 4, 3), dtype=np.float32) + 0.05, rng.uniform(0, 2 * np.pi, 5).astype(np.float32), np.float32(g))
            for g in (0.0, 0.8)]
    par = dict(maxIters=3)
    want = {1: O.MBIR1, 2: O.MBIR2, 3: O.MBIR3}[method](data, recon, O.ReconParams(**par), exact=True)
    assert rel({1: L.MBIR1, 2: L.MBIR2, 3: L.MBIR3}[method](data, recon, L.ReconParams(**par)), want) < 1e-4
