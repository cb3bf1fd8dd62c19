"""The branches of the Toeplitz and prior kernels that depend on the datasets and
the volume: sums of datasets without tilt, groups of up to four datasets with
their own spectra, tile heights, and the powers' range."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gammas", [(0.0,), (0.9, 0.0), (0.0, 0.5, 0.0)])
def test_toeplitz_untilted_datasets(L, O, gammas):
    """A dataset without tilt takes its sums from a table over (d_z, d_y), at any
    place among the others.  Tolerance: that of the other float operators."""
    rng = np.random.default_rng(17)
    dims = (9, 4, 11)
    ths = [rng.uniform(0, 2 * np.pi, 5 + i).astype(np.float32) for i in range(len(gammas))]
    pgs = [L.PolarGrid(t, 13, 12, np.float32(g)) for t, g in zip(ths, gammas)]
    opgs = [O.PolarGrid(t, 13, 12, np.float32(g)) for t, g in zip(ths, gammas)]
    x = rng.standard_normal((3,) + dims).astype(np.float32)
    want = O.normal(x, opgs, [p.gamma for p in opgs], O.NufftPlan(dims, eps=1e-12))
    assert rel(L.ToeplitzNormal(pgs, dims)(x), want) < 1e-5


@pytest.mark.parametrize("gammas", [(0.6,), (0.0, 0.8, 2.1), (0.4, 0.0, 0.9, 1.7, 2.6), (0.1,) * 8])
def test_mbir3_dataset_counts(L, O, gammas):
    """MBIR3 keeps a spectrum per dataset and takes them four at a time.  Bar as for
    the other reconstructions: 1e-4 of the FP64 oracle's volume."""
    recon = (8, 5, 9)
    rng = np.random.default_rng(4)
    m = O.synthetic_magnetization(recon, seed=4, sigma=1.0).astype(np.float64)
    plan = O.NufftPlan(recon, exact=True)
    data = []
    for g in gammas:
        th = rng.uniform(0, 2 * np.pi, 5).astype(np.float32)
        pg = O.PolarGrid(th, 9, 11, np.float32(g))
        data.append(((O.forward(m, pg, pg.gamma, plan) + 0.05).astype(np.float32), th, np.float32(g)))
    want = O.MBIR3(data, recon, O.ReconParams(maxIters=4), exact=True)
    assert rel(L.MBIR3(data, recon, L.ReconParams(maxIters=4)), want) < 1e-4


@pytest.mark.parametrize("n2", [3, 10, 11, 12, 13, 14, 16, 17, 22, 31])
def test_qggmrf_tile_heights(L, O, n2):
    """Every tile height (8, 10, 12, 14 rows), full and with rows left over; 1e-6 as
    for the other prior tests."""
    rng = np.random.default_rng(n2)
    x = rng.standard_normal((7, n2, 35)).astype(np.float32)
    g = np.zeros_like(x)
    want = O.qggmrf(g, x, 10.0, 1.1)
    L.opt.qggmrf(g, x, 10.0, 1.1)
    assert rel(g, want) < 1e-6


@pytest.mark.parametrize("scale", [1e-38, 1e-20, 1e-3, 1e6, 1e15])
@pytest.mark.parametrize("p", [1.0, 1.2, 1.5, 2.0, 2.3])
def test_qggmrf_powers(L, O, scale, p):
    """Differences from below the normal numbers to 1e15, exponents 2 - p of either
    sign and zero: the polynomials and the powf that takes over beyond them.  The
    oracle's values are rounded to the result's type: at 1e-38 and p = 2.3 they lie
    below its range (norm 4e-48)."""
    rng = np.random.default_rng(23)
    x = (scale * rng.standard_normal((6, 9, 40))).astype(np.float32)
    g = np.zeros_like(x)
    want = O.qggmrf(g, x, 1.0, p).astype(np.float32)
    L.opt.qggmrf(g, x, 1.0, p)
    assert rel(g, want) < 1e-6
