"""The prior gradient near the ends of the float range."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(6, 9, 40), (7, 14, 35), (5, 22, 33)])
def test_qggmrf_large_ratio(L, O, dims):
    """(|delta| / sigma)^(2 - p) between 2^126 and the largest float, whose reciprocal is
    below the normal numbers.  Neighbours always differ: eight values, one to each
    corner of a 2 x 2 x 2 cell.  The reciprocal has 2^-149 / 2 on 2.9e-39 at worst,
    2.4e-7, beside the few 6e-8 of the other operations: 1e-6 as for the other priors."""
    sigma, p = np.float32(1e-18), 1.3
    i, j, k = np.indices(dims) % 2
    x = ((4 * i + 2 * j + k) * 1.58e36).astype(np.float32)
    ratio = (np.array([1.58e36, 7 * 1.58e36]) / float(sigma)) ** (2.0 - float(np.float32(p)))
    assert 2.0 ** 126 < ratio[0] and ratio[1] < 3.4e38
    g = np.zeros_like(x)
    want = O.qggmrf(g, x, sigma, p)
    assert 0 < np.abs(want[1:-1, 1:-1, 1:-1]).min() and np.abs(want).max() < 3e38
    L.opt.qggmrf(g, x, float(sigma), p)
    assert rel(g, want) < 1e-6
