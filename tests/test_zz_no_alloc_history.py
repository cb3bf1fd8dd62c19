"""lamino_residual_noalloc does not depend on the calls before it.  The file is
named to be collected last, as its neighbour."""
import numpy as np
import pytest

from test_zz_no_alloc import _bind, _call

pytestmark = pytest.mark.gpu


def test_residual_noalloc_same_points_with_and_without_a_lattice(L):
    """A new plan takes the point kernel, a plan that lamino_residual has used the
    lattice; both evaluate the same points.  Four voxels at the corners of a wide
    volume and two detector points, picked for the float rounding of the points'
    coordinates to show (3e-5 of the value); 1e-5 as for every operator."""
    import torch
    rng = np.random.default_rng(515)
    th = rng.uniform(0, 2 * np.pi, 1).astype(np.float32)
    f = np.zeros((3, 1100, 6, 1100), np.float32)
    for v in ((2, 1, 5), (1097, 4, 1090), (3, 2, 1094), (1095, 0, 4)):
        f[(slice(None),) + v] = 30 * rng.standard_normal(3)
    pg = L.PolarGrid(th, 1, 2, np.float32(0.6))
    f = torch.from_numpy(f).cuda()
    yT = torch.zeros_like(f)
    fn, plan = _bind(L), L.NufftPlan(f.shape[1:])
    fresh = _call(L, fn, plan, pg, f, yT, 1e3)
    ref = L.residual(f, yT, pg, 1e3, plan=plan)
    assert fresh == pytest.approx(ref, rel=1e-5)
    assert _call(L, fn, plan, pg, f, yT, 1e3) == pytest.approx(fresh, rel=1e-5)
