"""The lattice transforms (type 1, type 2, forward, adjoint, sysmat) against the
FP64 oracle at the sizes where their tiles can go wrong: detectors and fine
grids that are not whole tiles (16 columns x 8 T lines, 4 x 4 cells, 32 rows,
64 and 256 columns), more than 256 fine-grid y, one angle, one detector row or
column, flat and thin volumes, tilts in every quadrant (footprints that wrap
around the fine grid), and every kernel width.

Tolerance: 1e-5 (the float positions' and float sums' share, as for every
operator) plus 10 eps for the kernel's own error in the four interpolated axes.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

CASES = [
    # volume, nproj, nrows, ncols, gamma, eps
    ((9, 5, 11), 3, 13, 17, 0.0, 1.2e-6),
    ((10, 10, 10), 5, 33, 63, 0.6, 1.2e-6),
    ((12, 7, 9), 1, 16, 65, np.pi / 2, 1.2e-6),
    ((8, 3, 30), 4, 21, 258, 2.2, 1.2e-6),
    ((30, 3, 8), 4, 40, 15, -2.5, 1.2e-6),
    ((5, 140, 4), 6, 30, 7, 0.9, 1.2e-6),
    ((1, 1, 1), 2, 4, 5, 0.4, 1.2e-6),
    ((6, 1, 7), 3, 1, 9, 0.4, 1.2e-6),
    ((6, 4, 7), 3, 9, 1, 5.0, 1.2e-6),
    ((7, 6, 5), 200, 24, 24, 0.3, 1.2e-6),
    ((11, 6, 9), 4, 18, 20, 0.7, 1e-3),
    ((11, 6, 9), 4, 18, 20, 0.7, 1e-4),
    ((11, 6, 9), 4, 18, 20, 0.7, 1e-5),
    ((11, 6, 9), 4, 18, 20, 0.7, 1e-7),
    ((103, 101, 105), 3, 16, 21, 0.6, 1.2e-6),  # over 8 million cells: the split fine-grid transform
]


@pytest.mark.parametrize("dims,nproj,nrows,ncols,gamma,eps", CASES)
def test_lattice_transforms_vs_oracle(L, O, dims, nproj, nrows, ncols, gamma, eps):
    rng = np.random.default_rng(31)
    tol = 1e-5 + 10 * eps
    th = rng.uniform(0, 2 * np.pi, nproj).astype(np.float32)
    pg = L.PolarGrid(th, nrows, ncols, np.float32(gamma))
    opg = O.PolarGrid(th, nrows, ncols, np.float32(gamma))
    plan, plan_o = L.NufftPlan(dims, eps), O.NufftPlan(dims, eps=1e-12)
    f = (rng.standard_normal(dims) + 1j * rng.standard_normal(dims)).astype(np.complex64)
    c = (rng.standard_normal(pg.dims()) + 1j * rng.standard_normal(pg.dims())).astype(np.complex64)
    assert rel(L.nufft3d2(f, pg, plan=plan), O.nufft3d2(f.astype(np.complex128), opg, plan_o)) < tol
    assert rel(L.nufft3d1(c, pg, dims, plan=plan), O.nufft3d1(c.astype(np.complex128), opg, plan_o)) < tol
    m = rng.standard_normal((3,) + dims).astype(np.float32)
    p = rng.standard_normal(pg.dims()).astype(np.float32)
    assert rel(L.forward(m, pg, plan=plan), O.forward(m, opg, opg.gamma, plan_o)) < tol
    assert rel(L.adjoint(p, pg, dims, plan=plan), O.adjoint(p, opg, dims, opg.gamma, plan_o)) < tol
    assert rel(L.sysmat(m, [pg, pg], plan=plan), 2 * O.sysmat(m, opg, opg.gamma, plan_o)) < tol


def test_columns_in_several_chunks(L, O):
    """A detector so wide that the node grid passes 4 GiB is taken in chunks of
    columns (here 25 T lines x 800 y x 8 bytes a column, 26816 columns at a time);
    a thin volume leaves sums that the oracle takes term by term.  Type 1 adds up to
    750 thousand nodes into a cell one after the other, whose rounding grows with
    the root of their number: 2^-24 sqrt(750e3) = 5e-5 beside the other 2.2e-5."""
    rng = np.random.default_rng(5)
    n, gamma, dims = 120_000, np.float32(0.6), (2, 400, 2)
    th = np.array([0.7], np.float32)
    pg, opg = L.PolarGrid(th, 1, n, gamma), O.PolarGrid(th, 1, n, gamma)
    plan, plan_o = L.NufftPlan(dims, 1.2e-6), O.NufftPlan(dims, exact=True)
    f = (rng.standard_normal(dims) + 1j * rng.standard_normal(dims)).astype(np.complex64)
    c = (rng.standard_normal(pg.dims()) + 1j * rng.standard_normal(pg.dims())).astype(np.complex64)
    assert rel(L.nufft3d2(f, pg, plan=plan), O.nufft3d2(f.astype(np.complex128), opg, plan_o)) < 2.2e-5
    assert rel(L.nufft3d1(c, pg, dims, plan=plan), O.nufft3d1(c.astype(np.complex128), opg, plan_o)) < 7.2e-5
