"""The lattice transforms where their assumptions are tight: lines exactly one
cell apart, fine grids that end in part of a tile, angles that are not numbers,
memory that runs out between calls, more datasets than a plan's usual number."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _grids(L, O, rng, nproj, nrows, ncols, gamma):
    th = rng.uniform(0, 2 * np.pi, nproj).astype(np.float32)
    return L.PolarGrid(th, nrows, ncols, np.float32(gamma)), O.PolarGrid(th, nrows, ncols, np.float32(gamma))


def _check_all(L, O, rng, dims, pg, opg, eps):
    """Every lattice operator within 1e-5 (float positions and sums) plus 10 eps (the
    kernel's error in the four interpolated axes) of the FP64 oracle."""
    tol = 1e-5 + 10 * eps
    plan, plan_o = L.NufftPlan(dims, eps), O.NufftPlan(dims, eps=1e-12)
    f = (rng.standard_normal(dims) + 1j * rng.standard_normal(dims)).astype(np.complex64)
    c = (rng.standard_normal(pg.dims()) + 1j * rng.standard_normal(pg.dims())).astype(np.complex64)
    assert rel(L.nufft3d2(f, pg, plan=plan), O.nufft3d2(f.astype(np.complex128), opg, plan_o)) < tol
    assert rel(L.nufft3d1(c, pg, dims, plan=plan), O.nufft3d1(c.astype(np.complex128), opg, plan_o)) < tol
    m = rng.standard_normal((3,) + dims).astype(np.float32)
    p = rng.standard_normal(pg.dims()).astype(np.float32)
    assert rel(L.forward(m, pg, plan=plan), O.forward(m, opg, opg.gamma, plan_o)) < tol
    assert rel(L.adjoint(p, pg, dims, plan=plan), O.adjoint(p, opg, dims, opg.gamma, plan_o)) < tol
    assert rel(L.sysmat(m, pg, plan=plan), O.sysmat(m, opg, opg.gamma, plan_o)) < tol


@pytest.mark.parametrize("eps", [1e-3, 1e-5, 1e-7])
@pytest.mark.parametrize("gamma", [0.0, np.pi / 2, np.pi])
@pytest.mark.parametrize("dims", [(90, 6, 64), (64, 5, 90)])
def test_lines_one_cell_apart_even_widths(L, O, dims, gamma, eps):
    """No tilt, a quarter and half a turn: the T lines would lie on the cells of the
    fine grid, where the even kernel widths' footprints start at integers."""
    rng = np.random.default_rng(3)
    pg, opg = _grids(L, O, rng, 6, 24, 33, gamma)
    _check_all(L, O, rng, dims, pg, opg, eps)


@pytest.mark.parametrize("eps", [1e-3, 1e-4, 1e-7])
@pytest.mark.parametrize("dims,nproj,nrows,spread", [((9, 9, 9), 100, 120, 2 * np.pi), ((32, 9, 32), 200, 154, 2 * np.pi),
                                                     ((30, 15, 30), 240, 154, 0.2), ((9, 25, 9), 300, 120, 0.02)])
def test_short_last_tile(L, O, dims, nproj, nrows, spread, eps):
    """Fine grids along y of 18, 30 and 50 cells end in half a tile; many rows, all of
    them near y = 0 with a small spread of angles, meet it and both its neighbours."""
    rng = np.random.default_rng(8)
    th = rng.uniform(0, spread, nproj).astype(np.float32)
    g = np.float32(0.5)
    _check_all(L, O, rng, dims, L.PolarGrid(th, nrows, 7, g), O.PolarGrid(th, nrows, 7, g), eps)


@pytest.mark.parametrize("nrows,ncols", [(16, 20), (17, 19)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_angles_that_are_not_numbers(L, bad, nrows, ncols):
    """Such an angle has no positions: its rows are not numbers, the others are those
    of the geometry without it, and sums over all rows are not numbers."""
    rng = np.random.default_rng(6)
    dims, g = (10, 6, 12), np.float32(0.5)
    th = rng.uniform(0, 2 * np.pi, 4).astype(np.float32)
    pg = L.PolarGrid(np.concatenate([th[:1], [np.float32(bad)], th[1:]]), nrows, ncols, g)
    clean = L.PolarGrid(th, nrows, ncols, g)
    others = [0, 2, 3, 4]
    plan = L.NufftPlan(dims)
    m = rng.standard_normal((3,) + dims).astype(np.float32)
    got = L.forward(m, pg, plan=plan)
    assert np.isnan(got[1]).all()
    assert rel(got[others], L.forward(m, clean, plan=plan)) < 1e-6
    f = (rng.standard_normal(dims) + 1j * rng.standard_normal(dims)).astype(np.complex64)
    assert rel(L.nufft3d2(f, pg, plan=plan)[others], L.nufft3d2(f, clean, plan=plan)) < 1e-6
    assert np.isnan(L.adjoint(rng.standard_normal(pg.dims()).astype(np.float32), pg, dims, plan=plan)).all()
    assert np.isnan(L.sysmat(m, pg, plan=plan)).all()


SCRATCH = """
import numpy as np, torch
import lamino_b200 as L
rng = np.random.default_rng(2)
dims = (16, 64, 16)
grid = lambda n: L.PolarGrid(np.array([0.3], np.float32), 4, n, np.float32(0.6))
small, wide = grid(24), grid(50_000)   # node grids of 2 MB and 3 GB
m = torch.from_numpy(rng.standard_normal((3,) + dims).astype(np.float32)).cuda()
plan = L.NufftPlan(dims)
want = L.forward(m, small, plan=plan).clone()
free, _ = torch.cuda.mem_get_info()
filler = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")
try:
    L.forward(m, wide, plan=plan)
    raise SystemExit("the wide detector fitted")
except L.LaminoError as e:
    assert e.code == 2, e
assert torch.equal(L.forward(m, small, plan=plan), want)
del filler
torch.cuda.empty_cache()
assert torch.isfinite(L.forward(m, wide, plan=plan)).all()
assert torch.equal(L.forward(m, small, plan=plan), want)
print("kept")
"""


def test_scratch_survives_a_failed_allocation():
    """A node grid that finds no memory is an error of that call alone: the geometries
    the plan already knows go on with the scratch that it had.  In a process of its
    own, whose memory nothing else holds."""
    import subprocess
    import sys
    from conftest import ROOT
    r = subprocess.run([sys.executable, "-c", SCRATCH], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "kept", r.stdout + r.stderr


def test_more_datasets_than_a_plan_usually_keeps(L, O):
    """A solver over 18 tilts in the NUFFT form captures its operator after one call;
    by then every lattice is there.  Same result as without graphs, in float sums
    of another order at most."""
    rng = np.random.default_rng(12)
    recon = (8, 4, 8)
    data = [(rng.random((3, 8, 9), dtype=np.float32), rng.uniform(0, 2 * np.pi, 3).astype(np.float32), np.float32(0.15 * i))
            for i in range(18)]
    par = dict(maxIters=4, op_kind="nufft", tol=0.0, xtol=0.0)
    got = L.MBIR1(data, recon, L.ReconParams(**par))
    assert rel(got, L.MBIR1(data, recon, L.ReconParams(use_graphs=0, **par))) < 1e-5
    got = L.MBIR3(data, recon, L.ReconParams(**par))
    assert rel(got, L.MBIR3(data, recon, L.ReconParams(use_graphs=0, **par))) < 1e-5
    # and the operator over them, twice in a row
    pgs = [L.PolarGrid(th, 20, 21, g) for _, th, g in data]
    opgs = [O.PolarGrid(th, 20, 21, g) for _, th, g in data]
    x = rng.standard_normal((3, 11, 6, 11)).astype(np.float32)
    plan, plan_o = L.NufftPlan(x.shape[1:]), O.NufftPlan(x.shape[1:], eps=1e-12)
    want = O.normal(x, opgs, [p.gamma for p in opgs], plan_o)
    for _ in range(2):
        assert rel(L.sysmat(x, pgs, plan=plan), want) < 2.2e-5
