"""The direct DFT of short rows (one tile of 32 modes, a warp per row) and just
beyond it, in length and (FP64, 1600 rows) in number, row blocks part full:
along x in the kinetic preconditioner, along the field's columns in the
potential one, and in FP32 inside a mixed step."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import vlasov_oracle as vo  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("nx,nv", [(5, 13), (6, 16), (17, 18), (31, 17), (33, 50), (61, 12), (62, 15), (63, 33),
                                   (65, 14), (66, 9), (55, 1601), (57, 1601), (59, 1599)])
def test_short_rows_match_oracle(nx, nv):
    """1e-12 (kinetic) and 1e-11 (potential) relative, as every variant of the preconditioners."""
    from vivlasov1d_b200.solver import Grid, TensorProductPreconditioner
    x = np.random.default_rng(nx + nv).standard_normal((nx, nv))
    og, grid = vo.Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05), Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05)
    X, Y = torch.from_numpy(vo.to_flat(x)).cuda(), grid.field()
    TensorProductPreconditioner.create("tensor_kinetic", grid=grid).tensorProduct(X, Y)
    want = vo.TensorKineticPreconditioner(og).apply(x)
    assert np.abs(vo.from_flat(Y.cpu().numpy()) - want).max() <= 1e-12 * np.abs(want).max()
    # the transform runs along v there: the sizes change places
    og, grid = vo.Grid(nv, nx, 4 * np.pi, 8.0, ht=0.05), Grid(nv, nx, 4 * np.pi, 8.0, ht=0.05)
    phi = 0.3 * np.cos(0.5 * np.arange(nv) * og.hx)
    X, Y = torch.from_numpy(vo.to_flat(np.ascontiguousarray(x.T))).cuda(), grid.field()
    TensorProductPreconditioner.create("tensor_potential", grid=grid, phi=torch.from_numpy(phi).cuda()).tensorProduct(X, Y)
    want = vo.TensorPotentialPreconditioner(og, phi).apply(np.ascontiguousarray(x.T))
    assert np.linalg.norm(vo.from_flat(Y.cpu().numpy()) - want) <= 1e-11 * np.linalg.norm(want)


@pytest.mark.parametrize("nx,nv", [(17, 40), (62, 41), (63, 42), (66, 43)])
def test_short_rows_mixed_step(monkeypatch, nx, nv):
    """FP32 inner solves: both runs stop inside the 1e-11 residual ball (2 ht atol)."""
    from vivlasov1d_b200.run import Run
    monkeypatch.setenv("VV_CLUSTER", "0")
    cfg = {"grid": {"nx": nx, "nv": nv, "L": 4 * np.pi, "vmin": -8.0, "vmax": 8.0, "ht": 0.1, "nt": 1},
           "solver": {"method": "matrixfree", "poisson_bracket": "ArakawaJ4", "preconditioner_type": "tensor",
                      "preconditioner_scheme": "tensor_kinetic", "petsc_ksp_rtol": 1e-4, "petsc_snes_atol": 1e-11,
                      "petsc_snes_max_iter": 20},
           "initial_data": {"charge": -1.0}}
    og = vo.Grid(nx, nv, 4 * np.pi, 8.0, -8.0, ht=0.1)
    f0 = torch.from_numpy(vo.to_flat(vo.initialise_distribution_function(og, vo.f0_twostream(0.05, 0.5))))
    a, b = Run(cfg, f0=f0, precision="mixed"), Run(cfg, f0=f0)
    ra, rb = a.step(), b.step()
    assert ra["residual"][-1] < 1e-11 and rb["residual"][-1] < 1e-11
    assert float((a.fc - b.fc).norm()) <= 2 * 0.1 * 1e-11 + 1e-12 * float(b.fc.norm())


@pytest.mark.parametrize("nx", [4417, 4600, 4735])
def test_longest_direct_rows(nx):
    """The longest rows whose twiddles and four rows fit a block's shared memory
    (48 nx bytes of 227,312).  A row's sums of nx products round to some
    sqrt(nx) 1.1e-16 < 1e-14 of its size: 1e-12 as for the short rows."""
    from vivlasov1d_b200.solver import Grid, TensorProductPreconditioner
    nv = 6
    x = np.random.default_rng(nx).standard_normal((nx, nv))
    og, grid = vo.Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05), Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05)
    X, Y = torch.from_numpy(vo.to_flat(x)).cuda(), grid.field()
    TensorProductPreconditioner.create("tensor_kinetic", grid=grid).tensorProduct(X, Y)
    want = vo.TensorKineticPreconditioner(og).apply(x)
    assert np.abs(vo.from_flat(Y.cpu().numpy()) - want).max() <= 1e-12 * np.abs(want).max()
