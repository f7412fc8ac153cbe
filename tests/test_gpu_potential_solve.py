"""The x solves of the potential preconditioner where the modes of a block
change: 8, 4, 2 and 1 modes whole in shared memory, then global memory, with
remainders of modes (nv/2 + 1 = 7, 9), rows transformed from the field's
columns (direct DFT) and by FFT, against the oracle (numpy FFTs, LAPACK
zgbtrf/zgbtrs); a smooth phi and a rough one that interchanges rows.  Tolerance:
the result moves by at most 40 times a relative change of x or phi (measured on
the oracle), and some 1e3 roundings of 1.1e-16 enter: 5e-12 < 1e-11."""
import numpy as np
import pytest
import torch

from oracle import vlasov_oracle as vo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [13, 16])
@pytest.mark.parametrize("nx", [8, 75, 76, 151, 152, 303, 304, 606, 607])
def test_potential_solve_block_sizes(nx, nv):
    from vivlasov1d_b200 import Grid, TensorProductPreconditioner
    og = vo.Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05)
    grid = Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05)
    rng = np.random.default_rng(nx + nv)
    xg = np.arange(nx) * og.hx
    x = rng.standard_normal((nx, nv))
    for phi in (0.3 * np.cos(0.5 * xg), 5.0 * rng.standard_normal(nx).cumsum()):
        ref = vo.TensorPotentialPreconditioner(og, phi).apply(x)
        assert np.isfinite(ref).all()
        pc = TensorProductPreconditioner.create("tensor_potential", grid=grid, phi=torch.from_numpy(phi).cuda())
        Y = grid.field()
        pc.tensorProduct(torch.from_numpy(vo.to_flat(x)).cuda(), Y)
        out = vo.to_flat(ref)
        assert np.linalg.norm(Y.cpu().numpy().ravel() - out.ravel()) < 1e-11 * np.linalg.norm(out)
