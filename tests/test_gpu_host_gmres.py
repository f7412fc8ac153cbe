"""The host-driven GMRES, which launches the next step's operator before it has
read the last step's status, against the time-step graph's loops over the same
kernels: the same bits, for solves that end inside a cycle, at its end and
after several."""
import math

import pytest
import torch

from oracle import vlasov_oracle as vo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [1, 2, 3, 5, 30])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_host_driven_equals_graph(monkeypatch, restart, precision):
    from vivlasov1d_b200.run import Run
    monkeypatch.setenv("VV_SHAPE", "1,2,1,0,0")   # one fixed shape, the multi-kernel path
    og = vo.Grid(128, 96, 4 * math.pi, 10.0, -10.0, ht=0.1)
    f0 = torch.from_numpy(vo.to_flat(vo.initialise_distribution_function(og, vo.f0_landau(0.2))))
    cfg = {"grid": {"nx": 128, "nv": 96, "L": 4 * math.pi, "vmin": -10.0, "vmax": 10.0, "ht": 0.1, "nt": 1},
           "solver": {"method": "matrixfree", "poisson_bracket": "ArakawaJ4", "preconditioner_type": "tensor",
                      "preconditioner_scheme": "tensor_kinetic", "petsc_ksp_rtol": 1e-6, "petsc_snes_atol": 1e-10},
           "initial_data": {"charge": -1.0}}
    out = []
    for graph in ("1", "0"):
        monkeypatch.setenv("VV_GRAPH", graph)
        run = Run(cfg, f0=f0, precision=precision)
        run.ksp.restart = restart
        reps = [run.step() for _ in range(2)]
        out.append((run.fc.clone(), [(r["gmres_its"], r["residual"]) for r in reps]))
    assert out[0][1] == out[1][1]
    assert torch.equal(out[0][0], out[1][0])
