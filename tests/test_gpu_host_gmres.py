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


@pytest.mark.parametrize("nx,nv,precision", [(64, 256, "fp64"), (100, 201, "fp64"), (64, 256, "mixed")])
def test_multi_kernel_step_of_small_grids(monkeypatch, nx, nv, precision):
    """Grids whose steps run on a cluster by default, kept off it: the graph
    step and the host-driven one launch the same kernels (the tuner's variants,
    one choice for both) in the same order, and follow the oracle."""
    import numpy as np
    from vivlasov1d_b200.run import Run
    monkeypatch.setenv("VV_CLUSTER", "0")
    og = vo.Grid(nx, nv, 4 * math.pi, 10.0, -10.0, ht=0.1)
    f0 = vo.initialise_distribution_function(og, vo.f0_landau(0.05))
    cfg = {"grid": {"nx": nx, "nv": nv, "L": 4 * math.pi, "vmin": -10.0, "vmax": 10.0, "ht": 0.1, "nt": 1},
           "solver": {"method": "matrixfree", "poisson_bracket": "ArakawaJ4", "preconditioner_type": "tensor",
                      "preconditioner_scheme": "tensor_kinetic", "petsc_ksp_rtol": 1e-8, "petsc_snes_atol": 1e-11},
           "initial_data": {"charge": -1.0}}
    out = []
    for graph in ("1", "0"):
        monkeypatch.setenv("VV_GRAPH", graph)
        run = Run(cfg, f0=torch.from_numpy(vo.to_flat(f0)), precision=precision)
        run.ctx.launch_count(reset=True)
        reps = [run.step() for _ in range(2)]
        # several kernels an iteration: not one launch a step
        assert run.ctx.launch_count() > 4 * sum(sum(r["gmres_its"]) for r in reps) > 0
        out.append((run.fc.clone(), [(r["gmres_its"], r["residual"]) for r in reps]))
    assert out[0][1] == out[1][1]
    assert torch.equal(out[0][0], out[1][0])
    orun = vo.Run(og, f0, ksp_rtol=1e-8, snes_atol=1e-11)
    for _ in range(2):
        orun.step()
    # inside the 1e-11 residual ball: 2 ht atol a step
    got = vo.from_flat(out[0][0].cpu().numpy())
    assert np.linalg.norm(got - orun.fc) <= 2 * 2 * 0.1 * 1e-11 + 1e-12 * np.linalg.norm(orun.fc)
