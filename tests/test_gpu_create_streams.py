"""A context is complete when its constructor returns: its first call may be on
a stream that does not wait for the default one.  The second context of a shape
takes its variants from the tuner's cache, so that no timing waits for its tables."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import vlasov_oracle as vo  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("kind,nx,nv,env", [("tensor_kinetic", 1024, 1024, {}),
                                            ("tensor_kinetic", 1024, 1024, {"VV_SHAPE": "3,1,0,0,0"}),
                                            ("tensor_potential", 75, 101, {}),
                                            ("tensor_potential", 75, 101, {"VV_AUTOTUNE": "0"})])
def test_new_context_on_a_side_stream(monkeypatch, kind, nx, nv, env):
    """1e-11: the bound of the preconditioner tests (1e-12 kinetic, 1e-11 potential)."""
    from vivlasov1d_b200.solver import Grid, TensorProductPreconditioner
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    og = vo.Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05)
    phi = 0.3 * np.cos(0.5 * np.arange(nx) * og.hx)
    x = np.random.default_rng(nx + nv).standard_normal((nx, nv))
    want = (vo.TensorPotentialPreconditioner(og, phi) if kind == "tensor_potential"
            else vo.TensorKineticPreconditioner(og)).apply(x)
    X, P = torch.from_numpy(vo.to_flat(x)).cuda(), torch.from_numpy(phi).cuda()
    Ys = [torch.empty_like(X) for _ in range(2)]
    torch.cuda.synchronize()
    keep = []
    with torch.cuda.stream(torch.cuda.Stream()):
        for Y in Ys:
            pc = TensorProductPreconditioner.create(kind, grid=Grid(nx, nv, 4 * np.pi, 8.0, ht=0.05),
                                                    phi=P if kind == "tensor_potential" else None)
            pc.tensorProduct(X, Y)
            keep.append(pc)
    torch.cuda.synchronize()
    for Y in Ys:
        got = vo.from_flat(Y.cpu().numpy(), nx, nv)
        assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
