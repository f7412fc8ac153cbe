"""The cluster-resident step (vv_cluster.cuh) at the edges of its shapes.

One thread-block cluster advances an instance by a whole step; VV_CLUSTER=n
fixes its CTAs and 0 selects the multi-kernel step.  The two run the same
algorithm with other summation orders: f agrees to 1e-12 of its norm (500 times
the spread of the multi-kernel variants among themselves, 2e-15) where both
stop at the same pass, and against the oracle likewise.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import vlasov_oracle as vo  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _cfg(nx, nv, bracket="ArakawaJ4", atol=1e-11, rtol=1e-8, max_iter=20, max_it=1000):
    return {"grid": {"nx": nx, "nv": nv, "L": 4 * np.pi, "vmin": -8.0, "vmax": 8.0, "ht": 0.1, "nt": 1},
            "solver": {"method": "matrixfree", "poisson_bracket": bracket, "preconditioner_type": "tensor",
                       "preconditioner_scheme": "tensor_kinetic", "petsc_ksp_rtol": rtol, "petsc_snes_atol": atol,
                       "petsc_snes_max_iter": max_iter, "petsc_ksp_max_iter": max_it},
            "initial_data": {"charge": -1.0}}


def _run(monkeypatch, ctas, nx, nv, precision="fp64", restart=30, **kw):
    from vivlasov1d_b200.run import Run
    monkeypatch.setenv("VV_CLUSTER", str(ctas))
    og = vo.Grid(nx, nv, 4 * np.pi, 8.0, -8.0, ht=0.1)
    f0 = vo.initialise_distribution_function(og, vo.f0_twostream(0.05, 0.5))
    r = Run(_cfg(nx, nv, **kw), f0=torch.from_numpy(vo.to_flat(f0)), precision=precision, restart=restart)
    monkeypatch.delenv("VV_CLUSTER")
    return r, og, f0


def _rel(a, b):
    return float((a - b).norm() / b.norm())


# smallest grids, rows shared out unevenly or to few CTAs, one row per CTA,
# odd and prime nx, every FFT length, the longest chunks and the widest rows
SHAPES = [(4, 8, 16), (5, 17, 16), (16, 16, 16), (20, 20, 8), (31, 33, 4), (33, 50, 16), (64, 17, 16), (64, 31, 2),
          (64, 256, 1), (64, 250, 16), (128, 129, 8), (256, 130, 16), (512, 64, 16), (100, 201, 16), (254, 40, 16)]


@pytest.mark.parametrize("nx,nv,ctas", SHAPES)
def test_cluster_step_matches_oracle(monkeypatch, nx, nv, ctas):
    """f and the profiles against the oracle; the pass and iteration counts
    against the multi-kernel step (whose arithmetic this one shares)."""
    run, og, f0 = _run(monkeypatch, ctas, nx, nv)
    ref, _, _ = _run(monkeypatch, 0, nx, nv)
    orun = vo.Run(og, f0, ksp_rtol=1e-8, snes_atol=1e-11)
    for _ in range(2):
        rep, mrep, orep = run.step(), ref.step(), orun.step()
        assert rep["picard_its"] == mrep["picard_its"] == orep.picard_its
        # the multi-kernel variants differ by one among themselves (the autotuner's choice)
        assert all(abs(a - b) <= 1 for a, b in zip(rep["gmres_its"], mrep["gmres_its"]))
    f = vo.from_flat(run.fc.cpu().numpy())
    assert np.linalg.norm(f - orun.fc) <= 1e-12 * np.linalg.norm(orun.fc)
    for mine, want in ((run.N, orun.n), (run.E, orun.e), (run.pc_int, orun.phi), (run.h1c, orun.h1c)):
        assert np.abs(mine.cpu().numpy() - want).max() <= 1e-11 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("bracket", ["ArakawaJ1", "ArakawaJ2"])
def test_cluster_step_brackets(monkeypatch, bracket):
    a, _, _ = _run(monkeypatch, 16, 64, 130, bracket=bracket)
    b, _, _ = _run(monkeypatch, 0, 64, 130, bracket=bracket)
    ra, rb = a.step(), b.step()
    assert ra["picard_its"] == rb["picard_its"]
    assert _rel(a.fc, b.fc) <= 1e-12


@pytest.mark.parametrize("nx,nv,ctas", [(64, 128, 4), (64, 2048, 16), (256, 1024, 16), (512, 300, 16), (50, 101, 16)])
def test_cluster_step_mixed(monkeypatch, nx, nv, ctas):
    """FP32 inner solves: the FP64 residual is refined to atol either way; two
    runs that stop inside the 1e-11 residual ball differ in f by at most
    2 ht atol in the 2-norm (the Jacobian is I/ht plus a skew part)."""
    a, _, _ = _run(monkeypatch, ctas, nx, nv, precision="mixed", rtol=1e-4)
    b, _, _ = _run(monkeypatch, 0, nx, nv, precision="mixed", rtol=1e-4)
    for _ in range(2):
        ra, rb = a.step(), b.step()
        assert ra["residual"][-1] < 1e-11 and rb["residual"][-1] < 1e-11
    assert float((a.fc - b.fc).norm()) <= 2 * 2 * 0.1 * 1e-11 + 1e-12 * float(b.fc.norm())


@pytest.mark.parametrize("restart", [1, 3, 32])
def test_cluster_restarts(monkeypatch, restart):
    """Restarted cycles (r = b - P^-1 J x) of the solve alone and of a step."""
    import ctypes as C
    from vivlasov1d_b200 import _lib
    outs = []
    for ctas in (8, 0):
        run, _, _ = _run(monkeypatch, ctas, 64, 96, restart=restart, rtol=1e-9, max_it=400)
        run.step()
        gen = torch.Generator(device="cuda").manual_seed(3)
        b = torch.rand(96, 64, generator=gen, dtype=torch.float64, device="cuda")
        x = torch.empty_like(b)
        o = _lib.vv_ksp_opts(rtol=1e-9, atol=1e-50, dtol=1e5, max_it=400, restart=restart)
        r = _lib.vv_ksp_result()
        run.ctx.call("vv_gmres", run.ctx.field(b), run.ctx.field(x), C.byref(o), C.byref(r))
        outs.append((run.fc.clone(), x, r.its, r.reason))
    (fa, xa, ia, ra), (fb, xb, ib, rb) = outs
    assert ra == rb and abs(ia - ib) <= 1
    assert _rel(fa, fb) <= 1e-11
    assert _rel(xa, xb) <= 1e-8      # both within rtol 1e-9 of the solution


def test_cluster_revert(monkeypatch):
    """A tolerance below round-off ends with a rejected pass: f is the iterate
    before it, with its residual."""
    run, _, _ = _run(monkeypatch, 16, 64, 128, atol=1e-300)
    rep = run.step()
    assert rep["stop_rule"] == "rose" and rep["reverted"]
    assert run.calculate_residual() == pytest.approx(rep["residual"][-2], rel=0.5)


def test_cluster_batch_with_instances_that_do_not_fit(monkeypatch):
    """FP64 256 x 1024 fits no cluster: it steps in the lockstep kernels beside the others' clusters."""
    from vivlasov1d_b200.batch import Batch
    sizes = [(64, 128), (256, 1024), (128, 256), (64, 1000), (256, 128)]
    runs = [_run(monkeypatch, 16, *s)[0] for s in sizes]
    refs = [_run(monkeypatch, 0, *s)[0] for s in sizes]
    batch = Batch(runs)
    for _ in range(2):
        reps = batch.step()
        for r, ref in zip(reps, refs):
            q = ref.step()
            assert r["status"] == 0 and r["picard_its"] == q["picard_its"]
    for a, b in zip(runs, refs):
        assert _rel(a.fc, b.fc) <= 1e-12
    assert batch.launch_count() > 0
    assert batch.time_kernel(0, it=2, reps=2) > 0


@pytest.mark.parametrize("nx,precision", [(64, "fp64"), (256, "fp64"), (50, "fp64"), (64, "mixed")])
def test_cluster_cta_without_rows(monkeypatch, nx, precision):
    """100 rows over 16 CTAs of 7: the last CTA owns none and may add nothing
    to a reduction, whatever its shared memory holds.  A run of 112 rows (same
    layout, every CTA full) whose f is NaN leaves NaN in every CTA's W and V_0."""
    from vivlasov1d_b200 import _lib
    kw = {"rtol": 1e-4} if precision == "mixed" else {}
    dirty, _, _ = _run(monkeypatch, 16, nx, 112, precision=precision, max_iter=2, **kw)
    run, _, _ = _run(monkeypatch, 16, nx, 100, precision=precision, **kw)
    ref, _, _ = _run(monkeypatch, 0, nx, 100, precision=precision, **kw)
    for _ in range(2):
        dirty.fc.fill_(float("nan"))
        with pytest.raises(_lib.VVError):
            dirty.step()
        rep = run.step()
        ref.step()
        assert rep["ksp_failures"] == 0
    # in the mixed mode two runs inside the 1e-11 residual ball differ by 2 ht atol a step
    assert float((run.fc - ref.fc).norm()) <= 2 * 2 * 0.1 * 1e-11 + 1e-12 * float(ref.fc.norm())


@pytest.mark.parametrize("bad", ["diverged", "nan"])
def test_cluster_batch_isolates_a_failing_instance(monkeypatch, bad):
    """A failing instance (f scaled until the residual passes 10, or NaN in f)
    between others of its cluster class and of another: it alone reports it, and
    the others' f equal those of a batch without it, bit for bit."""
    from vivlasov1d_b200 import _lib
    from vivlasov1d_b200.batch import Batch
    sizes = [(64, 128), (64, 200), (64, 100), (128, 256)]
    runs, ref = ([_run(monkeypatch, 16, *s, max_it=100)[0] for s in sizes] for _ in range(2))
    if bad == "nan":
        runs[1].fc[9, 5] = float("nan")
    else:
        runs[1].fc.mul_(1e3)
        runs[1].calculate_moments()
    want = _lib.VV_ERR_NAN if bad == "nan" else _lib.VV_ERR_DIVERGED
    b, bref = Batch(runs), Batch([ref[i] for i in (0, 2, 3)])
    for _ in range(2):
        reps, rref = b.step(), bref.step()
        assert [r["status"] for r in reps] == [_lib.VV_OK, want, _lib.VV_OK, _lib.VV_OK]
        for i, q in zip((0, 2, 3), rref):
            assert reps[i]["gmres_its"] == q["gmres_its"] and torch.equal(runs[i].fc, ref[i].fc)


@pytest.mark.parametrize("ctas", [16, 0])
def test_timing_counts_the_stencil_of_steps_and_solves(monkeypatch, ctas):
    """Timing enabled: one timed launch of the Jacobian stencil per GMRES
    iteration at least, in a step and in a solve, wherever they run without it."""
    import ctypes as C
    from vivlasov1d_b200 import _lib
    run, _, _ = _run(monkeypatch, ctas, 64, 130)
    plain, _, _ = _run(monkeypatch, ctas, 64, 130)
    run.step(), plain.step()
    run.ctx.timing_enable(True)
    its = sum(run.step()["gmres_its"])
    n, ms = run.ctx.timing_read()
    assert its > 0 and n >= its and ms > 0
    b, x = run.fc.clone(), torch.empty_like(run.fc)
    o = _lib.vv_ksp_opts(rtol=1e-9, atol=1e-50, dtol=1e5, max_it=400, restart=0)
    r = _lib.vv_ksp_result()
    run.ctx.call("vv_gmres", run.ctx.field(b), run.ctx.field(x), C.byref(o), C.byref(r))
    n, ms = run.ctx.timing_read()
    assert r.its > 0 and n >= r.its and ms > 0
    run.ctx.timing_enable(False)
    run.step()
    assert run.ctx.timing_read()[0] == 0
    for _ in range(2):
        plain.step()
    assert _rel(run.fc, plain.fc) <= 1e-12
