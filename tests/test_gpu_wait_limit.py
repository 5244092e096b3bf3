"""The bounded waits of the fused CG iteration (cg_fused.cuh) run out, on a B200: with a limit of 0 polls
every block gives up at its first meeting, nothing waits and nothing faults, the call returns
FX_E_TIMEOUT, and the next solve on the same handle has the bits of a handle that never ran out."""
import numpy as np
import pytest

import femorax_b200 as fx
from femorax_b200 import _lib as L
from femorax_b200 import meshes, serving
from tests.j2_newton_ref import top_shear_load
from tests.models_for_tests import j2_column

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)
DEV = torch.device("cuda:0")
DEFAULT = 1 << 22


@pytest.mark.parametrize("solver", [fx.ConjugateGradient, fx.KrylovSolver, fx.MixedPrecisionSolver])
def test_solver(solver):
    force = fx.InternalForce(fx.Model(meshes.layered_box(12, 11, 10, layers=2, seed=1)[0]).compile().mesh())
    n = force.num_equations
    assert n > 2 * 2048
    b = torch.as_tensor(np.random.default_rng(1).standard_normal(n), device=DEV)
    out = []
    for limits in ((), (0, DEFAULT), (0, 0, DEFAULT)):
        s = solver(fx.SolveOptions(relative_tolerance=1e-9))
        s.setup(fx.MatrixFreeOperator(force))
        for polls in limits:
            L.check(L.lib().fx_solver_set_wait_limit(s._h, polls))
            if polls:
                continue
            x = torch.ones(n, dtype=torch.float64, device=DEV)
            with pytest.raises(fx.FxError) as e:
                s.solve(b, x)
            assert e.value.code == L.FX_E_TIMEOUT
            assert (x == 1.0).all()
        x = torch.zeros(n, dtype=torch.float64, device=DEV)
        assert s.solve(b, x).converged
        out.append(x.cpu().numpy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("mixed", [False, True])
def test_batched_newton(mixed):
    meshes_, loads = [], []
    for size in ((5, 5, 24), (1, 1, 4), (6, 5, 20)):
        spec = j2_column(nx=size[0], ny=size[1], nz=size[2])
        comp = fx.Model(spec).compile()
        meshes_.append(comp.mesh())
        loads.append(top_shear_load(spec, serving.equation_map(comp), 8e3)[0])
    assert meshes_[0].num_equations > 2048
    out = []
    for limits in ((), (0, DEFAULT)):
        b = fx.BatchedNewton(meshes_, mixed=mixed)
        f = torch.as_tensor(b.combine(loads), device=DEV)
        u = torch.zeros_like(f)
        for polls in limits:
            L.check(L.lib().fx_nbatch_set_wait_limit(b._h, polls))
            if polls:
                continue
            with pytest.raises(fx.FxError) as e:
                b.step(f, u)
            assert e.value.code == L.FX_E_TIMEOUT
            assert not u.any()
        b.step(f, u)
        out.append(u.cpu().numpy())
    assert out[0].any() and np.array_equal(out[0], out[1])


@pytest.mark.parametrize("inner", ["fp32", "fp64"])
def test_engine_finishes_the_failed_slots_alone(inner):
    """The slots of more than one chunk run out and finish with that status; the one-chunk slot, which
    meets nobody, goes on to its solution; the freed slots then serve the same requests."""
    prepared = [serving.prepare(serving.Request(i, *size)) for i, size in
                enumerate(((14, 12, 7), (3, 4, 5), (10, 10, 12)))]

    def engine():
        return fx.BatchEngine(1 << 20, 8, options=fx.SolveOptions(relative_tolerance=1e-8), inner=inner)

    def run(e, slots):
        out = {}
        for _ in range(400):
            e.round()
            for s in [s for s in slots if e.finished(s)]:
                out[slots.pop(s)] = e.retire(s)
            if not slots:
                return out
        raise AssertionError("the engine did not finish")

    e = engine()
    want = run(e, {e.admit(f, b): i for i, (f, b, _) in enumerate(prepared)})
    e = engine()
    L.check(L.lib().fx_engine_set_wait_limit(e._h, 0))
    got = run(e, {e.admit(f, b): i for i, (f, b, _) in enumerate(prepared)})
    assert [got[i][1].status for i in range(3)] == [L.FX_E_TIMEOUT, L.FX_OK, L.FX_E_TIMEOUT]
    assert not got[0][1].converged and got[1][1].converged
    assert np.array_equal(got[1][0], want[1][0])
    L.check(L.lib().fx_engine_set_wait_limit(e._h, DEFAULT))
    again = run(e, {e.admit(f, b): i for i, (f, b, _) in enumerate(prepared)})
    for i in range(3):
        assert again[i][1].converged and np.array_equal(again[i][0], want[i][0]), i


def test_server_reports_the_failed_request():
    """Both loops serve the other requests and give the failed one's status."""
    stream = [serving.Request(0, 14, 12, 7), serving.Request(1, 3, 4, 5)]
    for loop in (serving.Server, serving.NativeServer):
        e = fx.BatchEngine(1 << 20, 8, options=fx.SolveOptions(relative_tolerance=1e-8))
        L.check(L.lib().fx_engine_set_wait_limit(e._h, 0))
        served, _ = loop(e, hbm_budget=1 << 34).run(stream, realtime=False)
        by_id = {s.id: s.result for s in served}
        assert by_id[0].status == L.FX_E_TIMEOUT and not by_id[0].converged, loop
        assert by_id[1].converged, loop
