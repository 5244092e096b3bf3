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
            x = torch.zeros(n, dtype=torch.float64, device=DEV)
            with pytest.raises(fx.FxError) as e:
                s.solve(b, x)
            assert e.value.code == L.FX_E_TIMEOUT
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
