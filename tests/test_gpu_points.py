"""The point-parallel Gauss-point operator (k_points_apply: 32 elements per block) at the edges of its
blocks, on a B200, bit for bit the oracle's: element counts around multiples of 32, with and without
the mass term, elastic and J2 sets (plastic, elastic and initial tangents), and vectors with infinite
and NaN entries (the zeros left out of the stress sums must not change what those give). Tied DOFs
with more and fewer slots than the heavy gather's batches of 256."""
import numpy as np
import pytest

import femorax_b200 as fx
from femorax_b200 import meshes
from tests.models_for_tests import j2_column, soil_column

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)
DEV = torch.device("cuda:0")


def apply(force, n, k, x):
    y = torch.zeros(n, dtype=torch.float64, device=DEV)
    force.apply_operator(k, torch.as_tensor(x, device=DEV), y)
    return y.cpu().numpy()


@pytest.mark.parametrize("lumped", [False, True], ids=["consistent", "lumped"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 97])
def test_element_counts(n, lumped, oracle_mod):
    spec = meshes.distort(meshes.box_model(n, 1, 1, (float(n), 1.0, 1.2), rho=3.0, lumped=lumped), 0.2, seed=n)
    spec.rayleigh = [meshes.Rayleigh(0.3, 1e-3, 2e-3, 5e-4, spec.groups[0].etags[: max(1, n // 2)])]
    mesh = fx.Model(spec).compile().mesh()
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    rng = np.random.default_rng(n)
    for k in ((1.0, 0.0, 0.0), (1.0, 0.4, 0.0), (0.7, 0.0, 3.0), (1.0, 0.2, 5.0)):
        x = rng.standard_normal(mesh.num_equations)
        assert np.array_equal(apply(force, mesh.num_equations, fx.OperatorCoefficients(*k), x), port.apply_operator(k, x)), k


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_entries(bad, oracle_mod):
    spec = meshes.distort(meshes.box_model(5, 4, 3), 0.2, seed=2)
    mesh = fx.Model(spec).compile().mesh()
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    x = np.random.default_rng(3).standard_normal(mesh.num_equations)
    x[mesh.num_equations // 2] = bad
    for k in ((1.0, 0.0, 0.0), (1.0, 0.0, 2.0)):
        got, want = apply(force, mesh.num_equations, fx.OperatorCoefficients(*k), x), port.apply_operator(k, x)
        assert np.array_equal(got, want, equal_nan=True) and not np.all(np.isfinite(want))


@pytest.mark.parametrize("size", [(1, 1, 2), (4, 4, 2), (3, 5, 6)])
def test_j2_sets(size, oracle_mod):
    mesh = fx.Model(j2_column(*size)).compile().mesh()
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    n = mesh.num_equations
    rng = np.random.default_rng(4)
    for amplitude, plastic in ((1e-7, False), (2e-3, True)):
        u = amplitude * rng.standard_normal(n)
        f = torch.zeros(n, dtype=torch.float64, device=DEV)
        force.compute(torch.as_tensor(u, device=DEV), torch.zeros_like(f), f)
        _, _, D, npl = port.force_j2(port.j2_state(), u, np.zeros(n))
        assert (npl > 0) == plastic
        for k in ((1.0, 0.0, 0.0), (1.0, 0.3, 2.0)):
            for initial in (False, True):
                x = rng.standard_normal(n)
                got = apply(force, n, fx.OperatorCoefficients(*k, initial=initial), x)
                assert np.array_equal(got, port.apply_j2(D, k, x, initial=initial)), (amplitude, k, initial)


@pytest.mark.parametrize("lumped", [False, True], ids=["consistent", "lumped"])
@pytest.mark.parametrize("n", [30, 31, 36, 38])  # point-parallel, a thread per element, and both again
def test_operator_on_both_sides_of_the_rule(n, lumped, oracle_mod):
    """K x, and with the mass term: its consistent form is point-parallel at every size."""
    mesh = fx.Model(meshes.distort(meshes.box_model(n, n, n, lumped=lumped), 0.1, seed=n)).compile().mesh()
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    for k in ((1.0, 0.0, 0.0), (1.0, 0.0, 3.0)):
        x = np.random.default_rng(n).standard_normal(mesh.num_equations)
        got = apply(force, mesh.num_equations, fx.OperatorCoefficients(*k), x)
        assert np.array_equal(got, port.apply_operator(k, x)), k


@pytest.mark.parametrize("size", [(37, 37, 73), (37, 37, 74)])  # below and above 100,000 elements
def test_j2_stiffness_on_both_sides_of_the_rule(size, oracle_mod):
    mesh = fx.Model(j2_column(*size)).compile().mesh()
    assert abs(mesh.count - 100000) < 1500
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    n = mesh.num_equations
    rng = np.random.default_rng(6)
    u = 2e-3 * rng.standard_normal(n)
    f = torch.zeros(n, dtype=torch.float64, device=DEV)
    force.compute(torch.as_tensor(u, device=DEV), torch.zeros_like(f), f)
    _, _, D, npl = port.force_j2(port.j2_state(), u, np.zeros(n))
    assert npl > 0
    x = rng.standard_normal(n)
    assert np.array_equal(apply(force, n, fx.OperatorCoefficients(), x), port.apply_j2(D, (1.0, 0.0, 0.0), x))


@pytest.mark.parametrize("size", [(16, 15, 2), (17, 16, 2), (33, 32, 2)])  # tied rows below and above 256 slots
def test_tied_dofs(size, oracle_mod):
    mesh = fx.Model(soil_column(*size)).compile().mesh()
    x = np.random.default_rng(5).standard_normal(mesh.num_equations)
    got = apply(fx.InternalForce(mesh), mesh.num_equations, fx.OperatorCoefficients(1.0, 0.2, 3.0), x)
    assert np.array_equal(got, oracle_mod.PortMesh(mesh).apply_operator((1.0, 0.2, 3.0), x))
