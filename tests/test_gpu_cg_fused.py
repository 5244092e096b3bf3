"""The CG iteration in one cooperative launch (cg_fused.cuh) at the edges of its chunks, on a B200: a
few iterations of ConjugateGradient on distorted bricks (the exact operator) against the same
recurrence in numpy on the oracle's operator, for vectors of less than one chunk of 2048, just over
one, odd lengths and many chunks, lane counts 1, 7 and 32, and a solution vector off the pairs'
16-byte alignment. The two differ by rounding: each of the k iterations forms its products and sums
with relative errors of a few n eps, so 1e-11 of the largest entry bounds them, and a chunk or an
entry left out shows at 1e-4 and above. The same at the largest vector that the fused form takes and
just past it. In FP32, and in every form, a solve has the same bits alone and in a batch
(test_gpu_batch.py, test_gpu_nbatch.py)."""
import numpy as np
import pytest

import femorax_b200 as fx
from femorax_b200 import meshes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)
DEV = torch.device("cuda:0")


def reference(port, b, diag, k):
    x, r = np.zeros_like(b), b.copy()
    z = r / diag
    p, rz = z.copy(), r @ z
    for _ in range(k):
        q = port.apply_operator((1.0, 0.0, 0.0), p)
        alpha = rz / (p @ q)
        x, r = x + alpha * p, r - alpha * q
        z = r / diag
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x


@pytest.mark.parametrize("size", [(1, 1, 1), (7, 9, 8), (8, 9, 8), (12, 11, 13), (23, 22, 21)])
def test_iterates(size, oracle_mod):
    spec = meshes.distort(meshes.box_model(*size), 0.15, seed=sum(size))
    spec.fix_node, spec.fix_dof = spec.fix_node[1:], spec.fix_dof[1:]  # odd numbers of equations
    mesh = fx.Model(spec).compile().mesh()
    n = mesh.num_equations
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    b = np.random.default_rng(1).standard_normal(n)
    d = torch.zeros(n, dtype=torch.float64, device=DEV)
    force.operator_diagonal(fx.OperatorCoefficients(), d)
    for lanes in (1, 7, 32):
        for k in (1, 4):
            want = reference(port, b, d.cpu().numpy(), k)
            s = fx.ConjugateGradient(fx.SolveOptions(relative_tolerance=1e-30, max_iterations=k, lanes=lanes))
            s.setup(fx.MatrixFreeOperator(force))
            got = []
            for off in (0, 1):  # the solution vector aligned to pairs, and not
                x = torch.zeros(n + off, dtype=torch.float64, device=DEV)[off:]
                r = s.solve(torch.as_tensor(b, device=DEV), x)
                assert r.iterations == k and not r.converged
                got.append(x.cpu().numpy())
            assert np.max(np.abs(got[0] - want)) <= 1e-11 * np.max(np.abs(want)), (lanes, k)
            assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("size", [(57, 57, 60), (57, 57, 62)], ids=["largest_fused", "past_it"])
def test_iterates_at_the_limit(size, oracle_mod):
    mesh = fx.Model(meshes.box_model(*size)).compile().mesh()
    n = mesh.num_equations
    chunks = -(-n // 2048)
    assert chunks == {60: 296, 62: 306}[size[2]]  # 2 blocks on each of 148 SMs: 296 fit
    force, port = fx.InternalForce(mesh), oracle_mod.PortMesh(mesh)
    b = np.random.default_rng(1).standard_normal(n)
    d = torch.zeros(n, dtype=torch.float64, device=DEV)
    force.operator_diagonal(fx.OperatorCoefficients(), d)
    want = reference(port, b, d.cpu().numpy(), 3)
    s = fx.ConjugateGradient(fx.SolveOptions(relative_tolerance=1e-30, max_iterations=3))
    s.setup(fx.MatrixFreeOperator(force))
    x = torch.zeros(n, dtype=torch.float64, device=DEV)
    assert s.solve(torch.as_tensor(b, device=DEV), x).iterations == 3
    assert np.max(np.abs(x.cpu().numpy() - want)) <= 1e-11 * np.max(np.abs(want))


def test_infinite_alpha():
    """r.z overflows while p.Ap and ||b|| do not: alpha is infinite, and the residual's norm after the
    step is infinite, as the sums over the vector's own entries give it for any lane count; the chunk's
    zeros past its end (inf times 0) take no part."""
    spec = meshes.box_model(7, 9, 8, E=1e-8)
    force = fx.InternalForce(fx.Model(spec).compile().mesh())
    n = force.num_equations
    assert n % 2048
    op = fx.MatrixFreeOperator(force)
    d, kz = (torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(2))
    op.diagonal(d)
    z = torch.as_tensor(1.0 + 0.3 * np.random.default_rng(5).random(n), device=DEV)
    z *= 1.7e154 / float(z @ (d * z)) ** 0.5  # z.Dz = 2.9e308, past the largest double
    b = d * z
    op.apply(z, kz)
    assert torch.isinf(b @ z) and torch.isfinite(z @ kz) and torch.isfinite(b @ b) and bool((kz != 0).all())
    for lanes in (32, 7):
        s = fx.ConjugateGradient(fx.SolveOptions(relative_tolerance=1e-10, max_iterations=1, lanes=lanes))
        s.setup(op)
        r = s.solve(b, torch.zeros_like(b))
        assert r.iterations == 1 and not r.converged and not r.indefinite
        assert r.final_residual == np.inf, (lanes, r.final_residual)


def test_created_beside_a_busy_default_stream():
    """A solver's counters start at zero for its own stream's solves also while the default stream, on
    which they are zeroed, still works through other kernels (and the memory held another solver's
    counts): creation waits for the zeros. The same solve as with the default stream idle."""
    def problem(size):
        spec = meshes.distort(meshes.box_model(*size), 0.15, seed=sum(size))
        return fx.InternalForce(fx.Model(spec).compile().mesh())

    def solve(force, stream):
        n = force.num_equations
        with torch.cuda.stream(stream):
            b = torch.as_tensor(np.random.default_rng(2).standard_normal(n), device=DEV)
            x = torch.zeros(n, dtype=torch.float64, device=DEV)
        stream.synchronize()
        for _ in range(100):  # (some 50 ms)
            torch.mm(m, m, out=out)
        s = fx.ConjugateGradient(fx.SolveOptions(relative_tolerance=1e-30, max_iterations=6))
        s.setup(fx.MatrixFreeOperator(force), stream=stream)
        r = s.solve(b, x, stream=stream)
        stream.synchronize()
        torch.cuda.synchronize()
        return r, x.cpu().numpy()

    small, large = problem((8, 9, 8)), problem((12, 11, 13))
    m = torch.randn(2048, 2048, dtype=torch.float64, device=DEV)
    out = torch.empty_like(m)
    side = torch.cuda.Stream()
    idle_r, idle = solve(small, torch.cuda.default_stream())
    solve(large, torch.cuda.default_stream())  # (its counters' memory is free again)
    for _ in range(3):
        r, x = solve(small, side)
        assert r.iterations == idle_r.iterations == 6
        assert np.array_equal(x, idle)
