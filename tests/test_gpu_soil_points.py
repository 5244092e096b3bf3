"""The PressureIndependMultiYield point kernels in blocks of 32 elements, the moved-surface commit and the point-parallel
element force, on a B200, against the same load path in numpy: every Gauss point's strain formed on the
host, every update by the host restatement (whole states, swapped at each commit), the element forces
summed there. Element counts around multiples of 32, both correctors, with and without a body force,
through confinement, the switch to the plastic stage, shear, a reversal and a second force evaluation
before a commit. The strains differ by rounding (a few eps), which the updates carry on: 1e-9 of the
largest force bounds it over these six steps; a surface left out of a commit shows at 1e-3."""
import numpy as np
import pytest

import femorax_b200 as fx
from femorax_b200 import meshes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)
DEV = torch.device("cuda:0")
CORNERS = np.array([(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1),
                    (-1, 1, 1)], float)


def gauss(X):
    """Per point gp: dN/dx [E, 8, 3], dvol [E], N [8] of elements with corners X [E, 8, 3]."""
    r = 1 / np.sqrt(3.0)
    for gp in range(8):
        g = np.array([r if gp & s else -r for s in (4, 2, 1)])
        f = 1 + CORNERS * g
        N = f.prod(1) / 8
        dn = np.stack([CORNERS[:, d] * f[:, [c for c in range(3) if c != d]].prod(1) / 8 for d in range(3)], 1)
        J = np.einsum("eai,ad->eid", X, dn)
        yield np.einsum("ad,edi->eai", dn, np.linalg.inv(J)), np.linalg.det(J), N


@pytest.mark.parametrize("material", ["pimy", "pimy_frictional"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 70])
def test_path(material, n):
    if material == "pimy":
        m = fx.PressureIndependMultiYield(2.0, 40500.0, 108000.0, 8.0, 0.1, 0.0, 100.0, 0.0, 20)
    else:
        m = fx.PressureIndependMultiYield(2.0, 60000.0, 150000.0, 5.0, 0.1, 30.0, 80.0, 0.5, 20)
    spec = meshes.distort(meshes.box_model(n, 1, 1, (float(n), 1.0, 1.0), E=1e5, nu=0.3, rho=2.0, lumped=True,
                                           b=(0.0, 0.1, -9.8) if n % 2 else (0.0, 0.0, 0.0)), 0.1, seed=n)
    mesh = fx.Model(spec).compile().mesh()
    E, P, q = mesh.count, mesh.padded, mesh.num_equations
    eq, node = mesh.eq.reshape(24, P)[:, :E], mesh.node.reshape(8, P)[:, :E]
    X = mesh.coords.reshape(3, -1)[:, node].transpose(2, 1, 0)  # E 8 3
    body = np.array(spec.groups[0].b)
    forces = []
    for mode in ("fused", "compacted"):
        f = fx.InternalForce(mesh)
        f.set_pimy(0, m)
        f.set_soil_corrector(mode)
        forces.append(f)
    com, tri = [m.initial_state(E) for _ in range(8)], [np.zeros((m.nstate, E)) for _ in range(8)]
    pos = np.zeros((q, 3))
    dof = np.zeros(q, int)
    for a in range(24):
        ok = eq[a] >= 0
        pos[eq[a][ok]], dof[eq[a][ok]] = X[ok, a // 3], a % 3
    noise = np.random.default_rng(n).standard_normal(q)
    zero = torch.zeros(q, dtype=torch.float64, device=DEV)
    moved = 0
    for step, (stage, gamma, commit) in enumerate(((0, 0.0, 1), (1, 1e-4, 1), (1, 8e-4, 1), (1, 1.4e-3, 0),
                                                   (1, 2e-4, 1), (1, -6e-4, 1), (1, 5e-4, 1))):
        if step == 1:
            for f in forces:
                f.set_material_stage(0, 1)
        u = np.where(dof == 2, -4e-4 * pos[:, 2], 0.0) + np.where(dof == 0, gamma * pos[:, 2], 0.0) + 2e-6 * noise
        ue = np.where(eq >= 0, u[np.maximum(eq, 0)], 0.0).T.reshape(E, 8, 3)
        fe = np.zeros((E, 8, 3))
        for gp, (dN, vol, N) in enumerate(gauss(X)):
            G = np.einsum("eai,eaj->eij", ue, dN)
            eps = np.stack([G[:, 0, 0], G[:, 1, 1], G[:, 2, 2], G[:, 0, 1] + G[:, 1, 0], G[:, 1, 2] + G[:, 2, 1],
                            G[:, 2, 0] + G[:, 0, 2]])
            sig = np.zeros((6, E))
            assert m.update_host(stage, com[gp], tri[gp], np.ascontiguousarray(eps), sig) == 0
            S = np.array([[sig[0], sig[3], sig[5]], [sig[3], sig[1], sig[4]], [sig[5], sig[4], sig[2]]])
            fe += np.einsum("ije,eaj,e->eai", S, dN, vol) - N[None, :, None] * body * vol[:, None, None]
        want = np.zeros(q)
        flat = fe.reshape(E, 24).T
        np.add.at(want, eq[eq >= 0], flat[eq >= 0])
        got = []
        for f in forces:
            out = torch.zeros(q, dtype=torch.float64, device=DEV)
            f.compute(torch.as_tensor(u, device=DEV), zero, out)
            got.append(out.cpu().numpy())
            if commit:
                f.commit_state()
        assert np.array_equal(got[0], got[1]), step
        assert np.max(np.abs(got[0] - want)) <= 1e-9 * np.max(np.abs(want)), step
        moved = max(moved, forces[0].plastic_points())
        if commit:
            com, tri = tri, com
    assert moved > 0
