"""The arrays a scene derives from its mesh on the device against the oracle's serial loops: the
same masses, first step, edge groups (through the free surface), node sources (through the
forces) and damage geometry, bit for bit. Meshes numbered at random, a fan whose hub has more
elements than a block has threads, and elements that have a node at two corners."""
import numpy as np
import pytest

from neofiz_gb300 import Contact, ExplicitSolver, Formulation, Integration, Kinematics, QuadMesh
from neofiz_gb300 import _abi, scenes
from oracle.oracle import OracleSolver

FIELDS = (_abi.FIELD_MASS, _abi.FIELD_SURFACE_EDGES, _abi.FIELD_SURFACE_NODES, _abi.FIELD_FR,
          _abi.FIELD_FZ, _abi.FIELD_VR, _abi.FIELD_STRESS, _abi.FIELD_DAMAGE_STRENGTH)


def fan(blades, rings, seed, collapsed=()):
    """`blades` quads around a hub and `rings` strips of quads around those."""
    g = np.random.RandomState(seed)
    n = 2 * blades
    a = 2.0 * np.pi * np.arange(n) / n
    r, z, quads = [0.02], [0.0], []
    for k in range(rings + 1):
        radius = 1.0e-3 * (k + 1) * g.uniform(0.97, 1.03, n)
        r.extend(0.02 + radius * np.cos(a))
        z.extend(radius * np.sin(a))
    for i in range(blades):
        quads.append([0, 1 + 2 * i, 2 + 2 * i, 1 + (2 * i + 2) % n])
    for k in range(rings):
        for i in range(n):
            p, q = 1 + k * n, 1 + (k + 1) * n
            quads.append([p + i, q + i, q + (i + 1) % n, p + (i + 1) % n])
    for i in collapsed:
        quads[i][3] = quads[i][2]
    label = g.permutation(len(r))
    quads = [list(np.roll(label[q], g.randint(4))) for q in quads]
    quads = [quads[i] for i in g.permutation(len(quads))]
    outer = label[1 + rings * n + np.arange(n)]
    place = np.argsort(label)
    return QuadMesh(np.array(r)[place], np.array(z)[place], quads,
                    np.stack([outer, np.roll(outer, -1)], 1)[::3])


@pytest.mark.gpu
@pytest.mark.parametrize("integration", [Integration.REDUCED, Integration.FULL])
@pytest.mark.parametrize("formulation", [Formulation.AXISYMMETRIC, Formulation.PLANE_STRAIN])
@pytest.mark.parametrize("blades,rings", [(3, 0), (5, 3), (130, 2), (300, 1)])
def test_setup_equals_the_oracle(gpu_lib, blades, rings, formulation, integration):
    mesh = fan(blades, rings, blades)
    g = np.random.RandomState(1)
    gf, eps = g.uniform(1e4, 1e5, mesh.elementCount), g.uniform(1e-4, 1e-2, mesh.elementCount)
    vr = g.uniform(-30.0, 30.0, mesh.nodeCount)
    pair = []
    for cls in (ExplicitSolver, OracleSolver):
        s = cls(mesh, scenes.tube_material(), formulation, integration,
                Kinematics.FINITE_STRAIN, 0.01, 0.5)
        s.setDamage(gf, eps)
        s.setPressureRamp(1.0e7, 1.0e-6)
        s.setContact(Contact(mesh))
        s.setVelocities(vr, -vr)
        first = s.timestep()
        s.run(6)
        pair.append((s, first))
    assert pair[0][1] == pair[1][1]
    for f in FIELDS:
        a, b = (s.readField(f) for s, _ in pair)
        assert a.tobytes() == b.tobytes(), f
    for s, _ in pair:
        s.close()


@pytest.mark.gpu
def test_repeated_corners_and_loose_nodes(gpu_lib):
    mesh = fan(9, 2, 4, collapsed=(0, 4))
    loose = QuadMesh([0.0, 1.0, 2.0], [0.0, 0.0, 1.0], [])
    for m in (mesh, loose):
        masses = []
        for cls in (ExplicitSolver, OracleSolver):
            s = cls(m, scenes.tube_material(), Formulation.AXISYMMETRIC, Integration.REDUCED,
                    Kinematics.FINITE_STRAIN, 1.0, 0.5)
            masses.append((s.readField(_abi.FIELD_MASS).tobytes(), s.timestep()))
            s.close()
        assert masses[0] == masses[1]
