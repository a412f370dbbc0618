"""Scenes on both sides of the size up to which one block sets them up (1,024 nodes), and the
smallest ones, against the oracle's serial loops."""
import numpy as np
import pytest

from neofiz_gb300 import Contact, ExplicitSolver, Formulation, Integration, Kinematics, QuadMesh
from neofiz_gb300 import _abi, scenes
from oracle.oracle import OracleSolver

FIELDS = (_abi.FIELD_MASS, _abi.FIELD_SURFACE_EDGES, _abi.FIELD_SURFACE_NODES, _abi.FIELD_FR,
          _abi.FIELD_FZ, _abi.FIELD_VR, _abi.FIELD_STRESS, _abi.FIELD_DAMAGE_STRENGTH)


@pytest.mark.gpu
@pytest.mark.parametrize("formulation", [Formulation.AXISYMMETRIC, Formulation.PLANE_STRAIN])
@pytest.mark.parametrize("nr,nz", [(1, 1), (1, 2), (1, 511), (31, 31), (4, 204), (2, 341)])
def test_setup_equals_the_oracle(gpu_lib, nr, nz, formulation):
    mesh = QuadMesh.cylinderWall(0.02, 0.02 + 1.0e-3 * nr, 1.0e-3 * nz, nr, nz)
    g = np.random.RandomState(nr + nz)
    vr = g.uniform(-30.0, 30.0, mesh.nodeCount)
    pair = []
    for cls in (ExplicitSolver, OracleSolver):
        s = cls(mesh, scenes.tube_material(), formulation, Integration.REDUCED,
                Kinematics.FINITE_STRAIN, 0.01, 0.5)
        s.setDamage(np.full(mesh.elementCount, 1.0e4), np.full(mesh.elementCount, 1.0e-3))
        s.setPressureRamp(1.0e7, 1.0e-6)
        s.setContact(Contact(mesh))
        s.setVelocities(vr, -vr)
        first = s.timestep()
        s.run(12)
        pair.append((s, first))
    (a, first_a), (b, first_b) = pair
    assert first_a == first_b and a.time() == b.time()
    for f in FIELDS:
        assert np.array_equal(a.readField(f), b.readField(f)), f
    a.close()
    b.close()
