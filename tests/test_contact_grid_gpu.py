"""The contact search on a grid with more cells than direct-indexed buckets (bodies far apart):
the same bits as the oracle's serial search, with every bucket in its slots and with buckets that
outgrow them."""
import numpy as np
import pytest

from neofiz_gb300 import (Contact, ExplicitSolver, Formulation, Integration, Kinematics, Outline,
                          _abi, scenes)
from oracle.oracle import OracleSolver

FIELDS = (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_FR, _abi.FIELD_FZ, _abi.FIELD_VZ,
          _abi.FIELD_CONTACT_MASTER, _abi.FIELD_CONTACT_STATE, _abi.FIELD_STRESS)
CELL = 1.0e-3


def build(cls, far):
    block = (Outline.rectangle(0.0, 0.0, 100 * CELL, 50 * CELL),
             Outline.rectangle(0.0, 50 * CELL, 100 * CELL, 100 * CELL),
             Outline.rectangle(7 * CELL, far * CELL, 12 * CELL, (far + 5) * CELL))
    mesh = Outline.assemble(CELL, *block)
    s = cls(mesh, scenes.tube_material(), Formulation.PLANE_STRAIN, Integration.REDUCED,
            Kinematics.FINITE_STRAIN, 0.02, 0.5)
    s.setContact(Contact(mesh).withFriction(0.3))
    down = np.where((mesh.z > 50 * CELL) & (mesh.z < 101 * CELL), -120.0, 0.0)
    s.setVelocities(np.where(down < 0.0, 15.0, 0.0), down)
    return s, mesh


@pytest.mark.gpu
@pytest.mark.parametrize("slots", [64, 3, 0])
@pytest.mark.parametrize("far", [357, 359, 361, 400])
def test_shared_buckets_equal_the_oracle(gpu_lib, far, slots):
    (g, mesh), (o, _) = build(ExplicitSolver, far), build(OracleSolver, far)
    cells = (int(100 / 1.5) + 1) * (int((far + 5) / 1.5) + 1)
    assert 16100 < cells <= 2 * mesh.nodeCount             # about and above 16,384 buckets
    for s in (g, o):
        s.setGridSlots(slots)
        s.run(25)
    for f in FIELDS:
        assert g.readField(f).tobytes() == o.readField(f).tobytes(), f
    cg, co = g._contactInfo(), o._contactInfo()
    assert (cg.pair_count, cg.segment_count) == (co.pair_count, co.segment_count)
    assert cg.pair_count > 0
    assert cg.energy == pytest.approx(co.energy, rel=1e-12)
    assert cg.dissipation == pytest.approx(co.dissipation, rel=1e-12)
    g.close()
    o.close()
