"""Device memory that a scene or a batch holds: its own arrays, and nothing of its set-up."""
import numpy as np
import pytest

from neofiz_gb300 import Contact, ExplicitSolver, Formulation, Integration, Kinematics, QuadMesh
from neofiz_gb300 import _abi
from neofiz_gb300.batch import BatchSolver, Instance
from neofiz_gb300.materials import Material

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def elastic():
    return Material("elastic", 200.0e9, 0.29, 7850.0)


def scene(mesh):
    return ExplicitSolver(mesh, elastic(), Formulation.AXISYMMETRIC, Integration.REDUCED,
                          Kinematics.FINITE_STRAIN, 1.0, 0.6)


def test_a_scene_holds_no_set_up_lists(gpu_lib):
    """87 bytes a node (positions, displacement, velocity, force 64, masses 16, three bytes of
    state, 4 of sources) and 12 of staging; 252 an element (12 ints of connectivity, material and
    sources, 12 of edge groups, 19 doubles of state and force terms); and up to 3 MB of partial
    sums and rounding."""
    scene(QuadMesh.solidCylinder(0.01, 0.1, 4, 8)).close()
    mesh = QuadMesh.solidCylinder(0.01, 0.1, 800, 1249)
    before = free()
    s = scene(mesh)
    held = before - free()
    s.close()
    assert held < 99 * mesh.nodeCount + 252 * mesh.elementCount + 3 * MB


def test_a_batch_holds_no_set_up_lists(gpu_lib):
    """The same without edge groups, with 8 bytes a node of staging."""
    def batch(nr, nz, count):
        m = QuadMesh.solidCylinder(0.01, 0.1, nr, nz)
        return BatchSolver([Instance(mesh=m, material=elastic(), t_end=1.0)] * count,
                           Formulation.AXISYMMETRIC, cfl=0.6, precision=_abi.PRECISION_FP64), m
    batch(4, 8, 2)[0].close()
    before = free()
    b, m = batch(100, 199, 50)
    held = before - free()
    b.close()
    # some twenty allocations of their own, each rounded up to 2 MB at most
    assert held < 50 * (94 * m.nodeCount + 204 * m.elementCount) + 20 * 2 * MB // 2


def test_contact_holds_no_cells_beside_its_slots(gpu_lib):
    """65,536 buckets of 64 slots of 72 bytes; 901 bytes an element and 400 a node."""
    def contact(nr, nz):
        m = QuadMesh.solidCylinder(0.01, 0.1, nr, nz)
        s = scene(m)
        before = free()
        s.setContact(Contact(m))
        s.synchronize()
        held = before - free()
        s.close()
        return held, m
    contact(4, 8)
    held, m = contact(100, 399)
    assert held < 65536 * 64 * 72 + 901 * m.elementCount + 400 * m.nodeCount + 4 * MB
