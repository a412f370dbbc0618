"""Fields read through the host (up to 4,096 values) and through the device (more): pairs split
into components, float state widened, in a scene and in a batch."""
import numpy as np
import pytest

from neofiz_gb300 import ExplicitSolver, _abi, scenes
from neofiz_gb300.batch import BatchSolver
from neofiz_gb300.materials import Formulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz", [(3, 6), (63, 63), (16, 240)])     # 28, 4,096 and 4,097 nodes
def test_components_come_back_as_written(gpu_lib, nr, nz):
    s, mesh, _ = scenes.taylor_rod(ExplicitSolver, nr=nr, nz=nz)
    g = np.random.RandomState(3)
    vr, vz = g.uniform(-1.0, 1.0, (2, mesh.nodeCount))
    vr[np.isclose(mesh.r, 0.0)] = 0.0                                # held on the axis
    s.setVelocities(vr, vz)
    assert np.array_equal(s.readField(_abi.FIELD_VR), vr)
    assert np.array_equal(s.readField(_abi.FIELD_VZ), vz)
    s.close()


@pytest.mark.parametrize("nr,nz", [(3, 6), (64, 64), (17, 241)])     # 18, 4,096 and 4,097 elements
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
def test_batch_fields_are_the_scenes(gpu_lib, precision, nr, nz):
    rod = scenes.taylor_sweep(1, seed=2, t_end=1.0)[0]
    rod.update(nr=nr, nz=nz)
    b = BatchSolver(scenes.sweep_instances([rod]), Formulation.AXISYMMETRIC, cfl=0.6,
                    precision=precision)
    s, _, _ = scenes.sweep_rod(ExplicitSolver, rod)
    s.setPrecision(precision)
    b.run(12)
    s.run(12)
    for f in (_abi.FIELD_HOURGLASS_R, _abi.FIELD_HOURGLASS_Z, _abi.FIELD_HOURGLASS_STIFFNESS,
              _abi.FIELD_STRESS, _abi.FIELD_VZ, _abi.FIELD_WALL_STATE):
        assert np.array_equal(b.read(f), s.readField(f)), f
    b.close()
    s.close()
