"""Node products on the FP64 pipe against those on the integer units, in the mixed form: a batch
instance stepped by one block of 128 threads on its SM has one warp per quarter SM, which takes
the FP64 pipe; the scene of the same rod has enough nodes for the integer units."""
import numpy as np
import pytest

from neofiz_gb300 import ExplicitSolver, _abi, scenes
from neofiz_gb300.batch import BatchSolver
from neofiz_gb300.materials import Formulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [590, 601])                # 33 x 591 and 33 x 602 nodes
def test_mixed_products_of_both_kinds_agree(gpu_lib, nz):
    rod = scenes.taylor_sweep(1, seed=5, t_end=1.0)[0]
    rod.update(nr=32, nz=nz)
    b = BatchSolver(scenes.sweep_instances([rod], length=70.0e-3), Formulation.AXISYMMETRIC,
                    cfl=0.6, precision=_abi.PRECISION_MIXED)
    b.setConfig(128, 0, 1, 16)
    s, _, _ = scenes.sweep_rod(ExplicitSolver, rod, length=70.0e-3)
    s.setPrecision(_abi.PRECISION_MIXED)
    b.run(30)
    s.run(30)
    for f in (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_VR, _abi.FIELD_VZ, _abi.FIELD_FR,
              _abi.FIELD_FZ, _abi.FIELD_STRESS):
        assert np.array_equal(b.readInstance(f, 0).view(np.uint64),
                              s.readField(f).view(np.uint64)), f
    b.close()
    s.close()
