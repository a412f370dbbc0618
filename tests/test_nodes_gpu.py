"""The node kernels on either side of the size where their products move to the integer units
(more than one warp of nodes per quarter SM: 608 whole warps of 152 SMs): the same bits as the
oracle's FP64 products, with and without the terms that are left out when they are zero."""
import numpy as np
import pytest

from neofiz_gb300 import ExplicitSolver, _abi, scenes
from neofiz_gb300.batch import BatchSolver
from neofiz_gb300.materials import Formulation
from oracle.oracle import OracleSolver

FIELDS = (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_VR, _abi.FIELD_VZ, _abi.FIELD_FR,
          _abi.FIELD_FZ, _abi.FIELD_STRESS, _abi.FIELD_WALL_STATE)


def bits(a):
    return a.view(np.uint64) if a.dtype == np.float64 else a


@pytest.mark.gpu
@pytest.mark.parametrize("gravity,damping", [((0.0, 0.0), 0.0), ((0.0, -9.81), 0.0),
                                             ((-3.0, 2.0e5), 0.2)])
@pytest.mark.parametrize("nz", [589, 590])                # 33 x 590 and 33 x 591 nodes
def test_node_products_equal_the_oracle(gpu_lib, nz, gravity, damping):
    pair = []
    for cls in (ExplicitSolver, OracleSolver):
        s, _, _ = scenes.taylor_rod(cls, nr=32, nz=nz, length=70.0e-3)
        s.setGravity(*gravity)
        if damping:
            s.setRelaxationDamping(damping, 2.0e5)
        s.run(30)
        pair.append(s)
    for f in FIELDS:
        assert np.array_equal(bits(pair[0].readField(f)), bits(pair[1].readField(f))), f
    assert pair[0].time() == pair[1].time()
    for s in pair:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [589, 590])
def test_mixed_node_products_equal_a_lone_instance(gpu_lib, nz):
    """One batch instance never has more than a warp per quarter SM of its own cluster's SMs."""
    rod = scenes.taylor_sweep(1, seed=5, t_end=1.0)[0]
    rod.update(nr=32, nz=nz)
    b = BatchSolver(scenes.sweep_instances([rod], length=70.0e-3), Formulation.AXISYMMETRIC,
                    cfl=0.6, precision=_abi.PRECISION_MIXED)
    s, _, _ = scenes.sweep_rod(ExplicitSolver, rod, length=70.0e-3)
    s.setPrecision(_abi.PRECISION_MIXED)
    b.run(30)
    s.run(30)
    for f in FIELDS[:-1]:
        assert np.array_equal(bits(b.readInstance(f, 0)), bits(s.readField(f))), f
    b.close()
    s.close()
