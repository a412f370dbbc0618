"""The burst measurement where clusters of blocks step an instance: tubes of more elements than
half a block has threads (two blocks each: 200 elements; four and eight: 600 and 1,100)."""
import numpy as np
import pytest

from neofiz_gb300 import QuadMesh, _abi, scenes
from neofiz_gb300.batch import BatchSolver
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu


def tube(slenderness, through_wall, along):
    """The burst case's tube, `along` elements high instead of a slice of two."""
    i = scenes.burst_instance(slenderness=slenderness, through_wall=through_wall)
    inner, outer = i.mesh.r.min(), i.mesh.r.max()
    i.mesh = QuadMesh.cylinderWall(inner, outer, (outer - inner) / through_wall * along,
                                   through_wall, along)
    i.fixed_axial = np.arange(i.mesh.nodeCount)
    return i


def measured(cls, tubes, precision, steps, config=None):
    b = cls(tubes, scenes.Formulation.AXISYMMETRIC, cfl=scenes.BURST_CFL, precision=precision)
    if config:
        b.setConfig(*config)
    b.setBurst(scenes.BURST_SAMPLE_STEPS, 25.0e-3, scenes.BURST_PEAK_MARGIN, traceCapacity=200)
    for n in steps:
        b.run(n)
    out = b.burstResults(), b.burstTrace(), b.state(), b.read(_abi.FIELD_UR)
    b.close()
    return out


def assert_equal(a, b):
    for k in a[0]:
        assert np.array_equal(a[0][k], b[0][k]), k
    assert np.array_equal(a[1], b[1])
    for k in ("steps", "time", "done"):
        assert np.array_equal(a[2][k], b[2][k]), k
    assert np.array_equal(a[3], b[3])


def test_fp64_tubes_burst_as_the_oracle_does(gpu_lib):
    tubes = [tube(8.0, 1, 200), tube(6.0, 2, 75), tube(10.0, 1, 133)]
    steps = (700, 1 << 40)
    g = measured(BatchSolver, tubes, _abi.PRECISION_FP64, steps)
    assert g[0]["traversed"].all()
    assert_equal(g, measured(OracleBatch, tubes, _abi.PRECISION_FP64, steps))


@pytest.mark.parametrize("sizes", [((4, 150), (4, 50), (1, 133)), ((10, 110), (4, 150))])
def test_fp64_larger_tubes_are_sampled_as_the_oracle_does(gpu_lib, sizes):
    tubes = [tube(20.0, nr, nz) for nr, nz in sizes]
    steps = (1100, 900)
    assert_equal(measured(BatchSolver, tubes, _abi.PRECISION_FP64, steps),
                 measured(OracleBatch, tubes, _abi.PRECISION_FP64, steps))


@pytest.mark.parametrize("precision", [_abi.PRECISION_MIXED, _abi.PRECISION_COMPENSATED])
def test_fp32_tubes_burst_as_in_one_block(gpu_lib, precision):
    """Against blocks of 128 threads, which have no teams and round alike."""
    tubes = [tube(8.0, 1, 200), tube(6.0, 4, 150), tube(6.0, 10, 110)]
    steps = (700, 6000)
    one = measured(BatchSolver, tubes, precision, steps, (128, 0, 1, 256))
    assert one[0]["samples"].min() > 10
    assert_equal(measured(BatchSolver, tubes, precision, steps), one)
