"""Batches with fewer instances than SMs, whose instances are stepped by clusters of blocks: every
instance equals its single scene bit for bit, at the sizes where the number of blocks per
instance changes (four warps of elements a block) and for odd counts and meshes."""
import numpy as np
import pytest

from neofiz_gb300 import ExplicitSolver, _abi, scenes
from neofiz_gb300.batch import BatchSolver
from neofiz_gb300.materials import Formulation

FIELDS = (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_VR, _abi.FIELD_VZ, _abi.FIELD_FR,
          _abi.FIELD_STRESS, _abi.FIELD_PLASTIC_STRAIN)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
@pytest.mark.parametrize("count,nr,nz", [(1, 8, 16), (1, 3, 43), (2, 11, 24), (19, 9, 59),
                                         (37, 7, 37), (39, 10, 60), (77, 6, 31), (150, 5, 27)])
def test_instances_equal_single_scenes(gpu_lib, precision, count, nr, nz):
    rods = scenes.taylor_sweep(count, seed=count, t_end=1.0)
    for k, r in enumerate(rods):
        r.update(nr=nr, nz=nz - k % 2)                    # ragged by a row
    b = BatchSolver(scenes.sweep_instances(rods), Formulation.AXISYMMETRIC, cfl=0.6,
                    precision=precision)
    b.run(23)
    b.run(17)
    for k in sorted({0, count // 2, count - 1}):
        s, _, info = scenes.sweep_rod(ExplicitSolver, rods[k])
        s.setPrecision(precision)
        s.run(40)
        for f in FIELDS:
            assert np.array_equal(b.readInstance(f, k), s.readField(f)), (k, f)
        assert b.state()["time"][k] == s.time()
        w = b.wallStats()[k]
        assert (w.contact_count, w.stuck_count) == (info["wall"].contactCount(),
                                                    info["wall"].stuckCount())
        assert w.impulse == pytest.approx(info["wall"].impulse(), rel=1e-13)
        s.close()
    b.close()


@pytest.mark.gpu
def test_compensated_team_equals_one_block(gpu_lib):
    """The compensated form has no single-scene twin: a team against a batch of the same rods
    wide enough for one block each (its trajectories do not depend on the launch shape)."""
    rods = scenes.taylor_sweep(3, seed=9, t_end=1.0)
    few = BatchSolver(scenes.sweep_instances(rods), Formulation.AXISYMMETRIC, cfl=0.6,
                      precision=_abi.PRECISION_COMPENSATED)
    many = BatchSolver(scenes.sweep_instances(rods * 60), Formulation.AXISYMMETRIC, cfl=0.6,
                       precision=_abi.PRECISION_COMPENSATED)
    few.run(60)
    many.run(60)
    for k in range(3):
        for f in (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_STRESS, _abi.FIELD_PLASTIC_STRAIN):
            assert np.array_equal(few.readInstance(f, k), many.readInstance(f, k))
    few.close()
    many.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED,
                                       _abi.PRECISION_COMPENSATED])
def test_tuning_tries_staged_nodes_above_48_kb(gpu_lib, precision):
    """2,525 nodes staged take 60 kB: every shape of the tuner launches, whichever of the lone
    and the shared kernel its blocks per SM select, and the run goes on as if untuned."""
    rods = scenes.taylor_sweep(3, seed=2, t_end=1.0)
    for r in rods:
        r.update(nr=24, nz=100)
    batches = [BatchSolver(scenes.sweep_instances(rods), Formulation.AXISYMMETRIC, cfl=0.6,
                           precision=precision) for _ in range(2)]
    batches[0].tune(2)
    if precision != _abi.PRECISION_COMPENSATED:           # its one-warp kernels round differently
        for b in batches:
            b.run(12)
        for f in (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_STRESS):
            assert np.array_equal(batches[0].read(f), batches[1].read(f)), f
    if precision == _abi.PRECISION_MIXED:
        for blocks in (1, 2):
            batches[0].setConfig(128, 1, blocks, 8)
            batches[0].run(8)
    for b in batches:
        b.close()
