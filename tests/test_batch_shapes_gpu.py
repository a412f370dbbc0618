"""Launch shapes of the batch: which are accepted, and that they step the instances alike."""
import numpy as np
import pytest

from neofiz_gb300 import ExplicitSolver, _abi, scenes
from neofiz_gb300.batch import BatchSolver
from neofiz_gb300.materials import Formulation

pytestmark = pytest.mark.gpu


def batch(rods, precision=_abi.PRECISION_FP64):
    return BatchSolver(scenes.sweep_instances(rods), Formulation.AXISYMMETRIC, cfl=0.6,
                       precision=precision)


@pytest.mark.parametrize("threads,blocks", [(256, 1), (128, 3), (32, 12)])
def test_fp64_shapes_of_384_threads_per_sm_are_accepted(gpu_lib, threads, blocks):
    """Shapes that FP64 batches took when their kernels held 168 registers a thread."""
    rods = scenes.taylor_sweep(5, seed=4, t_end=1.0)
    for r in rods:
        r.update(nr=5, nz=23)
    a, b = batch(rods), batch(rods)
    a.setConfig(threads, 0, blocks, 16)
    assert a.config() == {"threads": threads, "stage_nodes": 0, "blocks_per_sm": blocks,
                          "chunk_steps": 16}
    with pytest.raises(ValueError):
        a.setConfig(threads, 0, blocks + 1, 16)
    for s in (a, b):
        s.run(30)
    for f in (_abi.FIELD_UR, _abi.FIELD_UZ, _abi.FIELD_STRESS):
        assert np.array_equal(a.read(f), b.read(f)), f
    a.close()
    b.close()


def test_elapsed_leaves_out_the_building_of_graphs(gpu_lib):
    """A run whose launches are captured anew takes no more device time than one that replays
    them: 40 runs of one step each way, by turns. The capture takes 25 us of host time and up, the
    step 120 us; the two medians have to lie within 12 us."""
    b = batch(scenes.taylor_sweep(4, seed=1, t_end=1.0))
    b.run(20)
    anew, again = [], []
    for k in range(40):
        b.setConfig(256, 0, 1, 100 + k)
        anew.append(b.run(1))
        again.append(b.run(1))
    b.close()
    assert abs(np.median(anew) - np.median(again)) < 0.012, (np.median(anew), np.median(again))


@pytest.mark.parametrize("precision,count", [(_abi.PRECISION_MIXED, 256),
                                             (_abi.PRECISION_COMPENSATED, 512)])
def test_tuning_a_ragged_batch_does_not_lose_to_the_default(gpu_lib, precision, count):
    """Rods whose finest take four times the steps of the coarsest: the shape that tune keeps runs
    them no slower than the untuned one, within a tenth."""
    rods = scenes.taylor_sweep(count, seed=5, t_end=6.0e-6)
    a, b = batch(rods, precision), batch(rods, precision)
    b.tune()
    assert b.run() < 1.1 * a.run()
    a.close()
    b.close()


@pytest.mark.parametrize("precision,nr,nz,count,threads", [
    (_abi.PRECISION_MIXED, 8, 16, 16, 256),       # 153 nodes: two rounds of 128 threads
    (_abi.PRECISION_MIXED, 8, 16, 700, 128),      # more than the 256-thread blocks' 304 places
    (_abi.PRECISION_MIXED, 7, 12, 16, 128),       # 104 nodes
    (_abi.PRECISION_MIXED, 4, 8, 16, 128),        # 45 nodes: two rounds of 32 threads
    (_abi.PRECISION_MIXED, 4, 8, 1200, 32),
    (_abi.PRECISION_COMPENSATED, 8, 16, 16, 256),
    (_abi.PRECISION_FP64, 4, 8, 16, 32),
    (_abi.PRECISION_FP64, 10, 60, 700, 256)])
def test_default_blocks_are_narrow_only_where_that_helps(gpu_lib, precision, nr, nz, count, threads):
    rods = scenes.taylor_sweep(1, seed=4, t_end=1.0)
    rods[0].update(nr=nr, nz=nz)
    b = batch(rods * count, precision)
    assert b.config()["threads"] == threads
    b.run(9)
    s, _, _ = scenes.sweep_rod(ExplicitSolver, rods[0])
    if precision != _abi.PRECISION_COMPENSATED:           # which has no single scene
        s.setPrecision(precision)
        s.run(9)
        for k in (0, count - 1):
            assert np.array_equal(b.readInstance(_abi.FIELD_UZ, k), s.readField(_abi.FIELD_UZ))
    s.close()
    b.close()
