"""An instance's sums do not depend on its neighbours in the batch. How many blocks step an
instance follows from how many instances there are and how large they are: alone a rod has
clusters of eight blocks, among 160 it has one block."""
import numpy as np
import pytest

from neofiz_gb300 import _abi, scenes
from neofiz_gb300.batch import BatchSolver
from neofiz_gb300.materials import Formulation

pytestmark = pytest.mark.gpu


def rod(nr, nz, t_end):
    r = scenes.taylor_sweep(1, seed=21)[0]
    r.update(nr=nr, nz=nz, t_end=t_end)
    return r


def others(count, t_end):
    out = scenes.taylor_sweep(count, seed=5)
    for r in out:
        r.update(nr=4, nz=20, t_end=t_end)
    return out


def gradients(instances, cfl, objectives, sample=0):
    b = BatchSolver(instances, Formulation.AXISYMMETRIC, cfl=cfl)
    b.adjointForward(16, sample)
    values, grads = b.adjointBackwardMany(objectives)
    b.close()
    return values[:, 0], grads[:, 0]


# 2,400 elements wrap round the lanes that the sums are dealt to (eight blocks of 256)
@pytest.mark.parametrize("nr,nz,t_end", [(10, 60, 4.0e-6), (3, 11, 4.0e-6), (48, 50, 0.3e-6)])
def test_gradients_do_not_depend_on_the_neighbours(gpu_lib, nr, nz, t_end):
    one = rod(nr, nz, t_end)
    objectives = [_abi.OBJECTIVE_LENGTH_RATIO, _abi.OBJECTIVE_MUSHROOM]
    alone = gradients(scenes.sweep_instances([one]), 0.6, objectives)
    assert np.abs(alone[1]).max() > 0.0
    for count in (10, 40, 160):
        among = gradients(scenes.sweep_instances([one] + [one] * (count // 2)
                                                 + others(count - count // 2, t_end)),
                          0.6, objectives)
        assert np.array_equal(alone[0], among[0]) and np.array_equal(alone[1], among[1]), count


def test_sampled_peak_does_not_depend_on_the_neighbours(gpu_lib):
    def tube():
        return scenes.tube_instance(nz=100, height=20.0e-3, t_end=14.0e-6, scale=0.04)
    objectives = [_abi.OBJECTIVE_PEAK_CAPACITY]
    alone = gradients([tube()], 0.5, objectives, sample=5)
    for count in (40, 160):
        among = gradients([tube() for _ in range(count)], 0.5, objectives, sample=5)
        assert np.array_equal(alone[0], among[0]) and np.array_equal(alone[1], among[1]), count


def wall_totals(instances, precision, config=None):
    b = BatchSolver(instances, Formulation.AXISYMMETRIC, cfl=0.6, precision=precision)
    if config:
        b.setConfig(*config)
    b.run(150)
    b.run(75)
    w = b.wallStats()[0]
    b.close()
    return w.impulse, w.energy_loss, w.friction_dissipation


# every node of these rods' feet touches the wall: 161 and 25 of them, five warps and one. Blocks
# of 32, 128 and 256 threads by turns, for the neighbours' size or because the shape asks for it
@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED,
                                       _abi.PRECISION_COMPENSATED])
@pytest.mark.parametrize("nr,nz,config", [(160, 3, (128, 0, 1, 256)), (24, 1, (128, 0, 1, 256)),
                                          (160, 14, (256, 0, 1, 256))])
def test_wall_totals_do_not_depend_on_the_neighbours(gpu_lib, precision, nr, nz, config):
    one = rod(nr, nz, 1.0)

    def among(count, size):
        rods = [one] + [one] * (count // 2) + others(count - count // 2, 1.0)
        for r in rods[len(rods) - count // 3:]:
            r.update(nr=size, nz=2 * size)
        return scenes.sweep_instances(rods)

    alone = wall_totals(scenes.sweep_instances([one]), precision)
    assert all(t != 0.0 for t in alone)
    assert alone == wall_totals(scenes.sweep_instances([one]), precision, config)
    for count, size in ((3, 3), (40, 5), (40, 12), (160, 12), (700, 4)):
        assert wall_totals(among(count, size), precision) == alone, (count, size)
