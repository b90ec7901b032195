"""New topologies on one simulator: the resident kernel's rows come with the
upload, its plan and graphs stay while the new rows fit them, and springs are
placed for the general kernel when that is asked for.  Bits do not depend on
what was uploaded before."""
import numpy as np
import pytest

import mercury_b200 as mb
from mercury_b200 import robots
from mercury_b200 import simulator as S
from test_step_plan import population

pytestmark = pytest.mark.gpu


def bits(arrays):
    return [np.ascontiguousarray(a).view(np.uint32) for a in arrays]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(bits(a), bits(b)))


def voxel(sim, cells, steps, track):
    sim.set_voxel_population(cells, 0.1, 0.1)
    sim.Reset()
    sim.run_steps(steps, track)
    return sim.collect_arrays()


def land():
    sim = mb.Simulator(0)
    sim.set_materials(mb.materials.force_table())
    sim.set_mode(S.MODE_FORCE_LAND)
    sim.set_environment(**S.LAND)
    sim.setTimeStep(1e-4)
    return sim


@pytest.mark.parametrize("count,side", [(5, 4), (200, 3), (400, 6)])
def test_voxel_populations_one_after_another(count, side):
    """Sparse, full, nearly empty and sparse robots again: rows shrink and grow
    within the template's."""
    rng = np.random.default_rng([count, side])
    used = land()
    for fill in (0.5, 1.0, 0.02, 0.6):
        cells = np.where(rng.random((count, side, side, side)) < fill,
                         robots.FOUR[rng.integers(0, 4, (count, side, side, side))], 0).astype(np.uint8)
        for track in (False, True):
            assert same(voxel(used, cells, 30, track), voxel(land(), cells, 30, track))


@pytest.mark.parametrize("count,lo", [(1, 4), (40, 3), (300, 3)])
def test_uploads_one_after_another(count, lo):
    used = mb.Simulator(0)
    used.setTimeStep(1e-3)
    for seed in range(3):
        b = population(count, lo, 6, seed)
        fresh = mb.Simulator(0)
        fresh.setTimeStep(1e-3)
        for sim in (used, fresh):
            sim.set_batch(b)
            sim.Reset()
            sim.run_steps(20, seed == 1)
        assert same(used.collect_arrays(), fresh.collect_arrays())


def test_springs_are_placed_when_asked_for(monkeypatch):
    """The packed springs are those of the host packer, whether they are read
    before or after steps that did not need them placed."""
    b = population(30, 3, 6, 1)
    monkeypatch.setenv("MB_HOST_ROWS", "1")
    host = mb.Simulator(0)
    host.set_batch(b)
    want = host.packed_springs()
    monkeypatch.delenv("MB_HOST_ROWS")
    got = []
    for first in (True, False):
        sim = mb.Simulator(0)
        sim.setTimeStep(1e-3)
        sim.set_batch(b)
        if first:
            assert np.array_equal(sim.packed_springs(), want)
        sim.run_steps(10, True)
        assert np.array_equal(sim.packed_springs(), want)
        sim.run_steps(10, True)
        sim.devo(20, 1)
        sim.run_steps(10, True)
        got.append(sim.collect_arrays())
    assert same(*got)
