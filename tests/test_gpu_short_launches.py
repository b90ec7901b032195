"""Launches of a few steps, with and without tracking, in turn: the same bits
whichever steps, after an upload, after development (whose rows, with 4,096
records or more, are queued and waited for by the next launch) and with chunks of
a step."""
import numpy as np
import pytest

import mercury_b200 as mb
from mercury_b200 import robots
from mercury_b200 import simulator as S
from test_gpu_devo import OracleRun, check_same
from test_step_plan import population

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,lo,hi", [(1, 1, 1), (3, 2, 5), (150, 2, 4), (310, 2, 6)])
def test_short_and_long_launches_in_turn(count, lo, hi):
    b = population(count, lo, hi, 7)
    sim = mb.Simulator(0)
    sim.setTimeStep(1e-3)
    sim.set_batch(b)
    orc = OracleRun(b, mb.material_table(), np.float32(1e-3))
    k = 16 if count > 300 else 9  # 4,960 records: the rows are queued after the call's wait
    for cycle in range(3):
        for steps, track in ((1, True), (3, True), (2, True), (1, False), (4, False), (2, True)):
            sim.run_steps(steps, track)
            orc.steps(steps, track)
        check_same(sim, orc)
        assert sim.devo(k, seed=cycle) == orc.devo(k, cycle)
        if cycle == 1:  # another one before any step
            assert sim.devo(k, seed=40) == orc.devo(k, 40)
    sim.run_steps(6, True)
    orc.steps(6, True)
    check_same(sim, orc)


def test_chunks_of_a_step():
    b = population(20, 3, 6, 2)
    sim = mb.Simulator(0)
    sim.setTimeStep(1e-3)
    sim.set_launch_config(chunk=1)
    sim.set_batch(b)
    orc = OracleRun(b, mb.material_table(), np.float32(1e-3))
    for track in (True, False, True):
        sim.run_steps(5, track)
        orc.steps(5, track)
    check_same(sim, orc)


@pytest.mark.parametrize("faces", [False, True], ids=["water", "faces"])
@pytest.mark.parametrize("count", [3, 160])
def test_short_launches_in_water(count, faces):
    """Six tracked steps in one launch and in launches of one and two."""
    els = []
    for r in range(count):
        cells = robots.random_cells(2 + r % 5, np.random.default_rng([count, r]))
        els.append(robots.voxel_robot(cells, mass=0.1))
        if faces:
            els[-1].faces = robots.voxel_faces(cells)
    b, got = mb.pack(els), []
    for launches in ((6,), (1, 2, 1, 2)):
        sim = mb.Simulator(0)
        sim.set_materials(mb.materials.force_table())
        sim.set_mode(S.MODE_FORCE_WATER)
        sim.set_environment(**{**S.WATER, "face_drag": 1000.0 if faces else 0.0})
        sim.setTimeStep(1e-4)
        sim.set_batch(b)
        for n in launches:
            sim.run_steps(n, True)
        got.append(sim.collect_arrays())
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(*got))
