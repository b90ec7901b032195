"""Launch plans after development leave room for rows that grow again; when a
plan with tracking fits without that room only, the plan without tracking is made
anew, and no graph may launch the old one."""
import numpy as np
import pytest

import mercury_b200 as mb
from test_gpu_devo import OracleRun, check_same
from test_gpu_tm import random_robot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replaced", [20, 60])
def test_a_plan_without_room_replaces_both(replaced):
    """1,024 masses of about nine own springs: with an eighth more, two masses a
    thread fit a CTA on 24 warps (untracked), not on the 16 that track."""
    batch = mb.pack([random_robot(1024, np.random.default_rng(1024), 9)])
    sim = mb.Simulator(0)
    sim.setTimeStep(1e-3)
    sim.set_batch(batch)
    orc = OracleRun(batch, mb.material_table(), 1e-3)
    sim.run_steps(5, True)
    orc.steps(5)
    assert sim.devo(replaced, seed=0) == orc.devo(replaced, 0)
    with_room = None
    for track in (False, True, False, True):  # the same graphs' keys again
        sim.Reset()
        orc.t = 0.0
        sim.run_steps(8, track)
        orc.steps(8, track)
        check_same(sim, orc)
        if not track:
            now = sim.step_variant()
            assert now["register_rows"] == 1 and (with_room is None or now["smem_bytes"] < with_room["smem_bytes"])
            with_room = with_room or now
