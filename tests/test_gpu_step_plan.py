"""Populations whose launch plan takes all the shared memory of a CTA, against
the CPU oracle bit for bit, on the kernel that the host planner names."""
import numpy as np
import pytest

import mercury_b200 as mb
from oracle import core
from test_step_plan import SMEM, population

pytestmark = pytest.mark.gpu


def run(batch, steps, track):
    sim = mb.Simulator(0)
    sim.setTimeStep(1e-3)
    sim.set_batch(batch)
    sim.run_steps(steps, track)
    pos, vel, stress = sim.collect_arrays()
    p, v, s = batch.pos.copy(), batch.vel.copy(), np.zeros(batch.n_springs, np.float32)
    core.xpbd_run(batch, p, v, s, mb.material_table(), 1e-3, 0.0, steps, track)
    for a, b in ((pos, p), (vel, v)) + (((stress, s),) if track else ()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    return sim


@pytest.mark.parametrize("count,lo", [(480, 4), (512, 5), (400, 5), (590, 3)])
def test_full_ctas_bit_exact(count, lo):
    b = population(count, lo, 8, 1)
    sim = run(b, 20, False)
    v = sim.step_variant()
    assert v == mb.plan_step_variant(b)
    assert v["register_rows"] == 1 and SMEM - 1024 <= v["smem_bytes"] <= SMEM
