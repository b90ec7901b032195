"""Launch plans that take all the shared memory of a CTA, and the first that
does not fit, against the CPU oracle bit for bit, on the kernel that the host
planner names; whole populations of large bins."""
import numpy as np
import pytest

import mercury_b200 as mb
from oracle import core
from test_gpu_tm import random_robot
from test_step_plan import SMEM, population

pytestmark = pytest.mark.gpu


def run(batch, steps, track, **cfg):
    sim = mb.Simulator(0)
    sim.set_launch_config(**cfg)
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
def test_large_populations_bit_exact(count, lo):
    b = population(count, lo, 8, 1)
    sim = run(b, 20, False, bins=444)
    assert sim.step_variant() == mb.plan_step_variant(b, bins=444)
    assert sim.step_variant()["register_rows"] == 1


@pytest.mark.parametrize("track", [False, True])
@pytest.mark.parametrize("n", [1000, 1024])
def test_full_cta_bit_exact(n, track):
    """One robot with as many springs as the plan has room for, and with one
    more: in every slice of 32 masses one mass has its springs to lower masses,
    so that a spring more is a column of 32 slots more."""
    rng = np.random.default_rng(n)
    whole = random_robot(n, rng, 0)
    deg, pairs = np.zeros(n, int), []
    for _ in range(22):
        for m in range(63, n, 32):
            used = [b for a, b in pairs if a == m]
            free = np.setdiff1d(np.arange(m), used)
            low = free[np.argmin(deg[free])]
            pairs.append((m, low))
            deg[[m, low]] += 1
    pairs = np.array(pairs, np.uint16)
    lbar = rng.uniform(0.2, 1.0, len(pairs)).astype(np.float32)

    def robot(k):
        return mb.pack([mb.Element(whole.pos, whole.mass_material, pairs[:k], lbar[:k], np.full(k, 5, np.uint8),
                                   vel=whole.vel)])

    few, many = n // 4, len(pairs)  # the former fits, the latter does not
    assert mb.plan_step_variant(robot(few), track)["register_rows"] > mb.plan_step_variant(robot(many), track)["register_rows"]
    while many - few > 1:
        k = (few + many) // 2
        few, many = (k, many) if mb.plan_step_variant(robot(k), track)["register_rows"] else (few, k)
    v = run(robot(few), 20, track).step_variant(track)
    assert v == mb.plan_step_variant(robot(few), track) and v["register_rows"] == 1
    assert SMEM - 1024 < v["smem_bytes"] <= SMEM
    assert run(robot(many), 20, track).step_variant(track)["register_rows"] == 0


@pytest.mark.parametrize("track", [False, True])
@pytest.mark.parametrize("count,lo,hi", [(149, 1, 1), (300, 1, 4), (1000, 1, 2), (2000, 1, 1)])
def test_small_robots_bit_exact(count, lo, hi, track):
    """Bins of several small robots, and CTAs that get fewer bins than others."""
    b = population(count, lo, hi, 2)
    assert run(b, 20, track).step_variant(track)["register_rows"] == 1
