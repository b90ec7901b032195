"""The general step kernels (springs of a thread in tensor memory, two at a
time) against the CPU oracle, bit for bit: spring counts around the edges of
a warp, of a thread's pairs and of the block, lengths that leave the fast
square root and reciprocal, resident, split and streamed."""
import numpy as np
import pytest

import mercury_b200 as mb
from mercury_b200 import simulator as S
from oracle import core

pytestmark = pytest.mark.gpu

ENV_KEYS = ("g", "floor_stiffness", "friction_static", "friction_kinetic", "drag", "damping")
ENVS = {0: None, 1: S.LAND, 2: S.WATER}


def robot(n, m, rng):
    """n masses, m springs, 30 of them (where there are so many) at mass 0;
    two coincident masses, two 3e-6 apart, one 1e20 away."""
    pos = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    pos[1] = pos[0]
    pos[3] = pos[2] + np.float32(3e-6)
    pos[4] = 1e20
    pairs = np.stack([rng.integers(0, n, m), rng.integers(0, n, m)], 1).astype(np.uint16)
    hub = np.arange(m) < min(m, 30)
    pairs[hub] = np.stack([np.zeros(hub.sum()), 5 + np.arange(hub.sum()) % (n - 5)], 1)
    pairs[-1] = (0, 1)
    pairs[m // 2] = (3, 2)
    lbar = rng.uniform(0.2, 1.0, m).astype(np.float32)
    return mb.Element(pos, rng.integers(1, 23, n).astype(np.uint8), pairs, lbar, rng.integers(0, 23, m).astype(np.uint8),
                      vel=np.zeros((n, 3), np.float32), mass=np.full(n, 1.0, np.float32))


def check(sim, batch, mode, track, steps):
    table = mb.material_table()
    if mode:
        table = mb.materials.force_table()
        sim.set_materials(table)
        sim.set_mode(mode)
        sim.set_environment(**ENVS[mode])
    sim.setTimeStep(1e-4)
    sim.set_batch(batch)
    sim.run_steps(steps, track)
    got = sim.collect_arrays()
    p, v, s = batch.pos.copy(), batch.vel.copy(), np.zeros(batch.n_springs, np.float32)
    with np.errstate(all="ignore"):
        if mode:
            core.force_run(mode, batch, p, v, s, table, [ENVS[mode][k] for k in ENV_KEYS], 1e-4, 0.0, steps, track)
        else:
            core.xpbd_run(batch, p, v, s, table, 1e-4, 0.0, steps, track)
    for a, b in zip(got, (p, v, s) if track else (p, v)):
        u, w = np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32)
        assert np.all((u == w) | (np.isnan(a) & np.isnan(b)))


@pytest.mark.parametrize("mode", [0, 1, 2], ids=["reference", "land", "water"])
@pytest.mark.parametrize("track", [False, True])
@pytest.mark.parametrize("m", [31, 33, 1024, 1025, 2047, 2049, 6200])
def test_spring_counts_bit_exact(m, track, mode):
    rng = np.random.default_rng([m, mode])
    sim = mb.Simulator(0)
    check(sim, mb.pack([robot(max(40, m // 8), m, rng)]), mode, track, 6)
    assert sim.step_variant()["register_rows"] == 0


@pytest.mark.parametrize("cluster", [2, 4])
@pytest.mark.parametrize("mode", [0, 2], ids=["reference", "water"])
def test_split_bit_exact(mode, cluster):
    rng = np.random.default_rng([7, mode])
    sim = mb.Simulator(0)
    sim.set_launch_config(cluster=cluster)
    check(sim, mb.pack([robot(700, 4100, rng), robot(650, 5001, rng)]), mode, True, 6)
    assert sim.launch_config()["cluster"] == cluster
