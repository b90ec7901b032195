"""The resident step kernel with operands in tensor memory against the CPU
oracle, bit for bit: random topologies at the edges of its slices (32
masses), warps and columns, every mode, and inputs that leave the fast
length and reciprocal.  Both sides round every operation once in the same
order, so every comparison is exact."""
import ctypes

import numpy as np
import pytest

import mercury_b200 as mb
from mercury_b200 import _lib
from mercury_b200 import simulator as S
from oracle import core

pytestmark = pytest.mark.gpu

ENV_KEYS = ("g", "floor_stiffness", "friction_static", "friction_kinetic", "drag", "damping")
ENVS = {0: None, 1: S.LAND, 2: S.WATER}


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def same(a, b):
    """Equal bits; any NaN equals any NaN."""
    return np.all((bits(a) == bits(b)) | (np.isnan(a) & np.isnan(b)))


def random_robot(n, rng, springs=8, materials=253, mass=1.0):
    """n masses in a unit box, about `springs` springs per mass (at most 26
    at one mass), ends in either order, doubled springs, springs from a mass
    to itself and air among them."""
    pos = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    deg = np.zeros(n, np.int64)
    pairs = []
    for a, b in rng.integers(0, n, (springs * n, 2)):
        if deg[a] < 25 and deg[b] < 25:
            pairs.append((a, b))
            deg[a] += 1
            deg[b] += 1
    pairs = np.array(pairs, np.uint16).reshape(-1, 2)
    d = pos[pairs[:, 0]] - pos[pairs[:, 1]]
    lbar = (np.sqrt((d * d).sum(1)) * rng.uniform(0.9, 1.1, len(pairs)) + 1e-3).astype(np.float32)
    mat = rng.integers(0, materials + 1, len(pairs)).astype(np.uint8)
    return mb.Element(pos, rng.integers(1, 23, n).astype(np.uint8), pairs, lbar, mat,
                      vel=rng.normal(0.0, 0.1, (n, 3)).astype(np.float32), mass=np.full(n, mass, np.float32))


def check(batch, mode, steps, track, dt, cfg=None):
    sim = mb.Simulator(0)
    table = mb.material_table()
    if mode:
        table = mb.materials.force_table()
        sim.set_materials(table)
        sim.set_mode(mode)
        sim.set_environment(**ENVS[mode])
    sim.setTimeStep(dt)
    if cfg:
        sim.set_launch_config(**cfg)
    sim.set_batch(batch)
    assert sim.step_variant()["register_rows"] == 1
    for n in (1, steps - 1):  # the state goes through memory between launches
        sim.run_steps(n, track)
    pos, vel, stress = sim.collect_arrays()
    p, v, s = batch.pos.copy(), batch.vel.copy(), np.zeros(batch.n_springs, np.float32)
    with np.errstate(all="ignore"):
        if mode:
            core.force_run(mode, batch, p, v, s, table, [ENVS[mode][k] for k in ENV_KEYS], dt, 0.0, steps, track)
        else:
            core.xpbd_run(batch, p, v, s, table, dt, 0.0, steps, track)
    assert same(pos, p) and same(vel, v)
    if track:
        assert same(stress, s)


@pytest.mark.parametrize("mode", [0, 1, 2], ids=["reference", "land", "water"])
@pytest.mark.parametrize("track", [False, True])
@pytest.mark.parametrize("sizes", [(1, 2, 3), (31, 32, 33), (63, 255, 256, 257), (700, 768, 769), (1000, 1024)])
def test_random_topologies_bit_exact(sizes, track, mode):
    rng = np.random.default_rng([len(sizes), sizes[0], mode])
    els = [random_robot(n, rng, mass=0.1 if mode else 1.0) for n in sizes]
    check(mb.pack(els), mode, 12, track, 1e-4 if mode else 1e-3)


@pytest.mark.parametrize("track", [False, True])
def test_several_bins_a_cta_bit_exact(track):
    """More robots than SMs, of 2 to 500 masses, a few with no springs: warp
    groups beside each other, several bins each, two masses a thread."""
    rng = np.random.default_rng(5)
    els = [random_robot(int(rng.integers(2, 200)) if r % 5 else int(rng.integers(300, 500)), rng,
                        springs=0 if r % 50 == 7 else 9) for r in range(600)]
    check(mb.pack(els), 0, 8, track, 1e-3)


@pytest.mark.parametrize("track", [False, True])
def test_lengths_outside_the_fast_path_bit_exact(track):
    """Coincident and nearly coincident masses, coordinates whose squared
    distance overflows, infinite and NaN coordinates, with and without
    springs; other robots of the launch stay finite."""
    rng = np.random.default_rng(11)
    els = [random_robot(90, rng) for _ in range(6)]
    els[0].pos[::3] = els[0].pos[0]
    els[1].pos[1::2] = els[1].pos[::2] + np.float32(3e-6)
    els[2].pos[5:9] = [[3e19, 0, 0], [-3e19, 1, 0], [1e38, 0, 0], [1e30, 1e30, 0]]
    els[3].pos[4:7] = [[np.inf, 0, 0], [0, -np.inf, 0], [0, np.nan, 0]]
    keep = ~np.isin(els[4].pairs, [10, 11, 12]).any(1)  # masses without springs, far away
    e = els[4]
    els[4] = mb.Element(e.pos, e.mass_material, e.pairs[keep], e.mean_length[keep], e.spring_material[keep], vel=e.vel)
    els[4].pos[10:13] = [[np.inf, 0, 0], [1e25, 0, 0], [np.nan, 0, 0]]
    check(mb.pack(els), 0, 6, track, 1e-3)


def test_length_and_reciprocal_of_every_float():
    n = ctypes.c_uint64(1)
    _lib.check(_lib.LIB.mb_check_spring_math(0, ctypes.byref(n)))
    assert n.value == 0


@pytest.mark.parametrize("track", [False, True])
@pytest.mark.parametrize("sizes", [(1, 3, 2), (32, 33), (255, 256, 257), (700, 769)])
def test_face_drag_bit_exact(sizes, track):
    """Random triangles (doubled and degenerate ones among them) on random
    robots; one mass is a corner of 200, more than its columns hold, one
    robot has none."""
    rng = np.random.default_rng([9, sum(sizes)])
    els = []
    for n in sizes:
        e = random_robot(n, rng, 6)
        if n >= 3:
            e.faces = rng.integers(0, n, (2 * n, 3)).astype(np.uint16)
            if n >= 255:
                e.faces = np.concatenate([e.faces, np.stack([np.full(200, 5), rng.integers(6, n, 200), rng.integers(6, n, 200)], 1)
                                          .astype(np.uint16)])
        els.append(e)
    batch = mb.pack(els)
    env = S.WATER_FACES
    sim = mb.Simulator(0)
    table = mb.materials.force_table()
    sim.set_materials(table)
    sim.set_mode(2)
    sim.set_environment(**env)
    sim.setTimeStep(1e-4)
    sim.set_batch(batch)
    assert sim.step_variant()["register_rows"] == 1
    keys = ENV_KEYS + ("face_drag",)
    p, v, s = batch.pos.copy(), batch.vel.copy(), np.zeros(batch.n_springs, np.float32)
    t0 = 0.0
    for drag in (env["face_drag"], 0.0, env["face_drag"]):  # the drag off and on again between runs
        on = dict(env, face_drag=drag)
        sim.set_environment(**on)
        sim.run_steps(7, track)
        with np.errstate(all="ignore"):
            core.force_run(2, batch, p, v, s, table, [on[k] for k in keys], 1e-4, t0, 7, track)
        t0 = sim.getTotalTime()
    pos, vel, stress = sim.collect_arrays()
    assert same(pos, p) and same(vel, v)
    if track:
        assert same(stress, s)
