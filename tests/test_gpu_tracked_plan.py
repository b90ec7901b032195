"""Stress tracking on the resident kernel whatever the bins: with one and two
masses a thread, up to the 1,024 masses a bin may hold, against the CPU oracle
bit for bit; mean lengths whose reciprocal is not an ordinary one."""
import numpy as np
import pytest

import mercury_b200 as mb
from mercury_b200 import simulator as S
from oracle import core
from test_gpu_step_plan import run
from test_gpu_tm import ENV_KEYS, check, random_robot, same
from test_step_plan import population

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2], ids=["reference", "land", "water"])
@pytest.mark.parametrize("sizes", [(33,), (511, 513), (700, 768, 769), (1000, 1024)])
def test_tracked_bins_on_the_resident_kernel(sizes, mode):
    rng = np.random.default_rng([len(sizes), sizes[0], mode])
    batch = mb.pack([random_robot(n, rng, mass=0.1 if mode else 1.0) for n in sizes])
    sim = mb.Simulator(0)
    sim.set_mode(mode)
    sim.set_batch(batch)
    assert sim.step_variant(track_stresses=True)["register_rows"] == 1
    assert sim.step_variant(True) == mb.plan_step_variant(batch, True)
    check(batch, mode, 12, True, 1e-4 if mode else 1e-3)


@pytest.mark.parametrize("count,lo", [(260, 5), (414, 5), (512, 3)])
def test_tracked_populations_bit_exact(count, lo):
    b = population(count, lo, 8, 1)
    sim = run(b, 20, True)
    assert sim.step_variant(True)["register_rows"] == 1


@pytest.mark.parametrize("sizes", [(32, 40), (700, 800)])
def test_tracked_faces_bit_exact(sizes):
    rng = np.random.default_rng([3, sum(sizes)])
    els = [random_robot(n, rng, 6) for n in sizes]
    for e, n in zip(els, sizes):
        e.faces = rng.integers(0, n, (2 * n, 3)).astype(np.uint16)
    batch = mb.pack(els)
    table = mb.materials.force_table()
    sim = mb.Simulator(0)
    sim.set_materials(table)
    sim.set_mode(2)
    sim.set_environment(**S.WATER_FACES)
    sim.setTimeStep(1e-4)
    sim.set_batch(batch)
    assert sim.step_variant(True)["register_rows"] == 1
    sim.run_steps(8, True)
    p, v, s = batch.pos.copy(), batch.vel.copy(), np.zeros(batch.n_springs, np.float32)
    with np.errstate(all="ignore"):
        core.force_run(2, batch, p, v, s, table, [S.WATER_FACES[k] for k in ENV_KEYS + ("face_drag",)], 1e-4, 0.0, 8, True)
    assert all(same(a, b) for a, b in zip(sim.collect_arrays(), (p, v, s)))


@pytest.mark.parametrize("n", [40, 90])
def test_unusual_mean_lengths_bit_exact(n):
    """Zero, tiny, huge and negative mean lengths and ones whose significand is
    all ones: their reciprocals are not the fast path's."""
    rng = np.random.default_rng(n)
    els = [random_robot(n, rng) for _ in range(3)]
    odd = np.array([0.0, -0.0, 1e-42, 1e-39, 3e38, -0.25, np.nextafter(np.float32(1), np.float32(0)), 1e-30], np.float32)
    els[0].mean_length[:] = odd[rng.integers(0, len(odd), len(els[0].mean_length))]
    els[1].mean_length[5] = np.nextafter(np.float32(0.5), np.float32(0))
    check(mb.pack(els), 0, 8, True, 1e-3)
