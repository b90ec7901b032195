"""Simulators on threads of one process: launches that need much shared memory
beside launches of the same kernels that need little."""
import threading

import numpy as np
import pytest

import mercury_b200 as mb
from test_step_plan import population

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [{}, {"threads": 512, "springs_per_thread": 16, "masses_per_thread": 4}])
def test_simulators_on_threads(cfg):
    batches = [population(20, lo, hi, 3) for lo, hi in ((2, 3), (6, 6), (2, 2), (5, 6))]

    def simulator(b):
        sim = mb.Simulator(0)
        sim.setTimeStep(1e-3)
        sim.set_launch_config(use_graph=0, **cfg)
        sim.set_batch(b)
        return sim

    want = []
    for b in batches:
        sim = simulator(b)
        sim.run_steps(300)
        want.append(sim.collect_arrays()[0])
    got, errors = [None] * len(batches), []

    def work(i):
        try:
            sim = simulator(batches[i])
            for _ in range(300):
                sim.run_steps(1)
            got[i] = sim.collect_arrays()[0]
        except Exception as e:  # shown by the assertion below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(batches))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(got, want))
