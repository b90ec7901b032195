"""The launch plan of the resident step kernel over ordinary populations,
planned on the host: a CTA's shared memory stays within what the device
gives a CTA (232,448 bytes on B200), and none of it is static, which the
plan would not count."""
import os
import re

import numpy as np
import pytest

import mercury_b200 as mb
from mercury_b200 import robots

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMEM = 232448


def population(count, lo, hi, seed):
    els = []
    for r in range(count):
        rng = np.random.default_rng([seed, r])
        els.append(robots.voxel_robot(robots.random_cells(int(rng.integers(lo, hi + 1)), rng)))
    return mb.pack(els)


@pytest.mark.parametrize("lo", [3, 4, 5])
@pytest.mark.parametrize("count", [150, 236, 322, 392, 436, 512, 600, 700])
def test_plans_fit_a_cta(count, lo):
    b = population(count, lo, 8, count)
    v = mb.plan_step_variant(b)
    assert v["register_rows"] == 1 and v["smem_bytes"] <= SMEM
    assert mb.plan_step_variant(b, track_stresses=True)["smem_bytes"] <= SMEM


def test_the_resident_kernel_has_no_static_shared_memory():
    src = open(os.path.join(ROOT, "mercury_b200", "csrc", "mb_tm.cu")).read()
    kernel = src[src.index("tm_step_kernel("):src.index("tm_rows_kernel(")]
    assert not re.search(r"^(?!.*extern).*__shared__", kernel, re.M)
