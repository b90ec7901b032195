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


@pytest.mark.parametrize("count,side,least,most", [(4096, 1, 1, 8), (16384, 1, 1, 16), (4096, 2, 1, 12), (1638, 6, 12, 12),
                                                   (512, 6, 3, 4), (149, 8, 2, 2)])
def test_small_robots_share_bins(count, side, least, most):
    """Bins a CTA: robots of a slice or less share bins, so that a CTA steps its
    bins side by side; large ones have a bin each."""
    one = robots.voxel_robot(np.full((side,) * 3, robots.BONE, np.uint8))
    st = mb.plan(mb.pack([one] * count))
    assert st["ctas"] == 148 and st["bins"] % 148 == 0 and least <= st["bins"] // 148 <= most
    assert mb.plan_step_variant(mb.pack([one] * count))["register_rows"] == 1
