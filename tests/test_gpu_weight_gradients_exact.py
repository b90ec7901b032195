"""The surrogate's gradients on networks of small whole numbers, where every
activation and gradient is exact in BF16 and every sum in FP32: they equal the
oracle's in 64 bits whatever the order of the sums, so one wrong row, neighbour
or offset shows.  Row counts (216 a sample) around the weight gradient's tiles
of 128 rows, their last one of 32 or 96, and the edges of 1 to 27 splits."""
import numpy as np
import pytest

from mercury_b200.surrogate import Surrogate
from oracle import surrogate as so


def network(rng):
    """A few weights of +-1 a row, biases of 0 and 1."""
    p = {}
    for name, rows, cols, taps in (("W1", 32, 216, 24), ("W2", 32, 864, 6), ("W3", 32, 864, 4), ("W4", 128, 6912, 24),
                                   ("W5", 128, 128, 2), ("W6", 1, 128, 40)):
        w = np.zeros((rows, cols), np.float32)
        used = np.flatnonzero(np.arange(cols) % 8 < 5) if name == "W1" else np.arange(cols)
        for row in w:
            row[rng.choice(used, taps, replace=False)] = rng.choice([-1.0, 1.0], taps)
        p[name] = w
    for name, n in (("b1", 32), ("b2", 32), ("b3", 32), ("b4", 128), ("b5", 128), ("b6", 1)):
        p[name] = rng.integers(0, 2, n).astype(np.float32)
    return so.flatten(p)


def case(n):
    assert np.float32(n) * (np.float32(1) / np.float32(n)) == 1  # dy = 2 (y - t) / n is exact then
    rng = np.random.default_rng(n)
    flat = network(rng)
    genomes = rng.integers(0, 5, (n, 216)).astype(np.uint8)
    y = so.Net(flat, exact=True).forward(genomes)
    y = np.asarray(y[0] if isinstance(y, tuple) else y, np.float64).reshape(-1)
    targets = (y - n * rng.choice([-0.5, 0.5], n)).astype(np.float32)  # dy = +-1
    return flat, genomes, targets


SIZES = [1, 2, 3, 5, 10, 19, 38, 128]


@pytest.mark.parametrize("n", SIZES[:5])
def test_values_are_exact_in_bf16(n):
    flat, genomes, targets = case(n)
    lo, _, go = so.Net(flat, exact=True).loss_and_grads(genomes, targets)
    lr, _, gr = so.Net(flat).loss_and_grads(genomes, targets)
    for name in so.NAMES:
        assert np.array_equal(np.asarray(go[name], np.float64), np.asarray(gr[name], np.float64)), name
        assert np.count_nonzero(go[name]) > 0, name


@pytest.mark.gpu
@pytest.mark.parametrize("tcgen05", [True, False])
@pytest.mark.parametrize("n", SIZES)
def test_gradients_are_exact(n, tcgen05):
    flat, genomes, targets = case(n)
    s = Surrogate(0, max_batch=max(SIZES))
    s.use_tcgen05(tcgen05)
    s.set_params(flat)
    _, g = s.gradients(genomes, targets)
    _, _, go = so.Net(flat, exact=True).loss_and_grads(genomes, targets)
    gf = so.unflatten(g)
    for name in so.NAMES:
        a, b = gf[name].astype(np.float64), np.asarray(go[name], np.float64).reshape(-1)
        assert np.array_equal(a, b), (name, np.flatnonzero(a != b)[:8])
