"""The surrogate's weight and bias gradients at the edges of their kernels --
one split and several, a last tile of 128 rows partly filled, the cap of 64
splits, more samples than a tile of the head -- against the oracle.  Both
round activations and gradients to BF16 (2^-9) at six layers, at places that
can differ where sums do: 3e-2 of a tensor's norm."""
import numpy as np
import pytest

from mercury_b200.surrogate import Surrogate
from oracle import surrogate as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 10, 33, 304, 600])
def test_gradients_at_the_tile_edges(n):
    rng = np.random.default_rng(40 + n)
    flat = so.init_params(11)
    s = Surrogate(0, max_batch=600)
    s.set_params(flat)
    genomes = rng.integers(0, 5, (n, 216)).astype(np.uint8)
    targets = rng.normal(size=n).astype(np.float32)
    loss, g = s.gradients(genomes, targets)
    loss2, g2 = s.gradients(genomes, targets)
    assert loss == loss2 and np.array_equal(np.asarray(g).view(np.uint32), np.asarray(g2).view(np.uint32))
    lo, _, go = so.Net(flat).loss_and_grads(genomes, targets)
    assert abs(loss - lo) <= 1e-2 * lo
    gf = so.unflatten(g)
    for name in so.NAMES:
        a, b = gf[name].astype(np.float64), np.asarray(go[name], np.float64).reshape(-1)
        assert np.linalg.norm(a - b) < 3e-2 * np.linalg.norm(b), name
