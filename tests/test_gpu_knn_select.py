"""The neighbour selection of mb_knn_springs at its edges: clouds around one
warp and one word of the pair sets, the largest cloud, coincident points, and
infinite and NaN coordinates, against a plain restatement of the insertion
it stands for (index order, before the first of the list that is farther)."""
import numpy as np
import pytest

from mercury_b200 import robots

pytestmark = pytest.mark.gpu


def neighbours(p, i, k):
    with np.errstate(all="ignore"):
        d = p - p[i]
        d2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    k = min(k, len(p) - 1)
    near = []
    for j in range(len(p)):
        if j == i or (len(near) == k and not (k and d2[j] < d2[near[-1]])):
            continue
        at = len(near)
        if at == k:
            near.pop()
            at -= 1
        while at and d2[j] < d2[near[at - 1]]:
            at -= 1
        near.insert(at, j)
    return near


def pairs_of(p, k):
    got = {(min(i, j), max(i, j)) for i in range(len(p)) for j in neighbours(p, i, k)}
    return np.array(sorted(got), np.uint16).reshape(-1, 2)


def check(clouds, k):
    rng = np.random.default_rng(3)
    mats = [robots.FOUR[rng.integers(0, 4, len(p))] for p in clouds]
    so, pairs, _, lbar = robots.knn_springs(clouds, mats, k)
    for r, p in enumerate(clouds):
        s = slice(int(so[r]), int(so[r + 1]))
        want = pairs_of(p, k)
        assert np.array_equal(pairs[s], want)
        with np.errstate(all="ignore"):
            d = p[want[:, 0]] - p[want[:, 1]]
            length = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        assert np.array_equal(lbar[s], length, equal_nan=True)


@pytest.mark.parametrize("k", [1, 31, 32])
def test_cloud_sizes_around_a_warp(k):
    rng = np.random.default_rng(k)
    check([rng.normal(size=(n, 3)).astype(np.float32) for n in (1, 2, 31, 32, 33, 34, 63, 64, 65, 97, 129)], k)


def test_coincident_infinite_and_nan_points():
    rng = np.random.default_rng(5)
    clouds = [rng.normal(size=(80, 3)).astype(np.float32) for _ in range(4)]
    clouds[0][10:50] = clouds[0][3]
    clouds[1][[0, 40, 79]] = [[np.inf, 0, 0], [0, -np.inf, 0], [1e30, 0, 0]]
    clouds[2][[5, 60]] = np.nan
    clouds[3][:] = clouds[3][0]
    check(clouds, 25)


def test_largest_cloud():
    rng = np.random.default_rng(8)
    p = rng.uniform(size=(4096, 3)).astype(np.float32)
    so, pairs, _, _ = robots.knn_springs([p], [np.full(4096, 22, np.uint8)], 32)
    got = set(map(tuple, pairs.tolist()))
    for i in rng.integers(0, 4096, 40):
        assert all((min(i, j), max(i, j)) in got for j in neighbours(p, int(i), 32))
    d = np.full(4096, 0)
    np.add.at(d, pairs.reshape(-1).astype(int), 1)
    assert d.min() >= 32 and len(got) == int(so[-1]) <= 4096 * 32
