"""GPU: RANSAC at the sizes where its passes change: pairs with barely enough
matches (most samples repeat an index), more matches than a tile, one and two
CTAs a pair and more, hypothesis counts that are no multiple of anything, and
a call large enough for a copy of its own.  Scenes of full depth, where a
sample fixes its hypothesis: best hypothesis, counts and flags equal the
oracle's."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import PairMatches

pytestmark = pytest.mark.gpu


def scene(n, seed, outliers=0.3):
    rng = np.random.default_rng(seed)
    X = np.column_stack([rng.uniform(-40, 40, n), rng.uniform(-40, 40, n), rng.uniform(30, 120, n)])
    a, f, c = 0.2, 2000.0, (2000.0, 1500.0)
    R = np.array([[np.cos(a), 0, np.sin(a)], [0, 1, 0], [-np.sin(a), 0, np.cos(a)]])
    Y = (X - [9.0, 3.0, 2.0]) @ R.T
    uv = np.concatenate([f * X[:, :2] / X[:, 2:] + c, f * Y[:, :2] / Y[:, 2:] + c], 1)
    uv += rng.normal(0, 0.3, uv.shape)
    bad = rng.random(n) < outliers
    uv[bad, 2:] = rng.uniform(0, 4000, (bad.sum(), 2))
    return uv


@pytest.mark.parametrize("sizes,iters", [
    ((0, 11, 12, 13, 16, 24), 600),
    ((31, 32, 33, 64, 100), 257),
    ((2047, 2048, 2049, 5000), 600),
    ((300,) * 700, 65),
    ((200, 900), 1),
    ((260_000, 40_000), 70),
])
def test_ransac_equals_oracle(sizes, iters):
    uv = np.concatenate([scene(n, 7 * i + n) for i, n in enumerate(sizes)])
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    pairs = np.array([(i, i + 1) for i in range(len(sizes))], np.uint32)
    seeds = (pairs[:, 0].astype(np.uint64) * 7919 + pairs[:, 1]).astype(np.uint64)
    inl, n, best, refit = stitch_ba.ransac_fundamental(PairMatches(pairs, ptr, uv), 1.5, iters)
    oi, on, ob, orf = O.ransac_fundamental(ptr, uv, seeds, 1.5, iters)
    assert np.array_equal(best, ob)
    assert np.array_equal(n, on) and np.array_equal(inl, oi) and np.array_equal(refit, orf)
