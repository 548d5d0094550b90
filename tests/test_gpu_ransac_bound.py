"""GPU: the inlier counts of RANSAC while the bound that ends them moves: most
samples hold mismatches, so the warps of a CTA leave hypotheses half counted
against a best count that the others raise.  Best hypothesis, counts and flags
equal the oracle's, and a second call's equal the first's."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import PairMatches
from test_gpu_ransac_sizes import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outliers", [0.5, 0.8])
@pytest.mark.parametrize("sizes", [(1300,) * 6, (2048, 2049, 6000), (129, 160, 257, 500)])
def test_bounded_counts_equal_oracle(sizes, outliers):
    iters = 1500
    uv = np.concatenate([scene(n, 11 * i + n, outliers) for i, n in enumerate(sizes)])
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    pairs = np.array([(i, i + 1) for i in range(len(sizes))], np.uint32)
    seeds = (pairs[:, 0].astype(np.uint64) * 7919 + pairs[:, 1]).astype(np.uint64)
    m = PairMatches(pairs, ptr, uv)
    got = stitch_ba.ransac_fundamental(m, 1.5, iters)
    again = stitch_ba.ransac_fundamental(m, 1.5, iters)
    want = O.ransac_fundamental(ptr, uv, seeds, 1.5, iters)
    for a, b, c in zip(got, again, want):
        assert np.array_equal(a, b) and np.array_equal(a, c)
