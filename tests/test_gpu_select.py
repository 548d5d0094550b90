"""GPU: order statistics selected inside a CTA (depth ranges of the summary,
pair medians) at the sizes where they can go wrong: the ranks' edges, keys
that fill shared memory or exceed it by one, equal values, one value.

The summary's depths are bit-exact (no fused operation on either side); the
medians keep the bound of the other pair check tests (1e-9 of the largest:
the oracle's Sampson error differs by fused operations)."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import PairMatches, Problem, survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 9, 10, 11), (19, 20, 21, 511), (512, 513, 8191, 8192),
                                   (8193, 10, 20000, 0)])
@pytest.mark.parametrize("levels", [0, 3])
def test_depth_ranges_match_oracle(sizes, levels):
    """Camera c sees the first sizes[c] points; levels: that many distinct depths."""
    rng = np.random.default_rng(sum(sizes) + levels)
    nc, npts = len(sizes), max(sizes)
    pt = np.concatenate([np.arange(s) for s in sizes])
    cam = np.repeat(np.arange(nc), sizes)
    order = np.lexsort((cam, pt))
    X = rng.normal(0, 30, (npts, 3))
    if levels:
        X[:, 2] = rng.integers(0, levels, npts) * 7.0 - 5.0
    R = np.tile(np.eye(3), (nc, 1, 1))
    C = rng.normal(0, 5, (nc, 3))
    oc, op = cam[order].astype(np.uint32), pt[order].astype(np.uint32)
    p = Problem(intr=[[1000.0, 0, 0, 0, 0]], rot=R, center=C, cam_group=np.zeros(nc),
                points=X, obs_cam=oc, obs_pt=op, obs_uv=np.zeros((len(oc), 2)))
    out = stitch_ba.sparse_summary(p, agl=80.0)
    nb, _, _, depth_range, _ = O.sparse_summary(oc, op, R, C, X, agl=80.0)
    assert np.array_equal(out.depth_range, depth_range)
    assert np.array_equal(out.neighbours, nb)


@pytest.mark.parametrize("sizes", [(1, 2, 3, 0, 255, 256, 257), (3071, 3072, 3073, 9000),
                                   (700_000, 5, 400_000)])
def test_pair_medians_match_oracle(sizes):
    """Up to the pairs that go through global memory, and a call large enough
    to be copied in two pieces (1.1 million matches)."""
    rng = np.random.default_rng(len(sizes))
    p, _ = survey.generate("lawnmower77", seed=3, n_cams=8, n_points=400)
    n = sum(sizes)
    uv = rng.uniform([0, 0, 0, 0], [5472, 3648, 5472, 3648], (n, 4))
    uv[::5] = uv[0]                        # equal errors
    uv[1::7, :2] = p.intr[0, 1:3]          # the principal point: a zero quotient
    pairs = np.array([(i, i + 1) for i in range(len(sizes))], np.uint32)
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    med = stitch_ba.pair_fits(PairMatches(pairs, ptr, uv), p.rot, p.center, p.intr, p.cam_group)
    ref = O.pair_fits(pairs, ptr, uv, p.rot, p.center, p.intr, p.cam_group)
    some = np.array(sizes) > 0
    assert np.abs(med - ref)[some].max() <= 1e-9 * np.abs(ref[some]).max()
    assert np.array_equal(med[~some], ref[~some])
