"""GPU: order statistics selected inside a CTA (depth ranges of the summary)
at the sizes where they can go wrong: the ranks' edges, keys
that fill shared memory or exceed it by one, equal values, one value.

The summary's depths are bit-exact (no fused operation on either side)."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Problem

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
