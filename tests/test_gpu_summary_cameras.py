"""GPU: the summary with so many cameras that a CTA keeps fewer depth keys in
shared memory: cameras below, at and above that number, and the most cameras
whose counts it keeps there and one more.  Bit-exact, as the other summary
tests."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [12_000, 13_000, 24_576, 24_577])
def test_summary_of_many_cameras(nc):
    rng = np.random.default_rng(nc)
    npts = 9000
    sizes = np.full(nc, 2)
    sizes[:6] = 1023, 1024, 1025, 9000, 10, 9
    sizes[nc - 1] = 8193
    cam = np.repeat(np.arange(nc), sizes)
    pt = np.concatenate([rng.permutation(npts)[:s] for s in sizes])
    order = np.lexsort((cam, pt))
    oc, op = cam[order].astype(np.uint32), pt[order].astype(np.uint32)
    p = Problem(intr=[[1000.0, 0, 0, 0, 0]], rot=np.tile(np.eye(3), (nc, 1, 1)),
                center=rng.normal(0, 5, (nc, 3)), cam_group=np.zeros(nc),
                points=rng.normal(0, 30, (npts, 3)), obs_cam=oc, obs_pt=op,
                obs_uv=np.zeros((len(oc), 2)))
    out = stitch_ba.sparse_summary(p, agl=80.0)
    nb, sh, _, depth_range, _ = O.sparse_summary(oc, op, p.rot, p.center, p.points, agl=80.0)
    assert np.array_equal(out.depth_range, depth_range)
    assert np.array_equal(out.neighbours, nb) and np.array_equal(out.shared, sh)
