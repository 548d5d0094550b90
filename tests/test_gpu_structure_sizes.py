"""GPU: the sort and the pair list at the sizes where their work is cut: tiles
of 4096 items and one more, digits of one bit up, two and three passes (the
result in either buffer); points whose entries just fit a warp's lanes.

Against the oracle: depth ranges are bit-exact (no fused operation on either
side, and a misplaced item changes a camera's range), the reduced matrix to
1e-12 of its largest entry as in the other element-wise tests."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Options, Problem
from test_gpu_pcg_grid import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_obs,n_cams", [(1, 1), (4095, 1), (4096, 2), (4097, 31), (8193, 511),
                                          (20_000, 512), (70_001, 700)])
def test_observations_by_camera(n_obs, n_cams):
    rng = np.random.default_rng(n_obs)
    n_pts = max(1, n_obs // 5)
    key = rng.choice(n_pts * n_cams, n_obs, replace=False) if n_pts * n_cams > n_obs else \
        np.arange(n_obs) % (n_pts * n_cams)
    key.sort()
    op, oc = (key // n_cams).astype(np.uint32), (key % n_cams).astype(np.uint32)
    X = rng.normal(0, 30, (n_pts, 3))
    R, C = np.tile(np.eye(3), (n_cams, 1, 1)), rng.normal(0, 5, (n_cams, 3))
    p = Problem(intr=[[1000.0, 0, 0, 0, 0]], rot=R, center=C, cam_group=np.zeros(n_cams),
                points=X, obs_cam=oc, obs_pt=op, obs_uv=np.zeros((n_obs, 2)))
    out = stitch_ba.sparse_summary(p, agl=80.0)
    nb, _, _, depth_range, _ = O.sparse_summary(oc, op, R, C, X, agl=80.0)
    assert np.array_equal(out.depth_range, depth_range)
    assert np.array_equal(out.neighbours, nb)


@pytest.mark.parametrize("n_cams,span,n_points", [
    (2, 2, 5), (40, 31, 60), (40, 32, 60),  # 32 entries with the lens, 33
    (520, 4, 2500),                         # keys of 19 bits: three passes
])
def test_pair_list(n_cams, span, n_points):
    p = network(n_cams, span, n_points, 1, seed=span)
    r = O.lm_step(p, 1e-2, 4.0)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(1e-2, 4.0, Options())
    assert np.abs(d["S"] - r["S"]).max() <= 1e-12 * np.abs(r["S"]).max()
    assert np.array_equal(d["S"], d["S"].T)
