"""GPU: points of ba_triangulate where its two eigenvector methods meet: tracks
that settle at once, tracks of rays that are nearly or exactly parallel,
mismatched ones, one camera twice, and a point far behind the others.

The points are compared with numpy's eigenvectors of the same normal matrices
in 64 bits, both with the matrices' own sensitivity: a matrix rounded in its
last place moves the eigenvector by eps |A| / (lambda_3 - lambda_4), of which
each side makes a few (8 are allowed), relative to the point's distance."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Tracks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [2, 3, 9])
@pytest.mark.parametrize("n_tracks", [1, 127, 1500])
def test_points_match_eigenvectors(views, n_tracks):
    rng = np.random.default_rng(10 * views + n_tracks)
    nc = 24
    R = np.stack([O.from_angles(rng.uniform(0, 360), -90.0 + rng.uniform(-8, 8), 0.0)
                  for _ in range(nc)])
    C = np.column_stack([rng.uniform(0, 300, nc), rng.uniform(0, 200, nc), 80 + rng.uniform(-4, 4, nc)])
    K = np.array([[3650.0, 2736.0, 1824.0, 0.02, -0.01]])
    cam = np.stack([rng.permutation(nc)[:views] for _ in range(n_tracks)])
    X = np.column_stack([rng.uniform(0, 300, n_tracks), rng.uniform(0, 200, n_tracks),
                         rng.uniform(-5, 5, n_tracks)])
    X[::11] = [150.0, 100.0, -40000.0]          # all rays nearly parallel
    uv = np.zeros((n_tracks, views, 2))
    for t in range(n_tracks):
        for v in range(views):
            uv[t, v] = O.project(R[cam[t, v]], C[cam[t, v]], K[0], X[t])
    uv += rng.normal(0, 0.5, uv.shape)
    uv[3::17] = rng.uniform(0, 3600, uv[3::17].shape)   # mismatches: no point fits
    cam[5::23], uv[5::23] = cam[5::23, :1], uv[5::23, :1]  # one camera's ray, repeated
    ptr = (views * np.arange(n_tracks + 1)).astype(np.uint32)
    oc = np.ascontiguousarray(cam.reshape(-1), np.uint32)
    tr = Tracks(ptr, oc, np.ascontiguousarray(uv.reshape(-1, 2)), np.zeros(nc, np.uint32), 1)
    kept, pts, good = stitch_ba.triangulate(tr, R, C, K, 1e6)
    ko, _, go = O.triangulate(ptr, oc, tr.obs_uv, R, C, K, tr.cam_group, 1e6)
    assert np.array_equal(kept, ko) and np.array_equal(good, go)
    # normal matrices of the undistorted rays (geometry.rs:118-131)
    q = (uv - K[0, 1:3]) / K[0, 0]
    x = q.copy()
    for _ in range(8):
        r2 = (x * x).sum(-1, keepdims=True)
        x = q / (1.0 + K[0, 3] * r2 + K[0, 4] * r2 * r2)
    Pm = np.concatenate([R, -(R @ C[:, :, None])], 2)[cam]
    rows = (x[..., None] * Pm[:, :, 2:3] - Pm[:, :, :2]).reshape(n_tracks, -1, 4)
    w, v = np.linalg.eigh(np.swapaxes(rows, 1, 2) @ rows)
    ref = v[:, :3, 0] / v[:, 3:, 0]
    size = np.sqrt(1.0 + (ref**2).sum(1))
    # unit eigenvector's error, and its last component's relative one
    move = 8 * 2.0**-52 * w[:, 3] / (w[:, 1] - w[:, 0]) * size
    err = np.linalg.norm(pts - ref, axis=1) / size
    assert (err[kept] <= move[kept]).all(), (err[kept] / move[kept]).max()
