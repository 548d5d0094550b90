"""GPU: the tracks and observations that a round's problem keeps are those of
ba_triangulate, whose flags a caller uses to name them, on tracks whose
decisions are close (a gate in the middle of the residuals, rays near the
smallest angle, mismatches, one camera twice) and in coordinates far from the
origin, where rounding moves a point by more than its last digits.

The points may be formed by another method; both are eigenvectors of the same
normal matrix in 64 bits, so they differ by its sensitivity at most: a matrix
rounded in its last place moves the eigenvector by eps |A| / gap, of which each
side makes a few (8 a side are allowed).  And they differ by no more than the
header says, 2^-26 of the distance to a camera."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Problem, Tracks

pytestmark = pytest.mark.gpu


def tracks(n_tracks, offset, seed):
    rng = np.random.default_rng(seed)
    nc = 24
    R = np.stack([O.from_angles(rng.uniform(0, 360), -90.0 + rng.uniform(-8, 8), 0.0)
                  for _ in range(nc)])
    C = np.column_stack([rng.uniform(0, 300, nc), rng.uniform(0, 200, nc),
                         80 + rng.uniform(-4, 4, nc)]) + [offset, 0.5 * offset, 0.0]
    K = np.array([[3650.0, 2736.0, 1824.0, 0.02, -0.01]])
    views = rng.integers(2, 7, n_tracks)
    ptr = np.concatenate([[0], np.cumsum(views)]).astype(np.uint32)
    X = np.column_stack([rng.uniform(0, 300, n_tracks), rng.uniform(0, 200, n_tracks),
                         rng.uniform(-5, 5, n_tracks)]) + [offset, 0.5 * offset, 0.0]
    X[::11, 2] = -600.0                        # rays a few degrees apart
    cam = np.concatenate([rng.permutation(nc)[:v] for v in views]).astype(np.uint32)
    trk = np.repeat(np.arange(n_tracks), views)
    x = np.einsum("nij,nj->ni", R[cam], X[trk] - C[cam])
    p = x[:, :2] / x[:, 2:]
    r2 = (p * p).sum(1, keepdims=True)
    uv = K[0, 0] * (1 + K[0, 3] * r2 + K[0, 4] * r2 * r2) * p + K[0, 1:3]
    uv += rng.normal(0, 2.0, uv.shape)
    bad = rng.random(len(uv)) < 0.03
    uv[bad] = rng.uniform(0, 3600, (bad.sum(), 2))
    twice = ptr[5:-1:23].astype(np.int64)      # the second view repeats the first
    cam[twice + 1], uv[twice + 1] = cam[twice], uv[twice]
    return Tracks(ptr, cam, np.ascontiguousarray(uv), np.zeros(nc, np.uint32), 1), R, C, K


@pytest.mark.parametrize("thr", [1.0, 3.0, 50.0])
@pytest.mark.parametrize("offset", [0.0, 2.0e4, 1.0e6])
def test_a_round_keeps_what_triangulation_keeps(offset, thr):
    tr, R, C, K = tracks(20_000, offset, seed=7)
    kept, pts, good = stitch_ba.triangulate(tr, R, C, K, thr)
    with stitch_ba.Context() as ctx:
        n_pts, n_obs = ctx.upload_tracks(tr, R, C, K, thr)
        assert n_pts == int(kept.sum()) and n_obs == int(good.sum())
        q = Problem.empty(len(C), n_pts, n_obs, 1)
        ctx.solve(0, 1.0)
        ctx.download(q)
    ptr = tr.track_ptr.astype(np.int64)
    uv, cam = tr.obs_uv, tr.obs_cam
    x = n = (uv - K[0, 1:3]) / K[0, 0]
    for _ in range(8):
        r2 = (x * x).sum(1, keepdims=True)
        x = n / (1.0 + K[0, 3] * r2 + K[0, 4] * r2 * r2)
    Pm = np.concatenate([R, -(R @ C[:, :, None])], 2)[cam]
    rows = x[:, :, None] * Pm[:, 2:3] - Pm[:, :2]
    M = np.add.reduceat(np.einsum("nri,nrj->nij", rows, rows), ptr[:-1], axis=0)
    w = np.linalg.eigvalsh(M)[kept]
    a, b = pts[kept], q.points
    size = np.sqrt(1.0 + (a * a).sum(1))
    # the unit eigenvector's move, and that of its last component (1 / size)
    move = 16 * 2.0**-52 * w[:, 3] / (w[:, 1] - w[:, 0]) * size
    assert (np.linalg.norm(a - b, axis=1) / size <= move + 2.0**-50).all()
    dist = np.linalg.norm(a - C[cam[ptr[:-1][kept]]], axis=1)
    assert (np.linalg.norm(a - b, axis=1) <= 2.0**-26 * dist).all()
