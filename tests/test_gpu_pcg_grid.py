"""GPU: the grid PCG kernel at the sizes where its split changes: one CTA,
a group whose CTAs all decide (up to 32), a group led by its last CTA, rows
with more than 32 blocks, more blocks than shared memory holds, several lens
rows; both storage precisions.

The step is checked against the system it was computed from: the residual
S dx - g of a solve that stopped at |r|^2 < 1e-20 |b|^2 is 1e-10 |g| plus the
drift of the recurrence, at most one rounding of |S| |dx| per iteration (400
iterations), and the stopping test must have fired for that bound to hold.
"""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options, Problem

pytestmark = pytest.mark.gpu


def network(n_cams, span, n_points, groups, seed):
    """Nadir cameras on a line; point i is seen by `span` consecutive ones."""
    rng = np.random.default_rng(seed)
    rot = np.tile(np.diag([1.0, -1.0, -1.0]), (n_cams, 1, 1))
    center = np.column_stack([3.0 * np.arange(n_cams), rng.uniform(-9, 9, n_cams),
                              80.0 + rng.uniform(-2, 2, n_cams)])
    first = rng.integers(0, n_cams - span + 1, n_points)
    pts = np.column_stack([3.0 * (first + 0.5 * span) + rng.uniform(-5, 5, n_points),
                           rng.uniform(-20, 20, n_points), rng.uniform(-4, 4, n_points)])
    cam = (first[:, None] + np.arange(span)).reshape(-1)
    pt = np.repeat(np.arange(n_points), span)
    x = np.einsum("nij,nj->ni", rot[cam], pts[pt] - center[cam])
    uv = 3000.0 * x[:, :2] / x[:, 2:] + [2000.0, 1500.0] + rng.normal(0, 0.5, (len(cam), 2))
    prior = np.concatenate([center, np.tile([2.0, 2.0, 4.0], (n_cams, 1))], 1)
    return Problem(intr=np.tile([3000.0, 2000.0, 1500.0, 0.0, 0.0], (groups, 1)), rot=rot,
                   center=center + rng.normal(0, 0.05, center.shape),
                   cam_group=np.arange(n_cams) % groups, points=pts, obs_cam=cam, obs_pt=pt,
                   obs_uv=uv, prior_mask=np.ones(n_cams, np.uint8), prior=prior,
                   refine_intrinsics=True)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_cams,span,n_points,groups", [
    (2, 2, 40, 1),        # one CTA
    (12, 5, 300, 1),
    (40, 8, 500, 1),      # rows of 16 blocks with the lens block
    (40, 9, 500, 1),      # of 18
    (127, 6, 3000, 1),    # 32 CTAs of four rows: all decide
    (128, 6, 3000, 1),    # 33: the last one decides
    (150, 17, 2500, 1),   # rows of 33 blocks and the lens block
    (130, 90, 400, 1),    # more blocks than shared memory holds
    (60, 8, 900, 3),      # three lens rows
])
def test_grid_pcg_solves_its_system(precision, n_cams, span, n_points, groups):
    p = network(n_cams, span, n_points, groups, seed=n_cams + span)
    opt = Options(precision=precision, pcg_kernel="grid",
                  pcg_tol=1e-20 if precision == "fp64" else 1e-10)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(1.0, 1.0, opt)
        again = ctx.debug_step(1.0, 1.0, opt)
    assert 0 < d["pcg_iters"] < 400
    assert np.array_equal(d["dx"], again["dx"])
    S, g, dx = d["S"], d["g"], d["dx"]
    eps, tol = (2.0**-53, 1e-10) if precision == "fp64" else (2.0**-24, 1e-5)
    drift = 400 * eps * np.linalg.norm(np.abs(S) @ np.abs(dx))
    assert np.linalg.norm(S @ dx - g) <= tol * np.linalg.norm(g) + drift
