"""GPU: the grid PCG kernel on a survey whose last photo shares points with
every other one (a high overview beside a flight line).  Its block row costs
as much as several CTAs' rows, so the rows run out before the CTAs that the
group was sized for; above 32 CTAs the group is led by the CTA of the lens row,
the last one with rows.

The step is checked against the system it was computed from: the residual
S dx - g of a solve that stopped at |r|^2 < 1e-20 |b|^2 (FP64; 1e-10 in the
mixed form) is 1e-10 |g| (1e-5) plus the drift of the recurrence, at most one
rounding of |S| |dx| per iteration (400 iterations)."""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options, Problem

pytestmark = pytest.mark.gpu


def overview(n_cams, span, n_points, seed):
    """A flight line whose points are seen by `span` consecutive photos and by
    the last one."""
    rng = np.random.default_rng(seed)
    rot = np.tile(np.diag([1.0, -1.0, -1.0]), (n_cams, 1, 1))
    center = np.column_stack([3.0 * np.arange(n_cams), rng.uniform(-9, 9, n_cams),
                              80.0 + rng.uniform(-2, 2, n_cams)])
    center[-1] = [1.5 * n_cams, 0.0, 900.0]
    first = rng.integers(0, n_cams - span, n_points)
    pts = np.column_stack([3.0 * (first + 0.5 * span) + rng.uniform(-5, 5, n_points),
                           rng.uniform(-20, 20, n_points), rng.uniform(-4, 4, n_points)])
    cam = np.concatenate([first[:, None] + np.arange(span),
                          np.full((n_points, 1), n_cams - 1)], 1).reshape(-1)
    pt = np.repeat(np.arange(n_points), span + 1)
    x = np.einsum("nij,nj->ni", rot[cam], pts[pt] - center[cam])
    uv = 3000.0 * x[:, :2] / x[:, 2:] + [2000.0, 1500.0] + rng.normal(0, 0.5, (len(cam), 2))
    prior = np.concatenate([center, np.tile([2.0, 2.0, 4.0], (n_cams, 1))], 1)
    return Problem(intr=[[3000.0, 2000.0, 1500.0, 0.0, 0.0]], rot=rot,
                   center=center + rng.normal(0, 0.05, center.shape), cam_group=np.zeros(n_cams),
                   points=pts, obs_cam=cam, obs_pt=pt, obs_uv=uv,
                   prior_mask=np.ones(n_cams, np.uint8), prior=prior, refine_intrinsics=True)


@pytest.mark.parametrize("precision,n_cams", [
    ("fp64", 100),   # 26 CTAs of four rows: all decide
    ("fp64", 200),   # 51 planned, the last one without rows
    ("fp64", 300),   # 76, two without
    ("mixed", 300),  # 38 of eight rows
    ("mixed", 600),  # 76, two without
])
def test_step_solves_its_system(precision, n_cams):
    p = overview(n_cams, 4, 6 * n_cams, seed=n_cams)
    opt = Options(precision=precision, pcg_kernel="grid",
                  pcg_tol=1e-20 if precision == "fp64" else 1e-10)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(1.0, 1.0, opt)
    assert 0 < d["pcg_iters"] < 400
    S, g, dx = d["S"], d["g"], d["dx"]
    eps, tol = (2.0**-53, 1e-10) if precision == "fp64" else (2.0**-24, 1e-5)
    drift = 400 * eps * np.linalg.norm(np.abs(S) @ np.abs(dx))
    assert np.linalg.norm(S @ dx - g) <= tol * np.linalg.norm(g) + drift
