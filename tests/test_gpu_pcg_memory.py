"""GPU: the grid PCG holds no more device memory than the vectors and counters
that it replaced: models whose S blocks exceed shared memory, several lens
rows and a batch keep within the workspace limit that they needed before
(measured then), but for exchange words of 0.01 % of it."""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options, Problem

pytestmark = pytest.mark.gpu


def random_views(n_cams, n_points, views, groups, seed):
    """Points seen by `views` random cameras each: a dense reduced matrix."""
    rng = np.random.default_rng(seed)
    cam = np.sort(np.argsort(rng.random((n_points, n_cams)), 1)[:, :views], 1).reshape(-1)
    pt = np.repeat(np.arange(n_points), views)
    rot = np.tile(np.diag([1.0, -1.0, -1.0]), (n_cams, 1, 1))
    center = np.column_stack([rng.uniform(-30, 30, (n_cams, 2)), 80 + rng.uniform(-2, 2, n_cams)])
    pts = np.column_stack([rng.uniform(-30, 30, (n_points, 2)), rng.uniform(-4, 4, n_points)])
    x = np.einsum("nij,nj->ni", rot[cam], pts[pt] - center[cam])
    uv = 3000.0 * x[:, :2] / x[:, 2:] + [2000.0, 1500.0] + rng.normal(0, 0.5, (len(cam), 2))
    prior = np.concatenate([center, np.tile([2.0, 2.0, 4.0], (n_cams, 1))], 1)
    return Problem(intr=np.tile([3000.0, 2000.0, 1500.0, 0.0, 0.0], (groups, 1)), rot=rot,
                   center=center + rng.normal(0, 0.05, center.shape),
                   cam_group=np.arange(n_cams) % groups, points=pts, obs_cam=cam, obs_pt=pt,
                   obs_uv=uv, prior_mask=np.ones(n_cams, np.uint8), prior=prior,
                   refine_intrinsics=True)


BEFORE = {("one", "fp64"): 67106178, ("one", "mixed"): 45645046,
          ("three", "fp64"): 69480364, ("three", "mixed"): 47437808,
          ("batch", "fp64"): 168394044, ("batch", "mixed"): 116092620}


@pytest.mark.parametrize("case", [("one", 1), ("three", 3), ("batch", 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_workspace_limit_of_before(case, precision):
    name, groups = case
    if name == "batch":
        ps = [random_views(20 + 5 * m, 200, 8, 1, seed=m) for m in range(40)]
    else:
        ps = [random_views(300, 6000, 8, groups, seed=1)]
    limit = int(BEFORE[name, precision] * 1.0001)
    opt = Options(precision=precision, pcg_kernel="grid", workspace_limit_bytes=limit)
    info = stitch_ba.bundle_adjust_batch(ps, 2, 1.0, opt)[0]
    assert info.pcg_kernel == "grid" and info.device_bytes <= limit
