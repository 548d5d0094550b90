"""GPU: the FP64 form's sums per camera, each shared out to several CTAs: a
camera of no observation, of one, of one less and one more than the threads of
a CTA; with and without the lens terms.  Against the oracle, 1e-12 of the
largest entry as in the other element-wise tests."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Options, Problem
from test_gpu_pcg_grid import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("groups", [1, 2])
def test_camera_sums(refine, groups):
    q = network(5, 3, 129, groups, seed=groups)
    seen = [(0, 1, 2)] * 127 + [(0, 1), (0, 3)]  # 129, 128, 127, 1 and 0 observations
    cam = np.concatenate(seen)
    pt = np.repeat(np.arange(129), [len(s) for s in seen])
    pts = np.column_stack([np.random.default_rng(3).uniform(-9, 15, (129, 2)), np.zeros(129)])
    x = np.einsum("nij,nj->ni", q.rot[cam], pts[pt] - q.center[cam])
    uv = 3000.0 * x[:, :2] / x[:, 2:] + [2000.0, 1500.0]
    uv += np.random.default_rng(4).normal(0, 0.5, uv.shape)
    p = Problem(intr=q.intr, rot=q.rot, center=q.center, cam_group=q.cam_group, points=pts,
                obs_cam=cam, obs_pt=pt, obs_uv=uv, prior_mask=q.prior_mask, prior=q.prior,
                refine_intrinsics=refine)
    r = O.lm_step(p, 1e-2, 4.0)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(1e-2, 4.0, Options())
    for key in ("S", "g"):
        assert np.abs(d[key] - r[key]).max() <= 1e-12 * np.abs(r[key]).max()
