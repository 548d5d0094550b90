"""GPU: the final cost of a small survey in the mixed form does not depend on
rounding.  The settings are those that the integration notes give for models
of up to 200 cameras; the rounding is varied by the order of the points (the
order of every sum over them) and the PCG kernel (threads per CTA, autotuned
layouts).

Bound: the cost at which the reference's stop rule ends an FP64 solve depends
on the order of its sums by 1.17e-5 (four orders of a 500-camera survey on the
CPU; these small surveys on the GPU: 2e-8); the mixed
form, which stops after four undamped steps below 1e-6 each, has to end less
than half of that above it.  The stop itself is checked on the iteration log."""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options, Problem, survey

pytestmark = pytest.mark.gpu


def reordered(p, seed):
    """The same survey with its points in another order."""
    to = np.random.default_rng(seed).permutation(p.n_points).astype(np.uint32)
    o = np.argsort(to[p.obs_pt], kind="stable")
    pts = np.empty_like(p.points)
    pts[to] = p.points
    return Problem(intr=p.intr.copy(), rot=p.rot.copy(), center=p.center.copy(),
                   cam_group=p.cam_group, points=pts,
                   obs_cam=np.ascontiguousarray(p.obs_cam[o]),
                   obs_pt=np.ascontiguousarray(to[p.obs_pt][o]),
                   obs_uv=np.ascontiguousarray(p.obs_uv[o]), prior_mask=p.prior_mask,
                   prior=p.prior, refine_intrinsics=p.refine_intrinsics)


def stop_iteration(info, patience):
    """Iterations until `patience` accepted steps in a row decreased the cost by
    less than 1e-6, none of them with more damping than the last rejected step."""
    cost, rejected, small = info.initial_cost, np.inf, 0
    for i in range(info.iterations):
        if not info.accepted[i]:
            rejected = info.lam[i]
            continue
        rel = (cost - info.new_cost[i]) / cost
        cost = info.new_cost[i]
        small = small + 1 if rel < 1e-6 and info.lam[i] <= rejected else 0
        if small == patience:
            return i + 1
    return 60


@pytest.mark.parametrize("seed,kw", [(1, {}), (3, {}), (4, {}),
                                     (3, dict(n_cams=48, n_points=16000)),
                                     (6, dict(n_cams=110, n_points=60000))])
def test_mixed_cost_holds_over_rounding(seed, kw):
    p, _ = survey.generate("lawnmower77", seed=seed, **kw)
    _, ref = stitch_ba.bundle_adjust(p.copy(), 60, 1.0, return_info=True)
    opts = [dict(pcg_kernel="cluster"), dict(pcg_kernel="cluster_wide"), dict(autotune=True)]
    for k in range(9):
        q = reordered(p, k) if k >= 3 else p.copy()
        _, m = stitch_ba.bundle_adjust(q, 60, 1.0, Options(
            precision="mixed", coarse=True, pcg_max_iter=40, stop_patience=4,
            pcg_end_max_iter=200, pcg_end_rel=1e-5, **opts[k % 3]), return_info=True)
        assert m.iterations == stop_iteration(m, 4)
        assert m.final_cost <= ref.final_cost * (1.0 + 5e-6), (k, m.final_cost, ref.final_cost)
