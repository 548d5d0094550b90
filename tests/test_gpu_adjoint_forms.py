"""GPU: the adjoint's ways through its inputs: one lens group a model
(observation order) or several (camera order), several models in a context,
cameras with no observation, one, and more than their CTAs' threads; both
losses.  Against the oracle's Jacobians, with the bound of the other adjoint
test (1e-10 of the largest entry)."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Options, Problem, survey

pytestmark = pytest.mark.gpu


def cut(seed, n_cams, n_points, groups):
    p, _ = survey.generate("lawnmower77", seed=seed, n_cams=n_cams, n_points=n_points)
    keep = np.ones(p.n_obs, bool)
    keep[p.obs_cam == 0] = False                       # a camera without observations
    one = np.nonzero(p.obs_cam == 1)[0]
    keep[one[1:]] = False                              # and one with a single one
    return Problem(intr=np.repeat(p.intr, groups, 0), rot=p.rot, center=p.center,
                   cam_group=np.arange(n_cams) % groups, points=p.points, obs_cam=p.obs_cam[keep],
                   obs_pt=p.obs_pt[keep], obs_uv=p.obs_uv[keep], prior_mask=p.prior_mask,
                   prior=p.prior)


@pytest.mark.parametrize("groups", [1, 3])
@pytest.mark.parametrize("models", [1, 3])
@pytest.mark.parametrize("loss", ["cauchy", "huber"])
def test_gradients_match_oracle_jacobians(groups, models, loss):
    ps = [cut(5 + m, 9 + m, 1200 + 900 * m, groups) for m in range(models)]
    rng = np.random.default_rng(1)
    lam = [rng.standard_normal((p.n_obs, 2)) for p in ps]
    mu = [rng.standard_normal((p.n_cams, 3)) for p in ps]
    opt = Options(loss=loss)
    with stitch_ba.Context() as ctx:
        ctx.upload(ps)
        grad = ctx.intrinsics_grad(1.5, opt)
        gc, gp, gi = ctx.vjp(1.5, np.concatenate(lam), np.concatenate(mu), opt)
        _, _, again = ctx.vjp(1.5, None, None, opt)
    ref = dict(grad=[], gc=[], gp=[], gi=[])
    for p, l, u in zip(ps, lam, mu):
        lo = O.linearise(p, 1.5, loss=1 if loss == "huber" else 0)
        v = lo["valid"].astype(bool)
        grp = p.cam_group[p.obs_cam]
        for name, cot in (("gi", l), ("grad", 2.0 * lo["w"][:, None] * lo["e"])):
            g = np.zeros((groups, 5))
            jg = -np.einsum("kij,ki->kj", lo["jg"][v], cot[v])
            for k, c in enumerate((0, 3, 4)):
                g[:, c] = np.bincount(grp[v], jg[:, k], groups)
            for k in (0, 1):
                g[:, 1 + k] = np.bincount(grp[v], -cot[v, k], groups)
            ref[name].append(g)
        c6, p3 = np.zeros((p.n_cams, 6)), np.zeros((p.n_points, 3))
        np.add.at(c6, p.obs_cam[v], -np.einsum("kij,ki->kj", lo["jc"][v], l[v]))
        np.add.at(p3, p.obs_pt[v], -np.einsum("kij,ki->kj", lo["jp"][v], l[v]))
        c6[:, 3:] += u / p.prior[:, 3:]
        ref["gc"].append(c6), ref["gp"].append(p3)
    for got, name in ((grad, "grad"), (again, "grad"), (gc, "gc"), (gp, "gp"), (gi, "gi")):
        want = np.concatenate(ref[name])
        scale = np.abs(want).max(0) if name in ("grad", "gi") else np.abs(want).max()
        assert (np.abs(got - want) <= 1e-10 * np.maximum(scale, 1e-300)).all(), name
