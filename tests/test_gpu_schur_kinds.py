"""GPU: the reduced matrix where the kinds of a destination block's pairs meet:
an observation with itself, a camera that sees a point twice, a camera with a
lens entry, a lens with itself and with another; sub-segments of one pair and
of more than 512.  Against the oracle's matrix: 1e-12 of the largest entry in
FP64, as in the other element-wise test; the FP32 form's factors and products
carry a few roundings of 2^-24 each (8 are allowed per pair's product, and they
add at most like the absolute values the matrix is made of)."""
import numpy as np
import pytest

import ba_oracle as O
import stitch_ba
from stitch_ba import Options, Problem, survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_cams,n_points,groups,twice", [
    (3, 3, 1, False), (4, 2400, 1, False), (9, 900, 1, True), (9, 900, 3, True), (6, 300, 2, False)])
def test_reduced_matrix(precision, n_cams, n_points, groups, twice):
    p, _ = survey.generate("lawnmower77", seed=n_cams + n_points, n_cams=n_cams, n_points=n_points)
    rep = np.ones(p.n_obs, int)
    if twice:
        rep[::7] = 2
    k = np.repeat(np.arange(p.n_obs), rep)
    uv = p.obs_uv[k]
    uv[1:][k[1:] == k[:-1]] += 0.25
    p = Problem(intr=np.repeat(p.intr, groups, 0), rot=p.rot, center=p.center,
                cam_group=np.arange(n_cams) % groups, points=p.points, obs_cam=p.obs_cam[k],
                obs_pt=p.obs_pt[k], obs_uv=uv, prior_mask=p.prior_mask, prior=p.prior)
    lam = 1e-2
    r = O.lm_step(p, lam, 4.0)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(lam, 4.0, Options(precision=precision, pcg_kernel="grid"))
    err = np.abs(d["S"] - r["S"])
    if precision == "fp64":
        assert err.max() <= 1e-12 * np.abs(r["S"]).max()
    else:
        # |S_ij| <= sqrt(U_ii U_jj), the undamped camera sums on the diagonal
        u = np.sqrt(np.abs(np.diag(r["S"])) * 4 + 1e-9)
        assert (err <= 1024 * 2.0**-24 * np.outer(u, u)).all(), (err / np.outer(u, u)).max() * 2.0**24
    # A point seen twice by a camera adds a product and its transpose, one after
    # the other: only without such pairs are the mirrored sums the same bits.
    if not twice:
        assert np.array_equal(d["S"], d["S"].T)
