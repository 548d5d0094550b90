"""GPU: cluster PCG in clusters of one CTA (models of up to 32 block rows),
whose blocks take the search direction from the row state: from the smallest
model to the one that fills the CTA, with and without a single lens row, both
thread counts, and the first model of two CTAs beside them.

The step is checked against the system it was computed from: the residual
S dx - g of a solve that stopped at |r|^2 < 1e-10 |b|^2 is 1e-5 |g| plus the
drift of the recurrence, at most one FP32 rounding of |S| |dx| per iteration
(400 iterations)."""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options
from test_gpu_pcg_grid import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["cluster", "cluster_wide"])
@pytest.mark.parametrize("coarse", [False, True])
@pytest.mark.parametrize("n_cams,span,groups,ctas", [
    (2, 2, 1, 1), (17, 5, 1, 1), (29, 9, 3, 1), (31, 31, 1, 1), (32, 8, 1, 2)])
def test_step_solves_its_system(kernel, coarse, n_cams, span, groups, ctas):
    p = network(n_cams, span, 40 * n_cams, groups, seed=n_cams)
    opt = Options(precision="mixed", pcg_kernel=kernel, coarse=coarse, pcg_tol=1e-10)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        assert ctx.solve(1, 1.0, opt)[0].pcg_ctas == ctas
        d = ctx.debug_step(1.0, 1.0, opt)
    assert 0 < d["pcg_iters"] < 400
    S, g, dx = d["S"], d["g"], d["dx"]
    drift = 400 * 2.0**-24 * np.linalg.norm(np.abs(S) @ np.abs(dx))
    assert np.linalg.norm(S @ dx - g) <= 1e-5 * np.linalg.norm(g) + drift
