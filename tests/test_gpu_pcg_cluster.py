"""GPU: the cluster PCG kernel where what it keeps in shared memory changes:
all S blocks cached, rows whose blocks end between cached and turned ones,
mostly turned ones with ragged last runs, and two CTAs an SM with the models in
descending order.

The step is checked against the system it was computed from: the residual
S dx - g of a solve that stopped at |r|^2 < 1e-10 |b|^2 is 1e-5 |g| plus the
drift of the recurrence, at most one FP32 rounding of |S| |dx| per iteration
(400 iterations).  Where the blocks are read from changes no value: a batch
that runs two CTAs an SM gives each model the solve it has on its own, to the
run-to-run bounds of the other batch tests (cost 1e-12, positions 1e-9).
"""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options
from test_gpu_pcg_grid import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["cluster", "cluster_wide"])
@pytest.mark.parametrize("coarse", [False, True])
@pytest.mark.parametrize("n_cams,span,n_points", [
    (2, 2, 40),       # one CTA
    (60, 8, 900),     # all blocks cached
    (150, 34, 1500),  # rows of 67 blocks and the lens block
    (130, 90, 400),   # mostly turned, rows of up to 131 blocks
    (255, 120, 500),  # eight CTAs, row state and caches take most of the memory
])
def test_cluster_pcg_solves_its_system(kernel, coarse, n_cams, span, n_points):
    p = network(n_cams, span, n_points, 1, seed=n_cams + span)
    opt = Options(precision="mixed", pcg_kernel=kernel, coarse=coarse, pcg_tol=1e-10)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(1.0, 1.0, opt)
        again = ctx.debug_step(1.0, 1.0, opt)
    assert 0 < d["pcg_iters"] < 400
    assert np.array_equal(d["dx"], again["dx"])
    S, g, dx = d["S"], d["g"], d["dx"]
    drift = 400 * 2.0**-24 * np.linalg.norm(np.abs(S) @ np.abs(dx))
    assert np.linalg.norm(S @ dx - g) <= 1e-5 * np.linalg.norm(g) + drift


def test_batch_of_more_models_than_clusters():
    spans = [6 + (7 * m) % 41 for m in range(36)]
    probs = [network(130, sp, 300, 1, seed=m) for m, sp in enumerate(spans)]
    opt = Options(precision="mixed", coarse=True, pcg_kernel="cluster", pcg_max_iter=40)
    batch = [p.copy() for p in probs]
    infos = stitch_ba.bundle_adjust_batch(batch, 10, 1.0, opt)
    for m in (0, int(np.argmax(spans)), int(np.argmin(spans)), 35):
        r = probs[m].copy()
        _, si = stitch_ba.bundle_adjust(r, 10, 1.0, opt, return_info=True)
        assert infos[m].iterations == si.iterations
        assert abs(infos[m].final_cost - si.final_cost) <= 1e-12 * si.final_cost
        assert np.abs(batch[m].center - r.center).max() <= 1e-9
        assert np.abs(batch[m].points - r.points).max() <= 1e-9
