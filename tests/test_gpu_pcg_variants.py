"""GPU: the shapes of the PCG tests run the kernel variants they are meant for
(the names of the launched kernels, by the CUDA profiler of torch): the FP64
grid kernel's two-lane form up to 16 blocks a row, two CTAs of the cluster
kernel an SM where models outnumber the clusters; and a model whose blocks are
more than the cache slots that a CTA's shared memory holds."""
import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options
from test_gpu_pcg_grid import network

pytestmark = pytest.mark.gpu


def kernels_of(run):
    """Names of the kernels that run() launches."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    names = set()
    for _ in range(2):  # (a process' first session may start too late for its kernels)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            run()
            torch.cuda.synchronize()
        names = {e.key for e in prof.key_averages()}
    if not any("kernel" in n for n in names):
        pytest.skip("the CUDA profiler records no kernels here")
    return names


def pcg_kernels(run):
    names = kernels_of(run)
    return {n.split("(")[0].split("::")[-1] for n in names if "pcg" in n and "kernel" in n}


@pytest.mark.parametrize("n_cams,span,name", [
    (12, 5, "pcg_kernel<double, true>"),
    (40, 8, "pcg_kernel<double, true>"),    # rows of 16 blocks with the lens block
    (40, 9, "pcg_kernel<double, false>"),   # of 18
])
def test_grid_variants(n_cams, span, name):
    p = network(n_cams, span, 500, 1, seed=n_cams + span)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        run = lambda: ctx.debug_step(1.0, 1.0, Options(pcg_kernel="grid"), dense=False)
        assert pcg_kernels(run) == {name}


@pytest.mark.parametrize("models,name", [(36, "pcg_cluster_kernel<true, 512, 2>"),
                                         (4, "pcg_cluster_kernel<true, 512, 1>")])
def test_cluster_variants(models, name):
    """The batch of test_gpu_pcg_cluster, and a small one."""
    probs = [network(130, 6 + (7 * m) % 41, 300, 1, seed=m) for m in range(models)]
    opt = Options(precision="mixed", coarse=True, pcg_kernel="cluster", pcg_max_iter=40,
                  graph=False)
    run = lambda: stitch_ba.bundle_adjust_batch([p.copy() for p in probs], 2, 1.0, opt)
    assert pcg_kernels(run) == {name}


def test_more_blocks_than_slots():
    """1250 cameras that all share points: 79 rows of 1251 blocks in a CTA, whose
    slots alone (two bytes a block, 198 KB) leave no room for what it must hold.
    Checked as the other systems: the residual of the step is 1e-5 |g| plus the
    drift of the recurrence, one FP32 rounding of |S| |dx| an iteration."""
    p = network(1250, 1250, 12, 1, seed=5)
    p.center[:, 0] *= 0.02                     # a stack of photos over the points
    opt = Options(precision="mixed", pcg_kernel="cluster", pcg_tol=1e-10)
    with stitch_ba.Context() as ctx:
        ctx.upload(p)
        d = ctx.debug_step(1.0, 1.0, opt)
    assert 0 < d["pcg_iters"] < 400
    S, g, dx = d["S"], d["g"], d["dx"]
    drift = 400 * 2.0**-24 * np.linalg.norm(np.abs(S) @ np.abs(dx))
    assert np.linalg.norm(S @ dx - g) <= 1e-5 * np.linalg.norm(g) + drift
