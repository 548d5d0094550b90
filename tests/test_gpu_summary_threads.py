"""GPU: summaries of different camera counts from several threads at once give
what each gives alone (the kernel's shared-memory limit is the process')."""
import threading

import numpy as np
import pytest

import stitch_ba
from stitch_ba import Problem

pytestmark = pytest.mark.gpu


def scene(nc, seed):
    rng = np.random.default_rng(seed)
    npts = 3 * nc
    cam = np.stack([(np.arange(npts) + k) % nc for k in range(3)], 1).reshape(-1)
    pt = np.repeat(np.arange(npts), 3)
    return Problem(intr=[[1000.0, 0, 0, 0, 0]], rot=np.tile(np.eye(3), (nc, 1, 1)),
                   center=rng.normal(0, 5, (nc, 3)), cam_group=np.zeros(nc),
                   points=rng.normal(0, 30, (npts, 3)), obs_cam=cam, obs_pt=pt,
                   obs_uv=np.zeros((len(cam), 2)))


def test_threads_of_different_sizes():
    probs = [scene(nc, nc) for nc in (4, 300, 2500, 9000, 20000, 24576)]
    alone = [stitch_ba.sparse_summary(p, agl=80.0) for p in probs]
    failed = []

    def work(p, want, calls):
        try:
            for _ in range(calls):
                got = stitch_ba.sparse_summary(p, agl=80.0)
                assert np.array_equal(got.neighbours, want.neighbours)
                assert np.array_equal(got.depth_range, want.depth_range)
        except Exception as e:  # noqa: BLE001 (reported by the test)
            failed.append(f"{p.n_cams} cameras: {e}")

    ts = [threading.Thread(target=work, args=(p, w, 400 if p.n_cams < 5000 else 30))
          for p, w in zip(probs, alone)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed
