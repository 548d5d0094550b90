"""GPU: every wait of the grid PCG's exchanges runs out in a test: partial sums
in a group whose CTAs all decide and in one that its last CTA leads, the
leader's result, and neighbours' z, in both storage precisions.

A held-back CTA never publishes (a test hook); with a wait limit of about 1 ms
every waiter gives up, sets the error flag and returns, and the call returns
TIMEOUT with the state untouched.  The next call on the device solves."""
import time

import numpy as np
import pytest

import stitch_ba
from stitch_ba import Options, native
from test_gpu_pcg_grid import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n_cams,ctas", [
    ("fp64", 60, (2, 32)),     # four rows a CTA: all decide
    ("fp64", 160, (33, 200)),  # led
    ("mixed", 60, (2, 32)),    # eight rows a CTA
    ("mixed", 300, (33, 200)),
])
@pytest.mark.parametrize("held", ["first", "second", "last"])
def test_every_wait_ends(precision, n_cams, ctas, held):
    p = network(n_cams, 6, 20 * n_cams, 1, seed=n_cams)
    form = dict(precision=precision, pcg_kernel="grid")
    ref = p.copy()
    _, info = stitch_ba.bundle_adjust(ref, 2, 1.0, Options(**form), return_info=True)
    assert ctas[0] <= info.pcg_ctas <= ctas[1]
    cta = {"first": 1, "second": 2, "last": info.pcg_ctas}[held]
    q = p.copy()
    t0 = time.perf_counter()
    with pytest.raises(stitch_ba.BaError) as e:
        stitch_ba.bundle_adjust(q, 10, 1.0, Options(wait_limit_cycles=2_000_000,
                                                    fault_hold_pcg_cta=cta, **form))
    assert e.value.status == native.TIMEOUT and "gave up waiting" in str(e.value)
    assert time.perf_counter() - t0 < 30.0
    for a, b in zip(p.state(), q.state()):
        assert np.array_equal(a, b)
    stitch_ba.bundle_adjust(q, 2, 1.0, Options(**form))
    assert np.array_equal(q.center, ref.center) and np.array_equal(q.points, ref.points)
