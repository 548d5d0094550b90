"""CPU: a pair check of more pairs than a launch has CTAs is refused as bad
input, before anything is copied (no array is read, no GPU is needed)."""
import ctypes

import numpy as np
import pytest

from stitch_ba import native


@pytest.mark.parametrize("n_pairs", [1 << 31, (1 << 32) + 7, 1 << 40])
def test_too_many_pairs_are_refused(n_pairs):
    L = native.load()
    ptr, med = np.zeros(1, np.uint32), np.zeros(1)
    m = native.BaPairMatches(n_pairs, 0, ptr.ctypes.data, ptr.ctypes.data, None, None)
    st = L.ba_pair_fits(ctypes.byref(m), None, None, None, None, 0, 0, None, med.ctypes.data)
    assert st == native.BAD_INPUT and b"too many pairs" in L.ba_last_error()
