"""The bins by which the cuts of top-k and top-p are searched (on the host: the function is the kernel's own)."""
import ctypes as C

import numpy as np
import pytest

from spite_b200.kernels import build


@pytest.mark.parametrize("lo,scale", [(0.0, 128.0), (0.0, 8.0), (3.25, 2.0**17), (5.0, 2.0**27), (10.0, 2.0**27), (200.0, 2.0**37), (0.5, 2.0**20)])
def test_bins_never_fall(lo, scale):
    """From the row's maximum downwards a logit's bin never falls; below 0 for what lies above the bins, however far."""
    lib = build.load("sampling")
    steps = (np.arange(-4000, 6000) / 2).astype(np.float64) / scale + lo
    d = np.concatenate([np.linspace(0, 2 * lo + 4, 20001), steps[steps >= 0], [0.0, 1e30, np.inf]]).astype(np.float32)
    d.sort()
    bins = np.empty(d.size, np.int32)
    assert lib.spite_sample_bins(d.ctypes.data_as(C.c_void_p), d.size, C.c_float(lo), C.c_float(scale), bins.ctypes.data_as(C.c_void_p)) == 0
    assert (np.diff(bins.astype(np.int64)) >= 0).all()
    exact = (d.astype(np.float64) - lo) * scale
    assert (bins[exact < -0.5] < 0).all() and (bins[exact > 2048] >= 2048).all()
    within = (exact >= 0) & (exact < 2047)
    assert (np.abs(bins[within] - exact[within]) <= 0.5).all()
