"""The friends build's integer form of the circle cuts (build_friends_list.cl,
compute_scaling.cl: quotients of friend counts against 0.6f and 0.5f).  CPU."""
from __future__ import annotations

import numpy as np


def test_integer_form_of_the_circle_cuts():
    """5 p > 3 t and 2 p > t decide as the float quotients do, for every count."""
    p, t = np.meshgrid(np.arange(513), np.arange(513), indexing="ij")
    with np.errstate(invalid="ignore", divide="ignore"):
        q = p.astype(np.float32) / t.astype(np.float32)
    assert np.array_equal((q > np.float32(0.6))[p <= t], (5 * p > 3 * t)[p <= t])
    assert np.array_equal((q > np.float32(0.5))[p <= t], (2 * p > t)[p <= t])
