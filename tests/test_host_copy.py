"""The pipelined precompute's staging copies: every value as is, writable or
read-only source, and no warning."""

from __future__ import annotations

import warnings

import numpy as np
import pytest

from blackhole_native import synchrotron as syn


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [0, 1, 77, 100_003])
@pytest.mark.parametrize("writable", [True, False])
def test_host_copy(dtype, n, writable):
    src = np.random.default_rng(n).standard_normal(n).astype(dtype)
    src[:3] = [np.nan, np.inf, -0.0][: min(n, 3)]
    src.flags.writeable = writable
    dst = np.full(n + 2, 7.0, dtype=dtype)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        syn._host_copy(dst[1:n + 1], src)
    assert dst[1:n + 1].tobytes() == src.tobytes()
    assert dst[0] == 7.0 and dst[-1] == 7.0
