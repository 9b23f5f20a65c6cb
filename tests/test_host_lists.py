"""Sequence arguments of the plugin calls: host_f64's conversion equals NumPy's
for every form it takes, and raises what NumPy raises for the others."""

from __future__ import annotations

import numpy as np
import pytest

from blackhole_native import _device as dev


@pytest.mark.parametrize("x", [[], [1, 2.5, True], (np.float32(1.1), 3), [[1, 2], [3, 4]], ["1.5", "2"], [None, 1.0],
                               [np.array([1.0, 2.0]), np.array([3.0, 4.0])], [float("nan"), float("inf"), -0.0],
                               [10 ** 30], np.arange(3), range(3), 5.0])
def test_values(x):
    want = np.ascontiguousarray(np.asarray(x, dtype=np.float64).reshape(-1))
    got = dev.host_f64(x)
    assert got.dtype == np.float64 and got.shape == want.shape and got.tobytes() == want.tobytes()
    assert got.flags.writeable and got.flags.c_contiguous


@pytest.mark.parametrize("x", [["a"], [1j], [10 ** 400], [object()]])
def test_errors(x):
    with pytest.raises(Exception) as want:
        np.asarray(x, dtype=np.float64)
    with pytest.raises(want.type) as got:
        dev.host_f64(x)
    assert str(got.value) == str(want.value)
