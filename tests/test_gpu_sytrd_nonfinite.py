"""NaN and Inf through the reduction's exchange, whose empty slots hold a NaN pattern (all ones).

An input entry with that very pattern must not look like a slot that has not arrived: the call ends, reports no failed
wait and returns NaN, and the next call is right.  A wait on such a slot would end by its time limit with an error.
"""
import numpy as np
import pytest

from oracle import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [40, 70, 130, 300, 700])
@pytest.mark.parametrize("value", ["nan", "ones", "inf"])
def test_ends_and_returns_nan(xe, n, value, dtype):
    a = inputs.random_symmetric(n, seed=61 + n).astype(dtype)
    ref = xe.sytrd_upper(a, dtype)
    assert all(np.all(np.isfinite(x)) for x in ref[1:])
    bits = {8: np.uint64, 4: np.uint32}[a.dtype.itemsize]
    bad = np.array([{"nan": np.nan, "ones": 0, "inf": -np.inf}[value]], dtype)
    if value == "ones":
        bad.view(bits)[0] = np.iinfo(bits).max
    old = xe.get_option("wait_limit_ms")
    xe.set_option("wait_limit_ms", 2000)
    try:
        for i, j in ((0, 0), (0, n - 1), (n // 2, n // 2 + 1), (n - 2, n - 1), (n - 2, n - 2)):
            b = np.array(a, order="F", copy=True)
            b.view(bits)[i, j] = b.view(bits)[j, i] = bad.view(bits)[0]
            _, d, e, _ = xe.sytrd_upper(b, dtype)  # raises on a failed wait
            assert not np.all(np.isfinite(np.concatenate([d, e])))
    finally:
        xe.set_option("wait_limit_ms", old)
    for x, y in zip(ref, xe.sytrd_upper(a, dtype)):
        assert np.array_equal(x, y)
