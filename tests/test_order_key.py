"""Host restatement of the integer keys that stand for FP64 comparisons in the
records kernel (`order_key`, and the tests of a range's sign and of a
coordinate's size, csrc/mg_internal.cuh and mg_bin.cu): every comparison of
the values over zeros, denormals, neighbours, infinities and NaN (CPU only)."""

import numpy as np
import pytest

INF = 0x7FF0000000000000
TINY = np.nextafter(0.0, 1.0)
VALUES = np.array([0.0, -0.0, TINY, -TINY, 1.0, -1.0, np.nextafter(1.0, 2.0), 1e300, -1e300,
                   2.0**30, -2.0**30, np.nextafter(2.0**30, 0), np.inf, -np.inf])


def bits(v):
    return int(np.float64(v).view(np.int64))


def order_key(v):
    b = bits(v)
    return b if b >= 0 else (0 if b == -(1 << 63) else -(1 << 63) - b)


def test_keys_order_as_the_values():
    rng = np.random.default_rng(0)
    v = np.concatenate((VALUES, rng.normal(0, 1e3, 200), -np.abs(rng.normal(0, 1e-300, 20))))
    for a in v:
        for b in v:
            assert (order_key(a) >= order_key(b)) == (a >= b)
            assert (order_key(a) > order_key(b)) == (a > b)


@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_a_nan_bound_gives_an_empty_range(nan):
    # first c with E >= NaN and first c with E > NaN, then [first, last]
    k, edges = order_key(nan), [order_key(e) for e in np.linspace(-5, 5, 11)]
    first = next((c for c in range(10) if edges[c + 1] >= k), 10)
    last = next((c for c in range(10) if edges[c] > k), 10) - 1
    assert first > last


def test_range_and_coordinate_tests():
    for r in np.concatenate((VALUES, [np.nan, -np.nan])):
        rb = bits(r)
        empty = rb > INF or (rb < 0 and rb != -(1 << 63))
        assert empty == (not r >= 0.0)
        assert (rb == INF) == bool(np.isinf(r) and r > 0)
        hi = (rb >> 32) & 0x7FFFFFFF
        assert (hi < 0x41D00000) == bool(np.isfinite(r) and abs(r) < 2.0**30)
