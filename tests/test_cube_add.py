"""The native pass that adds an inserted cube to the host array (CPU only):
the same bits as the whole-array operations, sums to the rounding of an FP64
sum of n terms (n 2^-53 at the most, of non-negative terms), for one thread
and several, pads, a Stokes axis, a cropped view and a read-only array."""

import numpy as np
import pytest

from martini_gb300.martini import add_to_array


@pytest.mark.parametrize("shape,pads", [((1, 1, 1), (0, 0)), ((5, 7, 3), (1, 2)),
                                        ((9, 31, 17), (0, 0)), ((70, 65, 130), (3, 4)),
                                        ((4, 4, 5), (2, 1))])
@pytest.mark.parametrize("divide_all", [True, False])
@pytest.mark.parametrize("layout", ["plain", "stokes", "view"])
def test_matches_array_operations(shape, pads, divide_all, layout):
    rng = np.random.default_rng(shape[0])
    add = rng.uniform(0, 1, shape).astype(np.float32)
    prior = rng.uniform(0, 1, shape)
    px2 = 10.3**2
    want = (prior + add) / px2 if divide_all else prior + add.astype(np.float64) / px2
    if layout == "stokes":
        arr = prior[..., np.newaxis].copy()
    elif layout == "view":
        arr = np.pad(prior, ((1, 1), (2, 2), (0, 0)))[1:-1, 2:-2]
    else:
        arr = prior.copy()
    got = add_to_array(arr, add, pads, px2, divide_all)
    assert np.array_equal(arr.reshape(shape), want)
    inner = want[pads[0]:shape[0] - pads[0], pads[1]:shape[1] - pads[1]] * px2
    n = max(inner.shape[0] * inner.shape[1], 1)
    np.testing.assert_allclose(got, inner.sum(axis=(0, 1)), rtol=2 * n * 2.0**-53, atol=0)


def test_read_only_array_is_refused():
    arr = np.zeros((2, 2, 2))
    arr.flags.writeable = False
    with pytest.raises(ValueError):
        add_to_array(arr, np.ones((2, 2, 2), np.float32), (0, 0), 1.0, True)
