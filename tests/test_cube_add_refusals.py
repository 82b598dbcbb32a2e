"""What the native pass into the host cube refuses and accepts, as the array
operations `array += add` and `array /= px2` did: arrays of another shape
raise before anything is written (CPU only)."""

import numpy as np
import pytest

from martini_gb300.martini import add_to_array


@pytest.mark.parametrize("divide_all", [True, False])
@pytest.mark.parametrize("shape,add", [((4, 5, 3), (4, 5, 2)), ((4, 5, 3), (4, 4, 3)),
                                       ((4, 5, 3), (5, 4, 3)), ((4, 5, 3, 1), (4, 5, 2)),
                                       ((4, 5, 3, 2), (4, 5, 3)), ((4, 5), (4, 5, 3)),
                                       ((3, 5, 3), (4, 5, 3)), ((60,), (4, 5, 3))])
def test_another_shape_is_refused(shape, add, divide_all):
    arr = np.ones(shape)
    with pytest.raises(ValueError, match="shape"):
        add_to_array(arr, np.ones(add, np.float32), (0, 0), 2.0, divide_all)
    assert np.all(arr == 1.0)


@pytest.mark.parametrize("divide_all", [True, False])
@pytest.mark.parametrize("dtype", ["f4", ">f8", "c16", "g"])
def test_other_types_as_the_array_operations(dtype, divide_all):
    rng = np.random.default_rng(1)
    add = rng.uniform(0, 1, (6, 7, 5)).astype(np.float32)
    arr = rng.uniform(0, 1, (6, 7, 5, 1)).astype(dtype)
    if dtype == "c16":
        arr += 1j
    if dtype == "g":
        arr += np.longdouble(2) ** -60  # lost in FP64
    want = arr.copy()
    if divide_all:
        want += add.astype(np.float64)[..., np.newaxis]
        want /= 3.7
    else:
        want += add.astype(np.float64)[..., np.newaxis] / 3.7
    got = add_to_array(arr, add, (1, 2), 3.7, divide_all)
    assert arr.dtype == np.dtype(dtype) and np.array_equal(arr, want)
    inner = (want[1:-1, 2:-2] * 3.7).sum(axis=(0, 1)).reshape(-1)
    assert np.array_equal(got, inner)


@pytest.mark.parametrize("divide_all", [True, False])
@pytest.mark.parametrize("dtype", [np.int64, np.uint8, bool])
def test_types_that_hold_no_fractions_are_refused(dtype, divide_all):
    arr = np.ones((4, 5, 3), dtype)
    with pytest.raises(TypeError):
        add_to_array(arr, np.full((4, 5, 3), 0.5, np.float32), (0, 0), 2.0, divide_all)
    assert np.all(arr == 1)


def test_the_native_pass_gets_aligned_arrays(monkeypatch):
    from martini_gb300 import martini as m
    lib = m.N.load()
    seen = []

    class Lib:
        @staticmethod
        def mg_cube_add(array, add, *rest):
            seen.append((array % 8, add % 4))
            return lib.mg_cube_add(array, add, *rest)

    monkeypatch.setattr(m.N, "load", lambda: Lib)
    shape, n = (3, 4, 5), 60
    arr = np.frombuffer(bytearray(n * 8 + 4), dtype=np.float64, offset=4, count=n).reshape(shape)
    add = np.frombuffer(bytearray(n * 4 + 1), dtype=np.float32, offset=1, count=n).reshape(shape)
    add[...] = 0.5
    assert not arr.flags.aligned and not add.flags.aligned
    add_to_array(arr, add, (0, 0), 2.0, True)
    assert seen == [(0, 0)] and np.all(arr == 0.25)
