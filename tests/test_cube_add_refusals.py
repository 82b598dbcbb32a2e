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
