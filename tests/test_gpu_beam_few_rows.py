"""Beams whose ring of input rows does not fit in shared memory whole: few rows
and many columns, both, a last chunk of one column, and so many rows that no
chunk's taps fit.  Such a beam's time goes with its taps, as that of the beams
whose ring fits.

Tolerance: inputs and taps are non-negative, so a voxel's error is at most the
number of FP32 roundings on its way times 2^-24 of its value: at most 40 in a
row's sum, one for each row of each chunk and the final scaling; one a tap
where the cube is read through the cache."""

import numpy as np
import pytest
from scipy.signal import fftconvolve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kshape,direct", [
    ((20, 30, 36), (5, 101), False), ((7, 230, 3), (1, 185), False), ((25, 60, 33), (9, 93), False),
    ((90, 100, 8), (83, 121), False), ((18, 300, 5), (3, 161), False),
    ((40, 50, 4), (401, 91), False), ((40, 120, 2), (1501, 101), True)])
def test_chunked_beams(shape, kshape, direct):
    import torch
    from martini_gb300.engine import InsertionEngine, convolve_beam
    rng = np.random.default_rng(11)
    cube = rng.random(shape).astype(np.float32)
    kern = rng.random(kshape).astype(np.float32).astype(np.float64)
    pad = tuple(min(k // 2, (n - 1) // 2) for k, n in zip(kshape, shape))
    eng = InsertionEngine("cuda:0")
    got = convolve_beam(eng, torch.from_numpy(cube).to(eng.device), pad[0], pad[1], kern,
                        1.5).cpu().numpy()
    full = np.stack([fftconvolve(cube[..., c].astype(np.float64), kern, mode="full")
                     for c in range(shape[2])], axis=2)
    i0, j0 = (kshape[0] - 1) // 2 + pad[0], (kshape[1] - 1) // 2 + pad[1]
    ref = full[i0:i0 + got.shape[0], j0:j0 + got.shape[1]] * 1.5
    chunks = -(-kshape[1] // 16)
    roundings = kshape[0] * kshape[1] + 1 if direct else kshape[0] * chunks + 41
    assert np.abs(got - ref).max() <= roundings * 2.0 ** -24 * ref.max() + 1e-12


def test_time_goes_with_the_taps():
    import torch
    from martini_gb300.engine import InsertionEngine, convolve_beam
    eng = InsertionEngine("cuda:0")
    us = []
    for ky in (51, 101):
        cube = torch.rand((260, 256 + ky - 1, 64), device=eng.device)
        kern = np.random.default_rng(ky).random((5, ky))
        t = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            convolve_beam(eng, cube, 2, ky // 2, kern, 1.0)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b) * 1e3)
        us.append(sorted(t)[6])
    assert us[1] <= 2.5 * us[0], us
