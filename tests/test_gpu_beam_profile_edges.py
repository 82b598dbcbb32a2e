"""Sizes where the beam and the global-profile kernels can go wrong: one-tap and
one-pixel beams, tap counts off the kernel's groups of 8 and 4, channel counts
off its vectors and blocks, more rows than the ring holds, the widest beam of
the ring and one past it; bands of one channel, off the 31- and 32-channel
steps, and too wide for several or any of the warps' shared spectra.

Tolerances: all inputs are non-negative, so a voxel's error is at most the
number of FP32 roundings on its way times 2^-24 of its value (kx + ky for row
sums added to a total, kx ky for one running sum, and the final scaling); a
line value is the difference of two erfc values of at most 4 ulp each, within
1e-6 of the profile's peak."""

import numpy as np
import pytest
from scipy.signal import fftconvolve

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kshape,direct", [
    ((5, 4, 3), (1, 1), False), ((19, 23, 1), (3, 1), False), ((20, 18, 36), (1, 5), False),
    ((33, 40, 31), (9, 13), False), ((40, 61, 34), (11, 15), False), ((90, 34, 8), (73, 7), False),
    ((17, 100, 4), (3, 79), False), ((12, 110, 5), (5, 91), True)])
def test_beam_sizes(shape, kshape, direct):
    import torch
    from martini_gb300.engine import InsertionEngine, convolve_beam
    rng = np.random.default_rng(7)
    cube = rng.random(shape).astype(np.float32)
    kern = rng.random(kshape).astype(np.float32).astype(np.float64)
    pad = (kshape[0] // 2, kshape[1] // 2)
    pad = tuple(min(p, (n - 1) // 2) for p, n in zip(pad, shape))
    eng = InsertionEngine("cuda:0")
    got = convolve_beam(eng, torch.from_numpy(cube).to(eng.device), pad[0], pad[1], kern,
                        1.5).cpu().numpy()
    full = np.stack([fftconvolve(cube[..., c].astype(np.float64), kern, mode="full")
                     for c in range(shape[2])], axis=2)
    i0, j0 = (kshape[0] - 1) // 2 + pad[0], (kshape[1] - 1) // 2 + pad[1]
    ref = full[i0:i0 + got.shape[0], j0:j0 + got.shape[1]] * 1.5
    roundings = kshape[0] * kshape[1] + 1 if direct else kshape[0] + kshape[1] + 1
    assert np.abs(got - ref).max() <= roundings * 2.0 ** -24 * ref.max() + 1e-12


@pytest.mark.parametrize("n,nc", [(1, 1), (40, 31), (1025, 33), (5000, 1600), (700, 13000)])
@pytest.mark.parametrize("model", ["gaussian", "dirac"])
def test_profile_bands(n, nc, model):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine, global_profile
    rng = np.random.default_rng(n + nc)
    edges = orc.vrad_channel_edges(nc, 4.0, 100.0)
    half = max(2.0 * nc, 20.0)
    v = rng.uniform(100.0 - 1.1 * half, 100.0 + 1.1 * half, n)
    v[0] = 100.0
    sig = rng.uniform(2.0, 30.0, n).astype(np.float32)
    mhi = 10 ** rng.uniform(4, 6, n)
    ref = orc.init_spectra(model, mhi, np.full(n, 3.0), v, edges,
                           sig.astype(np.float64) if model == "gaussian" else None).sum(axis=0)
    eng = InsertionEngine("cuda:0")
    z = np.zeros(n)
    parts = DeviceParticles.from_host(eng.device, z, z, z, z, v=v, sigma=sig,
                                      amp=mhi / 9.0 / orc.MHI_TO_JY)
    m = N.MG_SPECTRUM_GAUSSIAN if model == "gaussian" else N.MG_SPECTRUM_DIRAC
    got = global_profile(eng, parts, m, 0.0, nc,
                         torch.from_numpy(edges).to(eng.device)).cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()
