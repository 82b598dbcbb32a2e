"""FP32 form with Gaussian SPH kernels, whose row and column factors a warp
shares: particles on and off the tile and cube edges, kernels narrower than a
pixel and wider than the cube, against the oracle at the package's bar (1e-5
of peak, 1e-6 of flux)."""

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nx,ny", [(1, 8, 16), (33, 8, 16), (400, 41, 35)])
@pytest.mark.parametrize("trunc", [2.0, 3.0, 6.0])
@pytest.mark.parametrize("lo,hi", [(-0.3, 0.3), (0.3, 1.3)])
def test_gaussian_kernels(n, nx, ny, trunc, lo, hi):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    rng = np.random.default_rng(n + int(trunc))
    x, y = rng.uniform(-2, nx + 1, n), rng.uniform(-2, ny + 1, n)
    x[0], y[0] = 7.5, 15.5
    if n > 2:
        x[1], y[1] = 8.0, 16.0
    h = 10 ** rng.uniform(lo, hi, n)
    kernels = [orc.kernel_constants(orc.KT_GAUSSIAN, trunc)]
    kidx = np.zeros(n, dtype=int)
    r = np.ceil(h * trunc * 0.42466090014400953 + 1.0)
    nc = 12
    edges = orc.vrad_channel_edges(nc, 4.0, 0.0)
    v, sig = rng.uniform(-20, 20, n), rng.uniform(4, 9, n)
    mhi = 10 ** rng.uniform(4, 5, n)
    spec = orc.init_spectra("gaussian", mhi, np.full(n, 3.0), v, edges, sig)
    ref = orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h, spec)
    eng = InsertionEngine("cuda:0")
    parts = DeviceParticles.from_host(eng.device, x, y, r, h, kidx, v=v, sigma=sig,
                                      amp=mhi / 9.0 / orc.MHI_TO_JY)
    e = torch.from_numpy(edges).to(eng.device)
    cube, flux = eng.insert(parts, [(N.MG_KERNEL_GAUSSIAN, trunc)], N.MG_SPECTRUM_GAUSSIAN, 0.0, nx,
                            ny, nc, e, form=N.MG_FORM_FP32)
    got = cube.cpu().numpy().astype(np.float64)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    assert abs(flux[0].item() - ref.sum()) <= 1e-6 * ref.sum()
