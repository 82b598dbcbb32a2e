"""The distribution passes behind the particle list, at the sizes where they
change shape: one particle, one tile of 8192 elements and one past it (a
single block, two tiles in one block, several blocks with a histogram), segment
counts of one (no digit bits), one pass and two, and particles off the cube
between particles on it.  The cube is compared with the oracle's scatter (the
package's bar, 1e-5 of peak and 1e-6 of flux) and two runs must give the same
bits, which needs the stable order."""

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nx,ny,nc", [
    (1, 8, 16, 4), (31, 8, 16, 20), (8192, 40, 33, 12), (8193, 24, 64, 40), (16385, 64, 48, 9),
    (25000, 100, 90, 140)])
@pytest.mark.parametrize("form", [0, 3], ids=["fp32", "bf16x6"])
def test_list_sizes(n, nx, ny, nc, form):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-6, nx + 5, n), rng.uniform(-6, ny + 5, n)
    x[0], y[0] = nx / 2, ny / 2
    h = 10 ** rng.uniform(-0.6, 0.5, n)
    kernels = orc.adaptive_tuple("WendlandC2Kernel")
    kidx, size, resc = orc.select_kernels(kernels, h)
    r = orc.sm_ranges(h, size)
    edges = orc.vrad_channel_edges(nc, 4.0, 0.0)
    v = rng.uniform(-2.2 * nc, 2.2 * nc, n)
    v[0] = 0.0
    sig = rng.uniform(3, 12, n)
    mhi = 10 ** rng.uniform(4, 5, n)
    spec = orc.init_spectra("gaussian", mhi, np.full(n, 3.0), v, edges, sig)
    ref = orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h * resc, spec)
    eng = InsertionEngine("cuda:0")
    parts = DeviceParticles.from_host(eng.device, x, y, r, h * resc, kidx, v=v, sigma=sig,
                                      amp=mhi / 9.0 / orc.MHI_TO_JY)
    e = torch.from_numpy(edges).to(eng.device)
    table = [(N.MG_KERNEL_WENDLAND_C2, 0.0), (N.MG_KERNEL_DIRAC, 0.0), (N.MG_KERNEL_GAUSSIAN, 6.0)]
    run = lambda: eng.insert(parts, table, N.MG_SPECTRUM_GAUSSIAN, 0.0, nx, ny, nc, e, form=form)
    cube, flux = run()
    again, _ = run()
    assert torch.equal(cube, again)
    got = cube.cpu().numpy().astype(np.float64)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    assert abs(flux[0].item() - ref.sum()) <= 1e-6 * ref.sum()
