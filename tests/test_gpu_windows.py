"""Stage windows of the tensor-core contraction around its 128-channel working
accumulators and 256-channel blocks: bands at the block edges, lines wider than
a window, and segments with few particles of three kernel classes (whose stages
span the whole band), against the oracle at the package's bar (1e-5 of peak,
1e-6 of flux), for every stage size."""

import ctypes as C

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu

# A channel of a line of width s holds 1 / (s sqrt(2 pi)) of its flux as the
# difference of two FP32 erf values near 1: 2^-24 / 0.0044 = 1.35e-5 at s = 90
WIDE_LINES = pytest.mark.xfail(strict=False, reason="FP32 line evaluation: up to 1.35e-5 of a "
                               "channel's value for lines 90 channels wide, in every form")


@pytest.mark.parametrize("n,nc,sigma", [(60, 128, 4.0), (60, 130, 4.0), (300, 256, 4.0),
                                        (40, 256, 45.0), (900, 257, 20.0),
                                        pytest.param(200, 520, 90.0, marks=WIDE_LINES)])
@pytest.mark.parametrize("form", [1, 2, 3], ids=["bf16x3", "f16x3", "bf16x6"])
@pytest.mark.parametrize("kc", [0, 32])
def test_windows(n, nc, sigma, form, kc):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    lib = N.load()
    lib.mg_tuning_reset()
    rng = np.random.default_rng(n + nc)
    nx, ny = 21, 37
    x, y = rng.uniform(-2, nx + 1, n), rng.uniform(-2, ny + 1, n)
    h = 10 ** rng.uniform(-0.6, 0.9, n)
    kernels = orc.adaptive_tuple("WendlandC2Kernel")
    kidx, size, resc = orc.select_kernels(kernels, h)
    r = orc.sm_ranges(h, size)
    edges = orc.vrad_channel_edges(nc, 2.0, 0.0)
    v = rng.uniform(-1.05 * nc, 1.05 * nc, n)
    sig = (sigma * 10 ** rng.uniform(-0.3, 0.1, n)).astype(np.float32)
    mhi = 10 ** rng.uniform(4, 5, n)
    spec = orc.init_spectra("gaussian", mhi, np.full(n, 3.0), v, edges, sig.astype(np.float64))
    ref = orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h * resc, spec)
    eng = InsertionEngine("cuda:0")
    parts = DeviceParticles.from_host(eng.device, x, y, r, h * resc, kidx, v=v, sigma=sig,
                                      amp=mhi / 9.0 / orc.MHI_TO_JY)
    e = torch.from_numpy(edges).to(eng.device)
    table = [(N.MG_KERNEL_WENDLAND_C2, 0.0), (N.MG_KERNEL_DIRAC, 0.0), (N.MG_KERNEL_GAUSSIAN, 6.0)]
    cube = torch.empty((nx, ny, nc), device=eng.device)
    flux = torch.empty(nc + 1, dtype=torch.float64, device=eng.device)
    prob = eng.problem(parts, table, N.MG_SPECTRUM_GAUSSIAN, 0.0, nx, ny, nc, 0, 0, e, cube, flux,
                       form)
    info = eng.plan(prob)
    t = N.Tuning(kc, 6, 1, 0)
    assert lib.mg_tuning_store(C.byref(prob), 1, info.n_pairs, C.byref(t)) == N.MG_OK
    eng.run(prob)
    eng.check()
    lib.mg_tuning_reset()
    got = cube.cpu().numpy().astype(np.float64)
    tol = 1e-5 if form != 1 else 4e-5  # bf16x3: 3 x 2^-18 a term
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    if form != 1:
        assert abs(flux[0].item() - ref.sum()) <= 1e-6 * ref.sum()
