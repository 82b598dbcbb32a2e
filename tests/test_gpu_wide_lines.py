"""Lines wider than a stage's 128-channel window over bands of several channel
blocks, whose stages are taken in parts, in every tensor-core form.

A channel of a wide line is the difference of two nearly equal error functions
in FP32, so the voxels' errors have a bound of their own: with each erfc value
off by 1.5e-7 of itself (the fitted form's 1.2e-7 and the rounding of its sum)
the line is off by 0.75e-7 (erfc|a| + erfc|b|) of its flux and by its three
roundings; the weights and the form's products add 5e-6 of the peak (half the
package's bar; 3.5e-5 with two BF16 pieces, 3 x 2^-18 a term).  Stages of 64 and
of 32 particles, and stored lines and lines evaluated in the contraction, take
the same lines through the same products in another order of accumulation:
within 1e-6 of the peak of each other, where a part that is dropped, doubled or
misplaced shows whatever the lines' errors."""

import ctypes as C

import numpy as np
import pytest
from scipy.special import erfc

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nc,sigma", [(200, 520, 90.0), (40, 513, 90.0), (900, 700, 150.0)])
@pytest.mark.parametrize("form", [1, 2, 3], ids=["bf16x3", "f16x3", "bf16x6"])
def test_lines_wider_than_a_window(n, nc, sigma, form):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    lib = N.load()
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
    amp = mhi / 9.0 / orc.MHI_TO_JY
    tail = erfc(np.abs(edges[None, :] - v[:, None]) / (np.sqrt(2.0) * sig[:, None]))
    off = amp[:, None] / np.abs(np.diff(edges)) * 0.75e-7 * (tail[:, :-1] + tail[:, 1:])
    bound = orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h * resc,
                               off + 3 * 2.0**-24 * spec)
    peak = ref.max()

    eng = InsertionEngine("cuda:0")
    parts = DeviceParticles.from_host(eng.device, x, y, r, h * resc, kidx, v=v, sigma=sig, amp=amp)
    e = torch.from_numpy(edges).to(eng.device)
    table = [(N.MG_KERNEL_WENDLAND_C2, 0.0), (N.MG_KERNEL_DIRAC, 0.0), (N.MG_KERNEL_GAUSSIAN, 6.0)]
    cube = torch.empty((nx, ny, nc), device=eng.device)
    flux = torch.empty(nc + 1, dtype=torch.float64, device=eng.device)
    prob = eng.problem(parts, table, N.MG_SPECTRUM_GAUSSIAN, 0.0, nx, ny, nc, 0, 0, e, cube, flux,
                       form)
    got = {}
    try:
        for kc in (0, 32):
            lib.mg_tuning_reset()
            info = eng.plan(prob)
            t = N.Tuning(kc, 6, 1, 0)
            assert lib.mg_tuning_store(C.byref(prob), 1, info.n_pairs, C.byref(t)) == N.MG_OK
            for stored in (True, False):
                cube.fill_(-1.0)
                if stored:
                    eng.run(prob)
                else:
                    eng.run_stages(prob, N.MG_STAGE_BIN)
                    eng.run_stages(prob, N.MG_STAGE_CONTRACT)
                    eng.run_stages(prob, N.MG_STAGE_FLUX)
                eng.check()
                got[kc, stored] = cube.cpu().numpy().astype(np.float64)
                if form != 1:
                    assert abs(flux[0].item() - ref.sum()) <= 1e-6 * ref.sum()
    finally:
        lib.mg_tuning_reset()
    for g in got.values():
        assert np.abs(g - got[0, True]).max() <= 1e-6 * peak
        assert (np.abs(g - ref) <= bound + (3.5e-5 if form == 1 else 5e-6) * peak).all()
