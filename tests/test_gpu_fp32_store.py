"""FP32 form with lines from the spectrum store: the bits of the lines
evaluated inside the contraction (the same function), at chunk edges (31, 32,
33 particles on a tile), bands narrower and wider than a channel block, and
both line models; the package's bar against the oracle (1e-5 of peak)."""

import ctypes as C

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 3000])
@pytest.mark.parametrize("nc", [1, 64, 65, 200])
@pytest.mark.parametrize("model", ["gaussian", "dirac"])
def test_store_matches_in_kernel_lines(n, nc, model):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    lib = N.load()
    rng = np.random.default_rng(n + nc)
    nx, ny = (8, 16) if n < 100 else (37, 50)
    x, y = rng.uniform(-2, nx + 1, n), rng.uniform(-2, ny + 1, n)
    x[0], y[0] = nx / 2, ny / 2
    h = 10 ** rng.uniform(-0.6, 0.8, n)
    kernels = orc.adaptive_tuple("QuarticSplineKernel")
    kidx, size, resc = orc.select_kernels(kernels, h)
    r = orc.sm_ranges(h, size)
    edges = orc.vrad_channel_edges(nc, 4.0, 0.0)
    v = rng.uniform(-2.1 * nc, 2.1 * nc, n)
    sig = rng.uniform(4, 15, n).astype(np.float32)
    mhi = 10 ** rng.uniform(4, 5, n)
    spec = orc.init_spectra(model, mhi, np.full(n, 3.0), v, edges, sig.astype(np.float64))
    ref = orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h * resc, spec)
    eng = InsertionEngine("cuda:0")
    gauss = model == "gaussian"
    parts = DeviceParticles.from_host(eng.device, x, y, r, h * resc, kidx, v=v,
                                      sigma=sig if gauss else None, amp=mhi / 9.0 / orc.MHI_TO_JY)
    e = torch.from_numpy(edges).to(eng.device)
    table = [(N.MG_KERNEL_QUARTIC_SPLINE, 0.0), (N.MG_KERNEL_DIRAC, 0.0),
             (N.MG_KERNEL_GAUSSIAN, 6.0)]
    cube = torch.empty((nx, ny, nc), device=eng.device)
    prob = eng.problem(parts, table, N.MG_SPECTRUM_GAUSSIAN if gauss else N.MG_SPECTRUM_DIRAC, 0.0,
                       nx, ny, nc, 0, 0, e, cube, None, N.MG_FORM_FP32)
    info = eng.plan(prob)
    eng.run(prob)
    eng.check()
    stored = cube.clone()
    need = C.c_size_t()  # no room for the store
    N.check(lib.mg_workspace_size(C.byref(prob), info.n_pairs, info.n_partial_items,
                                  C.byref(need)))
    N.check(lib.mg_insert(C.byref(prob), C.c_void_p(eng._ws.data_ptr()), need.value, info.n_pairs,
                          info.n_partial_items, None))
    torch.cuda.synchronize()
    assert torch.equal(cube, stored)
    assert np.abs(stored.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
