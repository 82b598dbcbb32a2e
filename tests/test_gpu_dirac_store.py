"""Dirac lines from the spectrum store: the bits of the lines evaluated inside
the contraction (the same product per channel), with velocities on channel
edges (two channels), outside the band and ascending or descending edges,
and the package's bar against the oracle (1e-5 of peak; bf16x3 4e-5)."""

import ctypes as C

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40, 5000])
@pytest.mark.parametrize("form", [1, 2, 3], ids=["bf16x3", "f16x3", "bf16x6"])
@pytest.mark.parametrize("flip", [False, True])
def test_store_matches_in_kernel_lines(n, form, flip):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    lib = N.load()
    rng = np.random.default_rng(n)
    nx, ny, nc = 30, 41, 300
    x, y = rng.uniform(-3, nx + 2, n), rng.uniform(-3, ny + 2, n)
    x[0], y[0] = nx / 3, ny / 3
    h = 10 ** rng.uniform(-0.6, 0.8, n)
    kernels = orc.adaptive_tuple("WendlandC2Kernel")
    kidx, size, resc = orc.select_kernels(kernels, h)
    r = orc.sm_ranges(h, size)
    edges = orc.vrad_channel_edges(nc, 4.0, 0.0)
    edges = edges[::-1].copy() if flip else edges
    v = rng.uniform(-2.1 * nc, 2.1 * nc, n)
    v[::7] = edges[rng.integers(0, nc + 1, len(v[::7]))]
    mhi = 10 ** rng.uniform(4, 5, n)
    spec = orc.init_spectra("dirac", mhi, np.full(n, 3.0), v, edges, None)
    ref = orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h * resc, spec)
    eng = InsertionEngine("cuda:0")
    parts = DeviceParticles.from_host(eng.device, x, y, r, h * resc, kidx, v=v,
                                      amp=mhi / 9.0 / orc.MHI_TO_JY)
    e = torch.from_numpy(edges).to(eng.device)
    table = [(N.MG_KERNEL_WENDLAND_C2, 0.0), (N.MG_KERNEL_DIRAC, 0.0), (N.MG_KERNEL_GAUSSIAN, 6.0)]
    cube = torch.empty((nx, ny, nc), device=eng.device)
    prob = eng.problem(parts, table, N.MG_SPECTRUM_DIRAC, 0.0, nx, ny, nc, 0, 0, e, cube, None, form)
    info = eng.plan(prob)
    eng.run(prob)
    eng.check()
    stored = cube.clone()
    need = C.c_size_t()  # no room for the store
    N.check(lib.mg_workspace_size(C.byref(prob), info.n_pairs, info.n_partial_items,
                                  C.byref(need)))
    assert info.workspace_bytes > need.value
    N.check(lib.mg_insert(C.byref(prob), C.c_void_p(eng._ws.data_ptr()), need.value, info.n_pairs,
                          info.n_partial_items, None))
    torch.cuda.synchronize()
    assert torch.equal(cube, stored)
    tol = 4e-5 if form == 1 else 1e-5
    assert np.abs(stored.cpu().numpy() - ref).max() <= tol * np.abs(ref).max()
