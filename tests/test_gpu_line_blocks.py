"""The three-piece form's channel blocks on cubes with few segments: 128 wide below
304 segments of 256 channels and 500 particles for each.  Lines against the oracle's
scatter at the package's bar (1e-5 of peak and 1e-6 of flux) on both sides of
each; the same particles among others that miss the cube, which changes the
blocks and nothing else, to 2e-6 of the peak (each side's product and line terms
against FP64 are below 1e-6); one workspace size for every spectral model; and
the narrow blocks faster than the wide ones for wide lines."""

import ctypes as C

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


def lines(eng, n, nx, ny, nc, off, sigma, seed, spectra=False, h_dex=(-0.4, 0.4)):
    """n particles on the cube and `off` beside it."""
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-2, nx + 1, n), rng.uniform(-2, ny + 1, n)
    h = 10 ** rng.uniform(*h_dex, n)
    kernels = orc.adaptive_tuple("WendlandC2Kernel")
    kidx, size, resc = orc.select_kernels(kernels, h)
    r = orc.sm_ranges(h, size)
    v, sig = rng.uniform(-2.0 * nc, 2.0 * nc, n), rng.uniform(*sigma, n).astype(np.float32)
    mhi = 10 ** rng.uniform(4, 5, n)
    edges = orc.vrad_channel_edges(nc, 4.0, 0.0)
    pad = lambda a, value: np.concatenate([a, np.full(off, value, dtype=np.asarray(a).dtype)])
    table = rng.random((n + off, nc), dtype=np.float32) if spectra else None
    parts = DeviceParticles.from_host(
        eng.device, pad(x, 1e5), pad(y, 1e5), pad(r, 1.0), pad(h * resc, 1.0), pad(kidx, 0),
        v=pad(v, 0.0), sigma=pad(sig, 5.0), amp=pad(mhi / 9.0 / orc.MHI_TO_JY, 1.0), spectra=table)
    e = torch.from_numpy(edges).to(eng.device)
    cube = torch.empty((nx, ny, nc), device=eng.device)
    flux = torch.empty(nc + 1, dtype=torch.float64, device=eng.device)
    kt = [(N.MG_KERNEL_WENDLAND_C2, 0.0), (N.MG_KERNEL_DIRAC, 0.0), (N.MG_KERNEL_GAUSSIAN, 6.0)]
    prob = eng.problem(parts, kt, N.MG_SPECTRUM_TABLE if spectra else N.MG_SPECTRUM_GAUSSIAN, 0.0,
                       nx, ny, nc, 0, 0, e, cube, flux, N.MG_FORM_BF16X6)

    def ref():
        spec = orc.init_spectra("gaussian", mhi, np.full(n, 3.0), v, edges, sig.astype(np.float64))
        return orc.insert_scatter(nx, ny, x, y, r, kernels, kidx, h * resc, spec)
    return prob, cube, flux, ref, (parts, e)


@pytest.mark.parametrize("nx,ny,nc,off", [
    (13, 9, 363, 0), (30, 40, 300, 0), (30, 40, 300, 20000), (40, 30, 257, 0), (160, 240, 256, 0),  # 300, 304 segments
    (152, 256, 256, 0), (152, 250, 260, 0), (17, 40, 129, 0)])
def test_lines_against_the_oracle(nx, ny, nc, off):
    from martini_gb300.engine import InsertionEngine
    eng = InsertionEngine("cuda:0")
    prob, cube, flux, ref, keep = lines(eng, 2000, nx, ny, nc, off, (4.0, 60.0), nx + nc)
    eng.plan(prob)
    eng.run(prob)
    eng.check()
    want, got = ref(), cube.cpu().numpy().astype(np.float64)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    assert abs(flux[0].item() - want.sum()) <= 1e-6 * want.sum()


@pytest.mark.parametrize("nx,ny,nc,sigma", [(24, 17, 300, (3.0, 8.0)), (11, 40, 700, (20.0, 60.0))])
def test_particles_beside_the_cube_change_the_blocks_only(nx, ny, nc, sigma):
    from martini_gb300.engine import InsertionEngine
    eng = InsertionEngine("cuda:0")
    cubes, plans = [], []
    most = 500 * -(-nx // 8) * -(-ny // 16) * -(-nc // 256)
    for off in (0, most - 4001, most - 4000):
        prob, cube, flux, _, keep = lines(eng, 4000, nx, ny, nc, off, sigma, 3)
        plans.append(eng.plan(prob).n_pairs)
        eng.run(prob)
        eng.check()
        cubes.append(cube.clone())
    assert (cubes[0] == cubes[1]).all() and plans[0] == plans[1] > plans[2]
    assert (cubes[0] - cubes[2]).abs().max() <= 2e-6 * cubes[0].max()


@pytest.mark.parametrize("n", [2999, 3000, 100000])  # 6 segments
def test_a_size_serves_every_model(n):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine
    eng = InsertionEngine("cuda:0")
    prob, cube, flux, _, keep = lines(eng, n, 20, 30, 140, 0, (4.0, 60.0), 5, spectra=True)
    pairs = int(eng.plan(prob).n_pairs) + 10
    partials = int(eng.last_plan.n_partial_items)
    eng.run(prob)
    eng.check()
    want = cube.clone()
    size = C.c_size_t()
    sizes = []
    for model in (N.MG_SPECTRUM_GAUSSIAN, N.MG_SPECTRUM_DIRAC, N.MG_SPECTRUM_TABLE):
        prob.spectral_model = model
        N.check(eng.lib.mg_workspace_size(C.byref(prob), pairs, partials, C.byref(size)))
        sizes.append(size.value)
    assert len(set(sizes)) == 1
    ws = torch.empty(sizes[0], dtype=torch.uint8, device=eng.device)
    s = C.c_void_p(torch.cuda.current_stream(eng.device).cuda_stream)
    N.check(eng.lib.mg_insert(C.byref(prob), C.c_void_p(ws.data_ptr()), ws.numel(), pairs, partials,
                              s))
    N.check(eng.lib.mg_check(C.c_void_p(ws.data_ptr()), s))
    assert torch.equal(cube, want)


@pytest.mark.parametrize("n,nx,ny,nc", [(20000, 60, 60, 300), (30000, 64, 64, 300)])
def test_narrow_blocks_faster_than_wide_ones(n, nx, ny, nc):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine
    eng = InsertionEngine("cuda:0")
    us = []
    for off in (0, 500 * -(-nx // 8) * -(-ny // 16) * -(-nc // 256) - n):
        prob, *keep = lines(eng, n, nx, ny, nc, off, (20.0, 40.0), 9, h_dex=(0.3, 0.6))
        eng.plan(prob)
        eng.run(prob)
        t = []
        for _ in range(15):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            eng.run_stages(prob, N.MG_STAGE_CONTRACT)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b) * 1e3)
        us.append(sorted(t)[7])
    assert us[0] <= 0.85 * us[1], us  # 0.64 and 0.59 measured
