"""mg_insert_planned: the run that continues from mg_plan's binning gives the
bits of a run that bins again (same records, counts and order), for every form
and for few and many particles, in accumulate mode and after a launch shape
was stored; a workspace without the problem's plan is reported, not used."""

import ctypes as C

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


def problem(eng, n, form, nc=40, accumulate=False, cube=None):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles
    rng = np.random.default_rng(n)
    nx, ny = 33, 50
    h = 10 ** rng.uniform(-0.6, 0.8, n)
    kernels = orc.adaptive_tuple("WendlandC2Kernel")
    kidx, size, resc = orc.select_kernels(kernels, h)
    edges = torch.from_numpy(orc.vrad_channel_edges(nc, 4.0, 0.0)).to(eng.device)
    parts = DeviceParticles.from_host(
        eng.device, rng.uniform(-4, nx + 4, n), rng.uniform(-4, ny + 4, n), orc.sm_ranges(h, size),
        h * resc, kidx, v=rng.uniform(-80, 80, n), sigma=rng.uniform(4, 9, n),
        amp=10 ** rng.uniform(0, 1, n))
    table = [(N.MG_KERNEL_WENDLAND_C2, 0.0), (N.MG_KERNEL_DIRAC, 0.0), (N.MG_KERNEL_GAUSSIAN, 6.0)]
    cube = torch.zeros((nx, ny, nc), device=eng.device) if cube is None else cube
    flux = torch.empty(nc + 1, dtype=torch.float64, device=eng.device)
    prob = eng.problem(parts, table, N.MG_SPECTRUM_GAUSSIAN, 0.0, nx, ny, nc, 0, 0, edges, cube,
                       flux, form, accumulate)
    return prob, cube, flux, (parts, edges)


@pytest.mark.parametrize("n", [1, 300, 40000])
@pytest.mark.parametrize("form", [0, 2, 3], ids=["fp32", "f16x3", "bf16x6"])
@pytest.mark.parametrize("accumulate", [False, True])
def test_same_bits(n, form, accumulate):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine
    lib = N.load()
    lib.mg_tuning_reset()
    eng = InsertionEngine("cuda:0")
    prob, cube, flux, keep = problem(eng, n, form, accumulate=accumulate)
    info = eng.plan(prob)
    t = N.Tuning(0, 2, 1, 0)  # other items per SM than the plan's
    assert lib.mg_tuning_store(C.byref(prob), 1, info.n_pairs, C.byref(t)) == N.MG_OK
    eng.run(prob)
    eng.check()
    want = cube.clone(), flux.clone()
    for _ in range(2):
        cube.zero_()
        eng.plan(prob)
        assert eng._binned
        eng._run_planned(prob)
        eng.check()
        assert torch.equal(cube, want[0]) and torch.equal(flux, want[1])
    lib.mg_tuning_reset()


def test_without_a_plan_is_reported():
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine
    eng = InsertionEngine("cuda:0")
    small, cube, flux, keep = problem(eng, 300, 3)
    large, cube2, flux2, keep2 = problem(eng, 40000, 3)
    eng.plan(large)
    eng.plan(small)  # the workspace is large enough for both and holds the small one's plan
    eng._run_planned(small)
    eng.check()
    eng._run_planned(small)  # the plan was used up
    with pytest.raises(N.MartiniGB300Error, match="no plan"):
        eng.check()
    eng.plan(small)
    eng._caps = (int(1e5), 100)
    eng._run_planned(large)  # another problem's plan
    with pytest.raises(N.MartiniGB300Error, match="no plan"):
        eng.check()
    eng.plan(small)
    eng.run(small)
    eng.check()
