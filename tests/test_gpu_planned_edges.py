"""mg_insert_planned after a plan that found the channel edges not monotonic:
the run reports them as mg_insert does, whatever the caller made of the plan's
return code, and the workspace serves the next problem."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 2, 3], ids=["fp32", "f16x3", "bf16x6"])
def test_edges_of_the_plan_stay_an_error(form):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    eng = InsertionEngine("cuda:0")
    rng = np.random.default_rng(form)
    n, nx, ny, nc = 200, 20, 24, 12
    h = rng.uniform(1.0, 4.0, n)
    parts = DeviceParticles.from_host(
        eng.device, rng.uniform(0, nx, n), rng.uniform(0, ny, n), np.ceil(h), h,
        v=rng.uniform(-20, 20, n), sigma=rng.uniform(4, 9, n), amp=rng.uniform(1, 2, n))
    good = torch.from_numpy(np.linspace(24.0, -24.0, nc + 1)).to(eng.device)
    bad = good.clone()
    bad[5] = bad[4]
    cube = torch.empty((nx, ny, nc), device=eng.device)
    flux = torch.empty(nc + 1, dtype=torch.float64, device=eng.device)

    def problem(edges):
        return eng.problem(parts, [(N.MG_KERNEL_WENDLAND_C2, 0.0)], N.MG_SPECTRUM_GAUSSIAN, 0.0,
                           nx, ny, nc, 0, 0, edges, cube, flux, form)

    eng.plan(problem(good))  # a workspace and capacities large enough
    prob, info, s = problem(bad), N.PlanInfo(), torch.cuda.current_stream(eng.device)
    args = C.c_void_p(eng._ws.data_ptr()), eng._ws.numel()
    stream = C.c_void_p(s.cuda_stream)
    assert eng.lib.mg_plan(C.byref(prob), *args, stream, C.byref(info)) == N.MG_ERR_NOT_MONOTONIC
    N.check(eng.lib.mg_insert_planned(C.byref(prob), *args, *eng._caps, stream))
    with pytest.raises(ValueError, match="monotonic"):
        eng.check()
    eng.plan(problem(good))
    eng._run_planned(problem(good))
    eng.check()
    assert cube.sum().item() > 0
