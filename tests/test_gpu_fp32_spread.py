"""The FP32 contraction with fewer work items than resident blocks: the items go
to different SMs, so 128 tiles of 1900 particles take about as long as one such
tile alone, and every item is taken once whatever their number (one, as many as
SMs, a few more, more than resident blocks)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PER = 1900  # one work item a tile (at least 2048 particles would make two)


def planned(nx, ny, per):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    nc = 64
    eng = InsertionEngine("cuda:0")
    tiles = [(i, j) for i in range(0, nx, 8) for j in range(0, ny, 16)]
    rng = np.random.default_rng(1)
    x = np.concatenate([i + rng.integers(0, 8, per) for i, _ in tiles]).astype(float)
    y = np.concatenate([j + rng.integers(0, 16, per) for _, j in tiles]).astype(float)
    n = len(x)
    one, amp = np.ones(n), rng.integers(1, 9, n).astype(float)
    parts = DeviceParticles.from_host(eng.device, x, y, one, one, None,
                                      v=rng.integers(0, nc, n) + 0.5, amp=amp)
    edges = torch.arange(nc + 1, device=eng.device, dtype=torch.float64)
    cube = torch.empty((nx, ny, nc), device=eng.device)
    flux = torch.empty(nc + 1, dtype=torch.float64, device=eng.device)
    prob = eng.problem(parts, [(N.MG_KERNEL_DIRAC, 0.0)], N.MG_SPECTRUM_DIRAC, 0.0, nx, ny, nc, 0,
                       0, edges, cube, flux, N.MG_FORM_FP32)
    assert eng.plan(prob).n_pairs == n
    want = np.zeros((nx, ny, nc))
    np.add.at(want, (x.astype(int), y.astype(int), parts.v.cpu().numpy().astype(int)), amp)
    return eng, prob, cube, want, parts, edges


@pytest.mark.parametrize("nx,ny,per", [(8, 16, 1900), (8, 16, 9000), (152 * 8, 16, 40),
                                       (153 * 8, 16, 40), (305 * 8, 16, 40), (460 * 8, 16, 40),
                                       (128, 128, 5000)])
def test_every_item_is_taken_once(nx, ny, per):
    # whole amplitudes: sums exact in FP32
    eng, prob, cube, want, *keep = planned(nx, ny, per)
    for _ in range(3):
        cube.fill_(-1.0)
        eng.run(prob)
        eng.check()
        np.testing.assert_array_equal(cube.cpu().numpy(), want)


def test_few_items_are_spread():
    import torch
    from martini_gb300 import _native as N
    us = []
    for nx, ny in ((8, 16), (128, 128)):
        eng, prob, *keep = planned(nx, ny, PER)
        eng.run(prob)
        t = []
        for _ in range(9):
            eng.run_stages(prob, N.MG_STAGE_BIN | N.MG_STAGE_SPEC)
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            eng.run_stages(prob, N.MG_STAGE_CONTRACT)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b) * 1e3)
        us.append(sorted(t)[4])
    # beside the item: the cube's clearing (4 MB) and the reduction's launch
    assert us[1] <= 1.25 * us[0] + 10.0, us
