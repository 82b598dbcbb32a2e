"""The FP32 contraction's first items: large and small ones side by side on every
SM, so that 152 tiles of 1900 particles and 304 of 100 take little longer than the
large ones alone, and every item is taken once whatever their sizes and number
(152, 304 and 456 first places, one less and more, and a queue behind them)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def planned(counts):
    """One tile of 8 x 16 pixels after the other along axis 0, with counts[k] particles."""
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    nc, nx, ny = 64, 8 * len(counts), 16
    eng = InsertionEngine("cuda:0")
    rng = np.random.default_rng(1)
    tile = np.repeat(np.arange(len(counts)), counts)
    n = len(tile)
    x = (8 * tile + rng.integers(0, 8, n)).astype(float)
    y = rng.integers(0, 16, n).astype(float)
    v, amp = rng.integers(0, nc, n) + 0.5, rng.integers(1, 9, n).astype(float)
    order = rng.permutation(n)
    one = np.ones(n)
    parts = DeviceParticles.from_host(eng.device, x[order], y[order], one, one, None, v=v[order],
                                      amp=amp[order])
    edges = torch.arange(nc + 1, device=eng.device, dtype=torch.float64)
    cube = torch.empty((nx, ny, nc), device=eng.device)
    prob = eng.problem(parts, [(N.MG_KERNEL_DIRAC, 0.0)], N.MG_SPECTRUM_DIRAC, 0.0, nx, ny, nc, 0,
                       0, edges, cube, None, N.MG_FORM_FP32)
    assert eng.plan(prob).n_pairs == n
    want = np.zeros((nx, ny, nc), np.float32)
    np.add.at(want, (x.astype(int), y.astype(int), v.astype(int)), amp)
    return eng, prob, cube, want, parts, edges


@pytest.mark.parametrize("tiles", [1, 151, 152, 153, 303, 304, 305, 455, 456, 457, 700, 1500])
def test_every_item_is_taken_once(tiles):
    # whole amplitudes: sums exact in FP32
    counts = np.random.default_rng(tiles).integers(0, 300, tiles)
    counts[tiles // 2] = 9000  # split over several items
    eng, prob, cube, want, *keep = planned(counts)
    for _ in range(3):
        cube.fill_(-1.0)
        eng.run(prob)
        eng.check()
        np.testing.assert_array_equal(cube.cpu().numpy(), want)


def test_large_items_go_to_different_sms():
    import torch
    from martini_gb300 import _native as N
    us = []
    for counts in ([1900] * 152, [1900] * 152 + [100] * 304):
        eng, prob, *keep = planned(counts)
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
    # a tenth more pairs on every SM, the cube's clearing, three times the blocks
    assert us[1] <= 1.35 * us[0] + 10.0, us
