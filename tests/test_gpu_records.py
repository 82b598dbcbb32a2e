"""The compiled records kernel against the host restatements of its shortcuts:
the plan's pair count equals the count of tiles that `reach2` and `row_tiles`
list (tests/test_tile_cull.py), and Dirac lines at, beside and between channel
edges land in the channels whose closed interval holds them by FP64 comparison
(the integer keys of tests/test_order_key.py), for rising and falling edges
through zero, both zeros and a denormal."""

import numpy as np
import pytest

from tests.test_tile_cull import reach2, row_tiles

pytestmark = pytest.mark.gpu

f32 = np.float32


@pytest.mark.parametrize("kernel,trunc", [(0, 0.0), (2, 0.0), (4, 3.0), (4, 6.0)],
                         ids=["c2", "cubic", "gaussian3", "gaussian6"])
@pytest.mark.parametrize("lo,hi", [(0.3, 4.0), (4.0, 60.0)])
def test_the_plan_counts_the_tiles_of_the_circle(kernel, trunc, lo, hi):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    n, nx, ny, nc = 1500, 203, 301, 8
    rng = np.random.default_rng(int(hi))
    rad = rng.uniform(lo, hi, n)
    h = rad / (trunc * 0.42466090014400953 if trunc else 1.0)
    x, y = rng.uniform(-hi, nx + hi, n), rng.uniform(-hi, ny + hi, n)
    near = rng.random(n) < 0.3
    x[near], y[near] = np.round(x[near]) + rng.choice([0, 1e-9, -1e-9, 0.5], near.sum()), \
        np.round(y[near])
    r = np.ceil(rad)
    want = 0
    for k in range(n):
        ilo, ihi = max(int(np.ceil(x[k] - r[k])), 0), min(int(np.floor(x[k] + r[k])), nx - 1)
        jlo, jhi = max(int(np.ceil(y[k] - r[k])), 0), min(int(np.floor(y[k] + r[k])), ny - 1)
        if ilo > ihi or jlo > jhi:
            continue
        rk = f32(h[k]) if not trunc else f32(f32(trunc) * f32(f32(h[k]) * f32(0.42466090014400953)))
        for tx in range(ilo // 8, ihi // 8 + 1):
            t0, t1 = row_tiles(x[k], y[k], (ilo, ihi, jlo, jhi), reach2(rk), tx)
            want += t1 - t0 + 1
    eng = InsertionEngine("cuda:0")
    parts = DeviceParticles.from_host(eng.device, x, y, r, h, None, v=np.zeros(n),
                                      sigma=np.full(n, 3.0), amp=np.ones(n))
    e = torch.from_numpy(np.linspace(16.0, -16.0, nc + 1)).to(eng.device)
    cube = torch.empty((nx, ny, nc), device=eng.device)
    prob = eng.problem(parts, [(kernel, trunc)], N.MG_SPECTRUM_GAUSSIAN, 0.0, nx, ny, nc, 0, 0, e,
                       cube, None, N.MG_FORM_BF16X6)
    assert eng.plan(prob).n_pairs == want


@pytest.mark.parametrize("order", [1, -1], ids=["rising", "falling"])
@pytest.mark.parametrize("form", [0, 3], ids=["fp32", "bf16x6"])
def test_dirac_lines_around_the_edges(order, form):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import DeviceParticles, InsertionEngine, global_profile
    rng = np.random.default_rng(2)
    edges = np.unique(np.concatenate((rng.uniform(-60, 60, 20), [0.0, -3.5, 1e4, -1e4])))
    edges = np.ascontiguousarray(edges[::order])
    nc = len(edges) - 1
    v = np.concatenate((edges, np.nextafter(edges, np.inf), np.nextafter(edges, -np.inf),
                        [-0.0, np.nextafter(0, 1), np.nextafter(0, -1), 2e4, -2e4, np.inf, np.nan]))
    n = len(v)
    lo, hi = np.minimum(edges[:-1], edges[1:]), np.maximum(edges[:-1], edges[1:])
    held = (v[:, None] >= lo) & (v[:, None] <= hi)
    eng = InsertionEngine("cuda:0")
    amp = 2.0 ** rng.integers(0, 8, n)
    # a pixel each: the cube's rows are the particles' own channels
    x, one = np.arange(n, dtype=float), np.ones(n)
    parts = DeviceParticles.from_host(eng.device, x, np.zeros(n), one, one, None, v=v, amp=amp)
    e = torch.from_numpy(edges).to(eng.device)
    cube, _ = eng.insert(parts, [(N.MG_KERNEL_DIRAC, 0.0)], N.MG_SPECTRUM_DIRAC, 0.0, n, 1, nc, e,
                         form=form)
    np.testing.assert_array_equal(cube.cpu().numpy()[:, 0] != 0, held)
    width = np.abs(np.diff(edges))
    ref = (held * amp[:, None] / width).sum(axis=0)
    got = global_profile(eng, parts, N.MG_SPECTRUM_DIRAC, 0.0, nc, e).cpu().numpy()
    np.testing.assert_allclose(got, ref, rtol=3 * 2.0**-24)  # width, product, amplitude in FP32
