"""Global profile of few particles and of wide lines and bands: the ranges of
particles and the chunks of channels at the sizes where they change shape (one
particle a warp and past it, one chunk and several, bands off and on the
chunks' edges, more particles than the blocks fill the chip with), and no more
time for wide lines than for as much work in narrow ones.

Tolerance as for the other bands: a line value is the difference of two erfc
values of at most 4 ulp each, within 1e-6 of the profile's peak for lines of
up to 8 channels' width."""

import time

import numpy as np
import pytest

from oracle import martini_oracle as orc

pytestmark = pytest.mark.gpu


def parts_of(eng, v, sig, amp):
    from martini_gb300.engine import DeviceParticles
    z = np.zeros(len(v))
    return DeviceParticles.from_host(eng.device, z, z, z, z, v=v, sigma=sig, amp=amp)


@pytest.mark.parametrize("n,nc", [(1, 64), (1, 65), (7, 1535), (8, 1536), (9, 1537), (33, 300),
                                  (257, 31), (300, 3100), (2431, 96), (2433, 128), (40000, 257)])
@pytest.mark.parametrize("model", ["gaussian", "dirac"])
@pytest.mark.parametrize("order", [1, -1], ids=["rising", "falling"])
def test_ranges_and_chunks(n, nc, model, order):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine, global_profile
    rng = np.random.default_rng(n + nc)
    edges = np.ascontiguousarray(np.sort(orc.vrad_channel_edges(nc, 4.0, 100.0))[::order])
    half = max(2.0 * nc, 20.0)
    v = rng.uniform(100.0 - 1.1 * half, 100.0 + 1.1 * half, n)
    v[0] = 100.0
    v[-1] = edges[nc // 2]  # a Dirac line on an edge lies in both channels
    sig = rng.uniform(2.0, 30.0, n).astype(np.float32)
    mhi = 10 ** rng.uniform(4, 6, n)
    ref = orc.init_spectra(model, mhi, np.full(n, 3.0), v, edges,
                           sig.astype(np.float64) if model == "gaussian" else None).sum(axis=0)
    eng = InsertionEngine("cuda:0")
    parts = parts_of(eng, v, sig, mhi / 9.0 / orc.MHI_TO_JY)
    m = N.MG_SPECTRUM_GAUSSIAN if model == "gaussian" else N.MG_SPECTRUM_DIRAC
    e = torch.from_numpy(edges).to(eng.device)
    got = global_profile(eng, parts, m, 0.0, nc, e)
    assert torch.equal(got, global_profile(eng, parts, m, 0.0, nc, e))
    assert np.abs(got.cpu().numpy() - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("n,nc,sigma", [(32, 256, 100.0), (200, 1024, 1000.0), (400, 8192, 1000.0)])
def test_wide_lines_take_no_longer_than_narrow_ones(n, nc, sigma):
    import torch
    from martini_gb300 import _native as N
    from martini_gb300.engine import InsertionEngine, global_profile
    eng = InsertionEngine("cuda:0")
    rng = np.random.default_rng(n)
    e = torch.from_numpy(np.arange(nc + 1) * 4.0).to(eng.device)
    v = rng.uniform(0.45, 0.55, n) * 4.0 * nc
    wide = min(nc, 9.0 * np.sqrt(2.0) * sigma / 4.0)
    k = int(n * wide / 32.0)  # lines of 32 channels, as many channels in all
    us = []
    for count, s in ((n, sigma), (k, 32.0 * 4.0 / (9.0 * np.sqrt(2.0)))):
        parts = parts_of(eng, np.resize(v, count), np.full(count, s), np.ones(count))
        t = []
        for _ in range(21):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            global_profile(eng, parts, N.MG_SPECTRUM_GAUSSIAN, 0.0, nc, e)
            torch.cuda.synchronize()
            t.append((time.perf_counter() - t0) * 1e6)
        us.append(sorted(t)[10])
    assert us[0] <= 1.35 * us[1] + 15.0, us
