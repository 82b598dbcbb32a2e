"""Particles that are not finite keep their footprint box: a NaN or infinite
amplitude or tabulated value, or a smoothing length of zero, shows in every
pixel of the box (a weight of zero times such a line is NaN, as in the
per-pixel sums of martini/martini.py:243-283) and not only within the kernel's
radius, where the particle list ends for finite ones; channels and tiles that
the box does not reach stay as they are without the particle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY, NC, N_PART = 80, 90, 40, 50


def inputs():
    r = np.random.default_rng(3)
    a = dict(x=r.uniform(0, NX, N_PART), y=r.uniform(0, NY, N_PART), h=r.uniform(2, 6, N_PART),
             v=r.uniform(-70, 70, N_PART), s=r.uniform(5, 9, N_PART), a=r.uniform(1, 2, N_PART),
             t=r.random((N_PART, NC)))
    # a wide box whose corner tiles the kernel does not reach
    a["x"][7], a["y"][7], a["h"][7], a["v"][7] = 40.3, 44.2, 30.0, 3.0
    return a, np.ceil(a["h"])


def insert(a, r, kernel, model, form):
    import torch
    from martini_gb300.engine import DeviceParticles, InsertionEngine
    eng = InsertionEngine("cuda:0")
    table = a["t"] if model == "table" else None
    parts = DeviceParticles.from_host(eng.device, a["x"], a["y"], r, a["h"], None, v=a["v"],
                                      sigma=a["s"], amp=a["a"], spectra=table)
    from martini_gb300 import _native as N
    code = dict(gaussian=N.MG_SPECTRUM_GAUSSIAN, dirac=N.MG_SPECTRUM_DIRAC,
                table=N.MG_SPECTRUM_TABLE)[model]
    edges = torch.from_numpy(np.arange(NC + 1)[::-1] * 4.0 - NC * 2.0).to(eng.device)
    cube, _ = eng.insert(parts, [(kernel, 3.0 if kernel == N.MG_KERNEL_GAUSSIAN else 0.0)], code,
                         0.0, NX, NY, NC, edges, form=form)
    return cube.cpu().numpy()


def box(a, r):
    i, j = np.arange(NX)[:, None], np.arange(NY)[None, :]
    return (np.abs(i - a["x"][7]) <= r[7]) & (np.abs(j - a["y"][7]) <= r[7])


@pytest.mark.parametrize("form", [0, 1, 2, 3], ids=["fp32", "bf16x3", "f16x3", "bf16x6"])
@pytest.mark.parametrize("kernel", [0, 2, 3, 4], ids=["c2", "cubic", "quartic", "gaussian"])
@pytest.mark.parametrize("model,key,value", [
    ("gaussian", "a", np.nan), ("gaussian", "a", np.inf), ("gaussian", "a", 1e300),
    ("dirac", "a", np.nan), ("dirac", "a", -np.inf), ("table", "t", np.nan),
    ("table", "t", -np.inf)])
def test_lines_that_are_not_finite_fill_the_box(model, key, value, kernel, form):
    a, r = inputs()
    want = insert(a, r, kernel, model, form)
    if key == "t":
        a["t"][7, 5] = value
        channel = 5
    else:
        a[key][7] = value
        channel = 19  # the line's: edges 80 - 4 c, velocity 3
    got = insert(a, r, kernel, model, form)
    assert not np.isfinite(got[..., channel][box(a, r)]).any()
    if form != 2:  # the scaled form scales the cube by its largest line
        tiles = np.zeros((NX, NY), bool)  # tiles of 8 x 16 pixels that meet the box
        for i, j in zip(*np.nonzero(box(a, r))):
            tiles[i // 8 * 8:i // 8 * 8 + 8, j // 16 * 16:j // 16 * 16 + 16] = True
        assert np.isfinite(got[~tiles]).all()
        np.testing.assert_array_equal(got[~tiles], want[~tiles])


@pytest.mark.parametrize("form", [0, 1, 3], ids=["fp32", "bf16x3", "bf16x6"])
@pytest.mark.parametrize("kernel", [0, 2], ids=["c2", "cubic"])
@pytest.mark.parametrize("model", ["gaussian", "table"])
@pytest.mark.parametrize("h", [0.0, 1e-25])
def test_a_length_of_zero_fills_the_box(h, model, kernel, form):
    a, r = inputs()
    a["h"][7] = h
    got = insert(a, r, kernel, model, form)
    assert not np.isfinite(got[..., 19][box(a, r)]).any()
