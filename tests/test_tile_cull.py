"""Host restatement of the tile list's culling (`reach2`, `row_tiles`,
csrc/mg_bin.cu) in FP32 against FP64 distances: every tile of a footprint box
that holds a pixel within the support radius must be listed, a tile listed
beyond the box never, and for radii past the limit the whole box is kept (CPU
only; the compiled code is covered by the GPU parity tests)."""

import numpy as np
import pytest

f32 = np.float32
TI, TJ = 8, 16


def reach2(rad):
    m = f32(f32(rad) * f32(1.00002)) + f32(2e-4)
    return f32(m) * f32(m)


def row_tiles(x, y, box, r2, tx):
    ilo, ihi, jlo, jhi = box
    xi, yi = int(np.floor(x)), int(np.floor(y))
    xf, yf = f32(x - xi), f32(y - yi)
    if r2 < f32(1e16):
        a, b = max(tx * TI, ilo), min(tx * TI + TI - 1, ihi)
        d = max(f32(f32(a - xi) - xf), f32(f32(xi - b) + xf), f32(0))
        rem = f32(r2 - f32(d * d))
        half = f32(np.sqrt(max(rem, f32(0))))
        jlo = max(jlo, yi + int(np.ceil(f32(yf - half))))
        jhi = jlo - 1 if rem < 0 else min(jhi, yi + int(np.floor(f32(yf + half))))
        if jhi < jlo:
            return 1, 0
    return jlo // TJ, jhi // TJ


@pytest.mark.parametrize("lo,hi", [(0.2, 3.0), (3.0, 40.0), (40.0, 3000.0)])
def test_culled_tiles_hold_no_pixel_of_the_support(lo, hi):
    rng = np.random.default_rng(int(hi))
    n_px = 200 if hi < 100 else 1200
    culled = 0
    for _ in range(300):
        rad = float(f32(rng.uniform(lo, hi)))
        x, y = rng.uniform(-rad, n_px + rad, 2)
        if rng.random() < 0.3:  # near the tile and pixel grid
            x, y = np.round(x) + rng.choice([0, 1e-9, -1e-9, 0.5]), np.round(y)
        r = np.ceil(rad)
        ilo, ihi = max(int(np.ceil(x - r)), 0), min(int(np.floor(x + r)), n_px - 1)
        jlo, jhi = max(int(np.ceil(y - r)), 0), min(int(np.floor(y + r)), n_px - 1)
        if ilo > ihi or jlo > jhi:
            continue
        i, j = np.arange(ilo, ihi + 1)[:, None], np.arange(jlo, jhi + 1)[None, :]
        inside = (x - i) ** 2 + (y - j) ** 2 < rad * rad
        need = {(a, b) for a, b in zip(*(v.ravel()[inside.ravel()] for v in np.broadcast_arrays(
            i // TI, j // TJ)))}
        got = set()
        for tx in range(ilo // TI, ihi // TI + 1):
            t0, t1 = row_tiles(x, y, (ilo, ihi, jlo, jhi), reach2(rad), tx)
            got |= {(tx, t) for t in range(t0, t1 + 1)}
        box = {(a, b) for a in range(ilo // TI, ihi // TI + 1)
               for b in range(jlo // TJ, jhi // TJ + 1)}
        assert need <= got <= box
        culled += len(box) - len(got)
    assert culled > 0


def test_radii_past_the_limit_keep_the_box():
    assert row_tiles(3.2, 4.1, (0, 99, 0, 99), reach2(2e8), 5) == (0, 6)
