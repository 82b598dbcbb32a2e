"""Performance cases: the work a user of this package has it do.

Every case goes through a public entry point: ``InsertionEngine.insert`` (plan, insertion and check
in one call, as ``Martini`` itself calls it), ``InsertionEngine.run`` on a problem planned once,
``insert_batch``, ``setup_on_gpu``, ``global_profile``, ``convolve_beam`` and
``Martini.insert_source_in_cube``.  Particles are inclined exponential HI discs (and, for the
stress cases, a Plummer halo and smoothing lengths over 2.6 decades), the distributions of the
package's own workloads, drawn on the GPU from the seed.

The flux sums are FP64 sums of FP32 voxels and the ``Martini`` array is an FP64 copy of the FP32
cube, so both are returned as float32, the precision of what they hold.
"""

import math

import numpy as np
import torch

from martini_gb300 import DataCube, Martini, SPHSource
from martini_gb300 import _native as N
from martini_gb300 import spectral_models, sph_kernels
from martini_gb300.engine import (DeviceParticles, InsertionEngine, convolve_beam, global_profile,
                                  insert_batch, setup_on_gpu)

FORMS = {"fp32": N.MG_FORM_FP32, "f16x3": N.MG_FORM_F16X3, "bf16x6": N.MG_FORM_BF16X6}
C2, C6, CUBIC, QUARTIC, GAUSS, DIRAC = (
    N.MG_KERNEL_WENDLAND_C2, N.MG_KERNEL_WENDLAND_C6, N.MG_KERNEL_CUBIC_SPLINE,
    N.MG_KERNEL_QUARTIC_SPLINE, N.MG_KERNEL_GAUSSIAN, N.MG_KERNEL_DIRAC)
# kernel: class of the adaptive tuple, type, truncation, 1 / FWHM (the length scale and the
# footprint size in FWHM), smallest valid length in px
GAUSS_SIGMA = 1.0 / (2.0 * math.sqrt(2.0 * math.log(2.0)))
KERNELS = {
    "wendland_c2": ("WendlandC2Kernel", C2, 0.0, 1.5933199337482513, 1.51),
    "wendland_c6": ("WendlandC6Kernel", C6, 0.0, 1.9803392771717987, 1.29),
    "cubic": ("CubicSplineKernel", CUBIC, 0.0, 1.3843671526381416, 1.16),
    "quartic": ("QuarticSplineKernel", QUARTIC, 0.0, 1.567997458608026, 1.2385),
    "gaussian3": ("GaussianKernel", GAUSS, 3.0, 3.0 * GAUSS_SIGMA, 2.3357),
}
MHI_TO_JY = 2.36e5     # Msun / (Mpc^2 Jy km/s)
K_B, M_P = 1.380649e-23, 1.67262192369e-27
HUBBLE = 70.0          # km/s/Mpc (h = 0.7, the source's default)
PX = 10.0              # arcsec

# One insertion.  distance in Mpc, radius (scale length) and smoothing lengths in kpc, dv in km/s.
DISC = dict(kind="insert", planned=False, accumulate=False, n=1_000_000, nx=512, ny=512, nc=256,
            pad=0, distance=3.0, radius=3.0, h_med=1.0, h_dex=0.3, h_lo=0.0, h_hi=0.0, halo=0.0,
            dv=4.0, kernel="wendland_c2", form="bf16x6", sigma="thermal")


def listed():
    return [
        # the smallest call: the reference's own small disc, a few thousand particles; latency,
        # launches and host work count
        dict(DISC, name="insert_disc5k_64_cubic", n=5_000, nx=64, ny=64, nc=32, kernel="cubic",
             sigma="7"),
        # the ordinary call: a resolved galaxy on a survey cube, default form
        dict(DISC, name="insert_disc1m_512"),
        # the high-resolution cube of the benchmark, planned once and inserted again and again
        dict(DISC, name="planned_disc4m_1024", planned=True, n=4_000_000, nx=1024, ny=1024, nc=512,
             distance=10.0, radius=10.0, h_med=0.5, h_dex=0.5, dv=2.0),
        # a Gaussian-kernel source on a ragged, padded cube (as before a beam convolution), in the
        # scaled FP16 form
        dict(DISC, name="insert_gauss300k_f16x3_pad", n=300_000, nx=301, ny=243, nc=150, pad=13,
             kernel="gaussian3", form="f16x3", dv=5.0),
        # the plain FP32 form on a small odd cube
        dict(DISC, name="insert_quartic100k_fp32", n=100_000, nx=187, ny=211, nc=75,
             kernel="quartic", form="fp32", sigma="9.5", dv=7.0),
        # line-of-sight particles with delta-function lines added into a cube that already holds
        # another spectral group
        dict(DISC, name="accumulate_dirac200k", planned=True, accumulate=True, n=200_000, nx=512,
             ny=512, nc=256, h_lo=0.05, h_hi=20.0, halo=0.1, sigma="dirac"),
        # wide smoothing lengths (coarse halo particles over hundreds of pixels): the densest work
        dict(DISC, name="stress500k_1024", planned=True, n=500_000, nx=1024, ny=1024, nc=256,
             h_lo=0.05, h_hi=20.0, halo=0.1),
        # a population of galaxies of 1e3 .. 1e6 particles on four cube shapes, one batch
        dict(name="batch_population48", kind="batch", galaxies=48, table=4, logn_lo=3.0,
             logn_hi=6.0, form="bf16x6"),
        # the spatially integrated spectrum of a source
        dict(name="global_profile_1m", kind="profile", n=1_000_000, nc=256, dv=4.0, sigma="thermal"),
        # beam convolution of an inserted, padded cube: 30 arcsec beam truncated at 4 FWHM
        dict(name="beam_512x256_27px", kind="beam", nx=512, ny=512, nc=256, beam=27, fwhm=3.0),
        # projection, kernel choice and pruning of a host-side source (on a cube wide enough to keep
        # every particle, so that its outputs have one length)
        dict(name="setup_500k", kind="setup", n=500_000, nx=1024, ny=1024, nc=256, dv=4.0,
             kernel="wendland_c2"),
        # the drop-in call on the reference's classes, from host arrays to the host cube
        dict(name="martini_100k_128", kind="martini", n=100_000, nx=128, ny=128, nc=128, dv=4.0,
             kernel="wendland_c2", form="bf16x6"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["insert"] * 7 + ["stress", "batch", "profile", "beam", "setup", "martini"])
    if kind == "insert":
        nx = _log(rng, 40, 700)
        return dict(DISC, planned=rng.random() < 0.4, accumulate=rng.random() < 0.2,
                    n=_log(rng, 2_000, 1_500_000), nx=nx, ny=max(33, int(nx * rng.uniform(0.6, 1.4))),
                    nc=_log(rng, 24, 400), pad=rng.choice([0, 0, 5, 14]),
                    distance=round(rng.uniform(2.5, 10.0), 3), radius=round(rng.uniform(2.0, 8.0), 3),
                    h_med=round(rng.uniform(0.4, 1.2), 3), h_dex=round(rng.uniform(0.2, 0.5), 3),
                    dv=rng.choice([2.0, 4.0, 5.2, 8.0]), kernel=rng.choice(sorted(KERNELS)),
                    form=rng.choice(["bf16x6", "bf16x6", "bf16x6", "f16x3", "fp32"]),
                    sigma=rng.choice(["thermal", "thermal", "7", "12.5", "dirac"]))
    if kind == "stress":
        nx = _log(rng, 200, 900)
        return dict(DISC, planned=rng.random() < 0.5, accumulate=rng.random() < 0.3,
                    n=_log(rng, 20_000, 300_000), nx=nx, ny=nx, nc=_log(rng, 60, 256), h_lo=0.05,
                    h_hi=round(rng.uniform(8.0, 20.0), 2), halo=0.1,
                    sigma=rng.choice(["thermal", "thermal", "dirac"]))
    if kind == "batch":
        return dict(kind="batch", galaxies=rng.randint(3, 60), table=rng.randint(5, 10_000),
                    logn_lo=3.0, logn_hi=round(rng.uniform(4.0, 5.8), 3),
                    form=rng.choice(["bf16x6", "bf16x6", "f16x3", "fp32"]))
    if kind == "profile":
        return dict(kind="profile", n=_log(rng, 3_000, 2_000_000), nc=_log(rng, 30, 600),
                    dv=rng.choice([2.0, 4.0]), sigma=rng.choice(["thermal", "7", "dirac"]))
    if kind == "beam":
        return dict(kind="beam", nx=_log(rng, 64, 512), ny=_log(rng, 64, 512), nc=_log(rng, 24, 256),
                    beam=rng.choice([9, 13, 17, 21, 27, 33]), fwhm=round(rng.uniform(1.5, 3.5), 3))
    kernel = rng.choice(sorted(KERNELS))
    if kind == "setup":
        nx = _log(rng, 1000, 2100)
        return dict(kind="setup", n=_log(rng, 5_000, 700_000), nx=nx, ny=nx + rng.randint(0, 40),
                    nc=_log(rng, 170, 400), dv=rng.choice([4.0, 5.2]), kernel=kernel)
    nx = _log(rng, 48, 160)
    return dict(kind="martini", n=_log(rng, 3_000, 200_000), nx=nx, ny=nx + rng.randint(0, 20),
                nc=_log(rng, 24, 140), dv=rng.choice([4.0, 8.0]), kernel=kernel,
                form=rng.choice(["bf16x6", "f16x3"]))


# ---- inputs ----------------------------------------------------------------------------------------


def _disc(g, n, device, radius=3.0, h_med=1.0, h_dex=0.3, h_lo=0.0, h_hi=0.0, halo=0.0,
          v_flat=200.0, incl=60.0):
    """Positions (kpc), velocities (km/s), HI masses (Msun), smoothing lengths (kpc) and
    temperatures (K) of an inclined exponential disc about the origin, the line of sight along x."""
    def uniform(*shape):
        return torch.rand(shape, generator=g, device=device, dtype=torch.float64)

    def normal(*shape):
        return torch.randn(shape, generator=g, device=device, dtype=torch.float64)

    phi = 2.0 * math.pi * uniform(n)
    R = -radius * torch.log(uniform(n).clamp_min(1e-12) * uniform(n).clamp_min(1e-12))
    z = 0.3 * normal(n)
    vphi = v_flat * torch.atan(R) / (math.pi / 2.0)
    c, s = torch.cos(phi), torch.sin(phi)
    disp = 10.0 * normal(n, 3)
    # disc normal along the line of sight, then tilted about y
    p = torch.stack((z, R * c, R * s), 1)
    v = torch.stack((torch.zeros_like(R), -vphi * s, vphi * c), 1) + disp
    ci, si = math.cos(math.radians(incl)), math.sin(math.radians(incl))
    tilt = torch.tensor([[ci, 0.0, si], [0.0, 1.0, 0.0], [-si, 0.0, ci]], dtype=torch.float64,
                        device=device)
    p, v = p @ tilt.T, v @ tilt.T
    if halo:
        k = int(halo * n)
        r = 20.0 / torch.sqrt(uniform(k).clamp_min(1e-9) ** (-2.0 / 3.0) - 1.0 + 1e-12)
        u = normal(k, 3)
        p[:k] = u / u.norm(dim=1, keepdim=True) * r.clamp_max(400.0)[:, None]
        v[:k] = 30.0 * normal(k, 3)
    mhi = 1e5 * 10.0 ** (0.2 * normal(n))
    if h_hi:
        h = 10.0 ** (math.log10(h_lo) + math.log10(h_hi / h_lo) * uniform(n))
    else:
        h = h_med * 10.0 ** (h_dex * normal(n))
    return p, v, mhi, h, 1e4 * 10.0 ** (0.3 * normal(n))


def _edges(nc, dv, centre):
    """Channel edges of a VRAD axis, km/s, decreasing."""
    return centre - dv * (np.arange(nc + 1) - 0.5 * nc)


def _project(p, v, mhi, h, T, distance, nx, ny, nc, dv, kernel, sigma, prune=True):
    """Pixel coordinates, ranges, kernel lengths and choice, velocity, width and amplitude of
    particles about (ra, dec) = (0, 0), those that reach the cube only."""
    pos = p.clone()
    pos[:, 0] += distance * 1e3
    vel = v + HUBBLE * 1e-3 * pos
    d = pos.norm(dim=1)
    vlos = (pos * vel).sum(1) / d
    deg = 180.0 / math.pi
    x = (nx / 2.0 - 0.5) - (pos[:, 1] / pos[:, 0]) * deg * 3600.0 / PX
    y = (ny / 2.0 - 0.5) + (pos[:, 2] / pos[:, 0]) * deg * 3600.0 / PX
    hpx = torch.atan(h / d) * deg * 3600.0 / PX
    _, _, _, inv_fwhm, least = KERNELS[kernel]
    own_scale = 1.0 if kernel == "gaussian3" else inv_fwhm
    own = hpx * own_scale >= least
    dirac = ~own & (hpx <= 0.5)
    gauss = ~own & ~dirac & (hpx >= 0.336)
    kidx = torch.where(own, 0, torch.where(dirac, 1, torch.where(gauss, 2, -1))).to(torch.int8)
    size = torch.where(dirac, 1.0, torch.where(gauss, 6.0 * GAUSS_SIGMA, inv_fwhm))
    scale = torch.where(dirac | gauss, 1.0, own_scale)
    r = torch.ceil(hpx * size)
    if sigma == "thermal":
        sig = torch.sqrt(K_B * T / M_P) / 1e3
    else:
        sig = torch.full_like(T, 0.0 if sigma == "dirac" else float(sigma))
    out = dict(x=x, y=y, sm_range=r, h_eff=(hpx * scale).float(), kernel_index=kidx, v=vlos,
               sigma=sig.float(), amp=mhi / (d * 1e-3) ** 2 / MHI_TO_JY)
    if prune:
        chan = nc / 2.0 - 0.5 - (vlos - HUBBLE * distance) / dv
        keep = ((x + r >= 0) & (y + r >= 0) & (x - r <= nx) & (y - r <= ny)
                & (chan + 4 * sig / dv >= 0) & (chan - 4 * sig / dv <= nc))
        out = {k: t[keep].contiguous() for k, t in out.items()}
    return out


def _insert_inputs(c, seed, device="cuda", n=None):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    q = _disc(g, n or c["n"], device, c["radius"], c["h_med"], c["h_dex"], c["h_lo"], c["h_hi"],
              c["halo"])
    nx, ny = c["nx"] + 2 * c["pad"], c["ny"] + 2 * c["pad"]
    a = _project(*q, c["distance"], nx, ny, c["nc"], c["dv"], c["kernel"], c["sigma"])
    return a, nx, ny, _edges(c["nc"], c["dv"], HUBBLE * c["distance"])


def _table(kernel):
    return [(KERNELS[kernel][1], KERNELS[kernel][2]), (DIRAC, 0.0), (GAUSS, 6.0)]


def _particles(a, sigma):
    """DeviceParticles, spectral model and constant width of an input set."""
    if sigma == "dirac":
        model, const, sig = N.MG_SPECTRUM_DIRAC, 0.0, None
    elif sigma == "thermal":
        model, const, sig = N.MG_SPECTRUM_GAUSSIAN, 0.0, a["sigma"]
    else:
        model, const, sig = N.MG_SPECTRUM_GAUSSIAN, float(sigma), None
    return DeviceParticles(a["x"], a["y"], a["sm_range"], a["h_eff"], a["kernel_index"], v=a["v"],
                           sigma=sig, amp=a["amp"]), model, const


def _population(c):
    """The galaxies of a batch: particle count, inclination, rotation and cube of each, from the
    case alone."""
    rng = np.random.default_rng(c["table"])
    out = []
    for _ in range(c["galaxies"]):
        n = int(round(10 ** rng.uniform(c["logn_lo"], c["logn_hi"])))
        incl = float(np.rad2deg(np.arccos(rng.uniform())))
        v_flat = float(rng.uniform(50.0, 300.0))
        nx, nc = ((32, 64), (64, 128), (128, 128), (256, 256))[int(rng.integers(4))]
        out.append((n, incl, v_flat, nx, nc))
    return out


def _batch_inputs(c, seed, device="cuda", most=None):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    for n, incl, v_flat, nx, nc in _population(c):
        q = _disc(g, min(n, most or n), device, v_flat=v_flat, incl=incl)
        yield (n, _project(*q, 3.0, nx, nx, nc, 4.0, "wendland_c2", "thermal"), nx, nc,
               _edges(nc, 4.0, HUBBLE * 3.0))


def _host_source(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    p, v, mhi, h, T = (t.cpu().numpy() for t in _disc(g, c["n"], "cuda"))
    ra, dec = (33.0, -12.0) if c["kind"] == "setup" else (0.0, 0.0)
    src = SPHSource(distance=3.0, T_g=T, mHI_g=mhi, xyz_g=p, vxyz_g=v, hsm_g=h, ra=ra, dec=dec)
    dc = DataCube(n_px_x=c["nx"], n_px_y=c["ny"], n_channels=c["nc"], px_size=PX,
                  channel_width=c["dv"], spectral_centre=src.vsys, ra=ra, dec=dec)
    return src, dc, getattr(sph_kernels, KERNELS[c["kernel"]][0])()


def _beam_inputs(c, seed):
    """A cube of smooth, mostly positive emission and the pixel-sampled beam image."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    pad = c["beam"] // 2
    nx, ny, nc = c["nx"] + 2 * pad, c["ny"] + 2 * pad, c["nc"]
    cube = torch.rand((nx, ny, nc), generator=g, device="cuda", dtype=torch.float32) ** 4
    line = torch.exp(-0.5 * ((torch.arange(nc, device="cuda") - nc / 2) / (nc / 5)) ** 2)
    cube *= line.float()
    s = c["fwhm"] * GAUSS_SIGMA
    u = np.arange(c["beam"]) - pad
    rot = 0.5 * u[:, None] + u[None, :]
    kern = np.exp(-0.5 * ((u[:, None] / s) ** 2 + (rot / (1.3 * s)) ** 2))
    return cube, pad, kern / kern.sum()


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(case=c)
    if kind == "martini":
        src, dc, kern = _host_source(c, seed)
        st["martini"] = Martini(source=src, datacube=dc, sph_kernel=kern, quiet=True,
                                spectral_model=spectral_models.GaussianSpectrum(sigma="thermal"),
                                form=c["form"])
        return st
    if kind == "setup":
        src, dc, kern = _host_source(c, seed)
        st.update(engine=InsertionEngine(), source=src, datacube=dc, kernel=kern,
                  model=spectral_models.GaussianSpectrum(sigma="thermal"))
        return st
    eng = st["engine"] = InsertionEngine()
    if kind == "insert":
        a, nx, ny, edges = _insert_inputs(c, seed)
        parts, model, const = _particles(a, c["sigma"])
        st.update(parts=parts, model=model, const=const, nx=nx, ny=ny,
                  edges=torch.from_numpy(edges).cuda(), table=_table(c["kernel"]))
        if c["accumulate"]:
            g = torch.Generator(device="cuda")
            g.manual_seed(int(seed) + 1)
            st["base"] = torch.rand((nx, ny, c["nc"]), generator=g, device="cuda")
        if c["planned"]:
            st["cube"] = torch.empty((nx, ny, c["nc"]), device="cuda")
            st["flux"] = torch.empty(c["nc"] + 1, dtype=torch.float64, device="cuda")
            st["problem"] = eng.problem(parts, st["table"], model, const, nx, ny, c["nc"], c["pad"],
                                        c["pad"], st["edges"], st["cube"], st["flux"],
                                        FORMS[c["form"]], accumulate=c["accumulate"])
            eng.plan(st["problem"])
    elif kind == "batch":
        st["items"] = []
        for _, a, nx, nc, edges in _batch_inputs(c, seed):
            st["items"].append(dict(parts=_particles(a, "thermal")[0], nx=nx, ny=nx, nc=nc,
                                    edges=torch.from_numpy(edges).cuda()))
    elif kind == "profile":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        a = _project(*_disc(g, c["n"], "cuda"), 3.0, 1, 1, c["nc"], c["dv"], "wendland_c2",
                     c["sigma"], prune=False)
        st["parts"], st["model"], st["const"] = _particles(a, c["sigma"])
        st["edges"] = torch.from_numpy(_edges(c["nc"], c["dv"], HUBBLE * 3.0)).cuda()
    else:
        st["cube"], st["pad"], st["beam"] = _beam_inputs(c, seed)
    return st


# ---- one pass --------------------------------------------------------------------------------------


def run(state):
    c, st = state["case"], state
    kind = c["kind"]
    if kind == "martini":
        m = st["martini"]
        m.reset()
        m.insert_source_in_cube(skip_validation=True)
        return {"cube": m.datacube._array.astype(np.float32), "flux": m.inserted_flux_density}
    eng = st["engine"]
    if kind == "setup":
        p, _, _, _ = setup_on_gpu(eng, st["source"], st["datacube"], st["kernel"], st["model"])
        return {"x": p.x, "y": p.y, "sm_range": p.sm_range, "h_eff": p.h_eff,
                "kernel_index": p.kernel_index, "v": p.v, "sigma": p.sigma, "amp": p.amp}
    if kind == "insert":
        if c["planned"]:
            if c["accumulate"]:
                st["cube"].copy_(st["base"])
            eng.run(st["problem"])
            return {"cube": st["cube"], "flux": st["flux"].float()}
        cube = st["base"].clone() if c["accumulate"] else None
        cube, flux = eng.insert(st["parts"], st["table"], st["model"], st["const"], st["nx"],
                                st["ny"], c["nc"], st["edges"], padx=c["pad"], pady=c["pad"],
                                form=FORMS[c["form"]], cube=cube, accumulate=c["accumulate"])
        return {"cube": cube, "flux": flux.float()}
    if kind == "batch":
        outs = insert_batch(eng, st["items"], _table("wendland_c2"), N.MG_SPECTRUM_GAUSSIAN,
                            form=FORMS[c["form"]])
        return {"cubes": torch.cat([q.reshape(-1) for q, _ in outs]),
                "flux": torch.cat([f for _, f in outs]).float()}
    if kind == "profile":
        return global_profile(eng, st["parts"], st["model"], st["const"], c["nc"],
                              st["edges"]).float()
    return convolve_beam(eng, st["cube"], st["pad"], st["pad"], st["beam"], 1.0)


# ---- what a pass cannot do without -----------------------------------------------------------------


def _pairs(a, nx, ny, nc, dv, edges):
    """Mean box pixels x support channels of a sample of particles (clipped to the cube)."""
    def span(t, r, n):
        return (torch.floor(t + r).clamp_max(n - 1) - torch.ceil(t - r).clamp_min(0) + 1).clamp_min(0)
    box = span(a["x"], a["sm_range"], nx) * span(a["y"], a["sm_range"], ny)
    chans = (9.0 * math.sqrt(2.0) * a["sigma"].double() / dv + 1.0).clamp_max(nc)
    return float((box * chans).mean()) if box.numel() else 0.0, float(chans.mean())


def work(case):
    c, kind = case, case["kind"]
    if kind == "insert":
        m = min(c["n"], 20_000)
        a, nx, ny, edges = _insert_inputs(c, 0, "cpu", m)
        kept = c["n"] * a["x"].numel() / m
        px, _ = _pairs(a, nx, ny, c["nc"], c["dv"], edges)
        cube = 4.0 * nx * ny * c["nc"]
        return {"bytes": cube * (2 if c["accumulate"] else 1) + 57.0 * kept, "flops": 2.0 * px * kept}
    if kind == "batch":
        by = fl = 0.0
        for n, a, nx, nc, edges in _batch_inputs(c, 0, "cpu", 2_000):
            kept = n * a["x"].numel() / min(n, 2_000)
            by += 4.0 * nx * nx * nc + 57.0 * kept
            fl += 2.0 * kept * _pairs(a, nx, nx, nc, 4.0, edges)[0]
        return {"bytes": by, "flops": fl}
    if kind == "profile":
        sig = {"thermal": 9.1, "dirac": 0.0}.get(c["sigma"]) if c["sigma"] in ("thermal", "dirac") \
            else float(c["sigma"])
        return {"bytes": 20.0 * c["n"] + 8.0 * c["nc"],
                "flops": 30.0 * c["n"] * min(c["nc"], 9.0 * math.sqrt(2.0) * sig / c["dv"] + 1.0)}
    if kind == "beam":
        pad = c["beam"] // 2
        return {"bytes": 4.0 * c["nc"] * ((c["nx"] + 2 * pad) * (c["ny"] + 2 * pad)
                                          + c["nx"] * c["ny"]),
                "flops": 2.0 * c["nx"] * c["ny"] * c["nc"] * c["beam"] ** 2}
    if kind == "setup":
        return {"bytes": (72.0 + 57.0) * c["n"], "flops": 150.0 * c["n"]}
    return {"bytes": 12.0 * c["nx"] * c["ny"] * c["nc"] + 57.0 * c["n"],
            "flops": 2.0 * c["n"] * 200.0 * 20.0}


# ---- the same results in 64 bits ---------------------------------------------------------------------


def _c6_indefinite(R, z):
    # line-of-sight integral of the Wendland C6 kernel, with the closed form's published constants
    q = torch.sqrt(R * R + z * z)
    L = torch.log(q + z)
    return (-231 * R**10 * z - 385 * R**8 * z**3 - 1155 * R**8 * z - 462 * R**6 * z**5
            - 1540 * R**6 * z**3 - 462 * R**6 * z - 330 * R**4 * z**7 - 1386 * R**4 * z**5
            - 462 * R**4 * z**3 + 66 * R**4 * z - (128 + 1 / 3) * R**2 * z**9 - 660 * R**2 * z**7
            - 277.2 * R**2 * z**5 + 44 * R**2 * z**3 + 8 / 3 * z**11 * q
            + (16 + 4 / 15) * R**2 * z**9 * q + 70.4 * z**9 * q + 360.8 * R**2 * z**7 * q
            + 132 * z**7 * q + 550 * R**2 * z**5 * q - 11 * R**2 * z + 7.21875 * R**12 * L
            + 24.7813 * R**10 * z * q + 173.25 * R**10 * L + 530.75 * R**8 * z * q
            + 288.75 * R**8 * L + 47.4792 * R**8 * z**3 * q + 767.25 * R**6 * z * q
            + 58.0167 * R**6 * z**5 * q + 819.5 * R**6 * z**3 * q + 41.7 * R**4 * z**7 * q
            + 752.4 * R**4 * z**5 * q + 896.5 * R**4 * z**3 * q - 21 * z**11
            - (128 + 1 / 3) * z**9 - 66 * z**7 + 13.2 * z**5 - 11 / 3 * z**3 + z)


def _quartic_shell(R, A):
    z = torch.sqrt((A * A - R * R).clamp_min(0))
    q, R2 = torch.sqrt(z * z + R * R), R * R
    v = (A**4 * z - 2 * A**3 * z * q + 2 * A**2 * z * (3 * R2 + z * z)
         - A * R2 * (4 * A**2 + 3 * R2) * torch.asinh(z / R) / 2 - A * z * q * (5 * R2 + 2 * z * z) / 2
         + R2 * R2 * z + 2 * R2 * z**3 / 3 + z**5 / 5)
    return torch.where(R < A, v, torch.zeros_like(v))


def _weights(kind, trunc, dx, dy, h):
    """Kernel integrals over pixels at offsets dx, dy (px) of particles of length h (px)."""
    r2 = dx * dx + dy * dy
    if kind == DIRAC:
        return ((dx.abs() < 0.5) & (dy.abs() < 0.5)).double()
    if kind == GAUSS:
        s = h * GAUSS_SIGMA
        e = [torch.erf((d + 0.5) / s / math.sqrt(2)) - torch.erf((d - 0.5) / s / math.sqrt(2))
             for d in (dx, dy)]
        dr = torch.sqrt(r2)
        zmax = torch.sqrt((trunc**2 - r2 / (s * s)).clamp_min(0))
        norm = math.erf(trunc / math.sqrt(2)) - 2 * trunc / math.sqrt(2 * math.pi) * math.exp(
            -trunc**2 / 2)
        w = 0.25 * torch.erf(zmax / math.sqrt(2)) * e[0] * e[1] / norm
        return torch.where((dr - math.sqrt(0.5)) / s > trunc, torch.zeros_like(w), w)
    R2 = (r2 / (h * h)).clamp_min(1e-24)
    if kind == C2:
        A = torch.sqrt((1 - R2).clamp_min(0))
        f = 5 * R2 * R2 * (0.5 * R2 + 3) * torch.log((1 + A) / torch.sqrt(R2)) + A * (
            -27 / 2 * R2 * R2 - 14 / 3 * R2 + 2 / 3)
        f = torch.where(R2 < 1, f, torch.zeros_like(f)) * (21 / 2 / math.pi)
    elif kind == C6:
        R = torch.sqrt(R2.clamp_max(1))
        f = _c6_indefinite(R, torch.sqrt((1 - R * R).clamp_min(0))) - _c6_indefinite(
            R, torch.zeros_like(R))
        f = torch.where(R2 < 1, f, torch.zeros_like(f)) * (2 * 1365 / 64 / math.pi)
    elif kind == QUARTIC:
        R = torch.sqrt(R2)
        f = (10 * _quartic_shell(R, 0.2) - 5 * _quartic_shell(R, 0.6) + _quartic_shell(R, 1.0)) * (
            2 * 15625 / 512 / math.pi)
    else:
        R4 = 4 * R2
        A, B = torch.sqrt((1 - R4).clamp_min(0)), torch.sqrt((4 - R4).clamp_min(0))
        root = torch.sqrt(R4)
        inner = (A - 0.5 * A**3 - 1.5 * R4 * A + 3 / 32 * A * (3 * R4 + 2)
                 + 9 / 32 * R4 * R4 * (torch.log(1 + A) - torch.log(root)))
        ring = (-B * (3 * R4 + 56) / 4 + A * (4 * R4 + 50) / 8
                - 3 / 8 * R4 * (R4 + 16) * torch.log((2 + B) / (1 + A))
                + 2 * (3 * R4 + 4) * (B - A) + 2 * (B**3 - A**3))
        outer = (-B * (3 * R4 + 56) / 4 - 3 / 8 * R4 * (R4 + 16) * torch.log((2 + B) / root)
                 + 2 * (3 * R4 + 4) * B + 2 * B**3)
        f = torch.where(R4 <= 1, inner + 0.25 * ring,
                        torch.where(R4 < 4, 0.25 * outer, torch.zeros_like(R4)))
        f = f * 4 / 1.59689476201133
    return f / (h * h)


def _lines(a, sigma, edges):
    """Channel spectra [n, nc] of the particles' lines."""
    e = torch.from_numpy(edges).cuda()
    v, w = a["v"][:, None], (e[1:] - e[:-1]).abs()
    if sigma == "dirac":
        phi = ((v <= e[:-1]) & (v >= e[1:])).double()  # edges decrease; both channels on an edge
    else:
        t = torch.erf((e[None, :] - v) / (math.sqrt(2) * a["sigma"].double()[:, None]))
        phi = 0.5 * (t[:, :-1] - t[:, 1:])
    return a["amp"][:, None] * phi / w


def _exact_cube(a, nx, ny, edges, kernel, sigma):
    """The cube (Jy/pix^2) as a sum over the particles whose footprint box holds the pixel, by
    16 x 16 pixel tiles."""
    S, side, nc = _lines(a, sigma, edges), 16, len(edges) - 1
    cube = torch.zeros((nx, ny, nc), dtype=torch.float64, device="cuda")
    x, y, r = a["x"], a["y"], a["sm_range"]
    lo = [((torch.ceil(t - r)).clamp_min(0) // side).long() for t in (x, y)]
    hi = [(torch.floor(t + r).clamp(-1, n - 1) // side).long() for t, n in ((x, nx), (y, ny))]
    span = [(b - t + 1).clamp_min(0) for t, b in zip(lo, hi)]
    count = span[0] * span[1]
    pid = torch.repeat_interleave(torch.arange(x.numel(), device="cuda"), count)
    first = torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
    e = torch.arange(pid.numel(), device="cuda") - first
    nty = (ny + side - 1) // side
    kind = a["kernel_index"].long().clamp_min(0)
    tile = (lo[0][pid] + e // span[1][pid]) * nty + lo[1][pid] + e % span[1][pid]
    order = torch.argsort(tile * 3 + kind[pid], stable=True)
    keys, pid = (tile * 3 + kind[pid])[order], pid[order]
    uniq, n_in = torch.unique_consecutive(keys, return_counts=True)
    at = 0
    for key, n in zip(uniq.tolist(), n_in.tolist()):
        t, k = divmod(key, 3)
        i0, j0 = (t // nty) * side, (t % nty) * side
        i = torch.arange(i0, min(i0 + side, nx), device="cuda", dtype=torch.float64)
        j = torch.arange(j0, min(j0 + side, ny), device="cuda", dtype=torch.float64)
        ktype, trunc = _table(kernel)[k]
        for b in range(at, at + n, 32768):
            q = pid[b:min(b + 32768, at + n)]
            dx = x[q][:, None, None] - i[None, :, None]
            dy = y[q][:, None, None] - j[None, None, :]
            rq = r[q][:, None, None]
            w = _weights(ktype, trunc, *torch.broadcast_tensors(dx, dy),
                         a["h_eff"][q].double()[:, None, None])
            w = w * ((dx.abs() <= rq) & (dy.abs() <= rq))
            add = w.reshape(len(q), -1).T @ S[q]
            cube[i0:i0 + len(i), j0:j0 + len(j)] += add.reshape(len(i), len(j), nc)
        at += n
    return cube


def _flux(cube, pad):
    c = cube[pad:cube.shape[0] - pad, pad:cube.shape[1] - pad]
    per = c.sum((0, 1))
    return torch.cat((per.sum()[None], per))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "insert":
        a, nx, ny, edges = _insert_inputs(c, seed)
        cube = _exact_cube(a, nx, ny, edges, c["kernel"], c["sigma"])
        if c["accumulate"]:
            g = torch.Generator(device="cuda")
            g.manual_seed(int(seed) + 1)
            cube += torch.rand((nx, ny, c["nc"]), generator=g, device="cuda")
        return {"cube": cube, "flux": _flux(cube, c["pad"])}
    if kind == "batch":
        cubes, flux = [], []
        for _, a, nx, nc, edges in _batch_inputs(c, seed):
            cube = _exact_cube(a, nx, nx, edges, "wendland_c2", "thermal")
            cubes.append(cube.reshape(-1))
            flux.append(_flux(cube, 0))
        return {"cubes": torch.cat(cubes), "flux": torch.cat(flux)}
    if kind == "profile":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        a = _project(*_disc(g, c["n"], "cuda"), 3.0, 1, 1, c["nc"], c["dv"], "wendland_c2",
                     c["sigma"], prune=False)
        edges = _edges(c["nc"], c["dv"], HUBBLE * 3.0)
        total = torch.zeros(c["nc"], dtype=torch.float64, device="cuda")
        for b in range(0, c["n"], 1 << 18):
            total += _lines({k: t[b:b + (1 << 18)] for k, t in a.items()}, c["sigma"], edges).sum(0)
        return total
    if kind == "beam":
        cube, pad, kern = _beam_inputs(c, seed)
        k = torch.from_numpy(kern.astype(np.float32)).cuda().double()
        nx, ny, nc = c["nx"], c["ny"], c["nc"]
        out = torch.zeros((nx, ny, nc), dtype=torch.float64, device="cuda")
        cube = cube.double()
        m = c["beam"] - 1
        for i in range(c["beam"]):
            for j in range(c["beam"]):
                out.add_(cube[m - i:m - i + nx, m - j:m - j + ny] * k[i, j])
        return out
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    if kind == "martini":
        q = _disc(g, c["n"], "cuda")
        edges = _edges(c["nc"], c["dv"], HUBBLE * 3.0)
        a = _project(*q, 3.0, c["nx"], c["ny"], c["nc"], c["dv"], c["kernel"], "thermal")
        cube = _exact_cube(a, c["nx"], c["ny"], edges, c["kernel"], "thermal")
        return {"cube": cube / PX**2, "flux": cube.sum()}
    # the set-up at the sky position of the source: the same tangent-plane projection in the
    # source's own frame (the cube is centred on the source and its axes turn with it)
    p, v, mhi, h, T = _disc(g, c["n"], "cuda")
    a = _project_sky(p, v, mhi, h, T, c, math.radians(33.0), math.radians(-12.0))
    return {"x": a["x"], "y": a["y"], "sm_range": a["sm_range"], "h_eff": a["h_eff"].double(),
            "kernel_index": None, "v": a["v"], "sigma": a["sigma"].double(), "amp": a["amp"]}


def _project_sky(p, v, mhi, h, T, c, ra, dec):
    """The projection about (ra, dec): the source frame turned by dec about y and ra about z moves
    every particle and the cube's centre alike, so tangent-plane offsets, distances and radial
    velocities are those of the unrotated frame up to that rotation."""
    cd, sd, cr, sr = math.cos(dec), math.sin(dec), math.cos(ra), math.sin(ra)
    rot = torch.tensor([[cd, 0, sd], [0, 1, 0], [-sd, 0, cd]], dtype=torch.float64, device="cuda") \
        @ torch.tensor([[cr, sr, 0], [-sr, cr, 0], [0, 0, 1]], dtype=torch.float64, device="cuda")
    unit = torch.tensor([cd * cr, cd * sr, sd], dtype=torch.float64, device="cuda")
    east = torch.tensor([-sr, cr, 0.0], dtype=torch.float64, device="cuda")
    north = torch.tensor([-sd * cr, -sd * sr, cd], dtype=torch.float64, device="cuda")
    pos = p @ rot + unit * 3e3
    frame = torch.stack((pos @ unit - 3e3, pos @ east, pos @ north), 1)
    vel = v @ rot
    turned = torch.stack((vel @ unit, vel @ east, vel @ north), 1)
    return _project(frame, turned, mhi, h, T, 3.0, c["nx"], c["ny"], c["nc"], c["dv"], c["kernel"],
                    "thermal")
