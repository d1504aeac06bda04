"""The work that a user of this library has it do, as measurable cases through its public entry points: whole sweeps
through `xpg_b200.integrate` and `xpg_b200.batch.integrate_batch`, the per-reflection passes through
`xpg_b200.make_kernels`, the forward model's likelihood passes through `xpg_b200.forward`, and spot finding through
`xpg_b200.spotfind.make_finder`. Everything is synthetic and seeded.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call (frames, reflections, plans), on the GPU; a sweep's
                         crystal is the case's, its intensities and counts are the seed's
    run(state)           one pass, and its outputs
    work(case)           bytes and operations that one pass cannot do without
    exact(case, seed)    the outputs in 64 bits by plain torch, where they follow from the inputs alone
"""
from __future__ import annotations

import math

import numpy as np
import torch

# ------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------

# detectors (px) and cells of this repository's workloads (xpg_b200.synth)
CELLS = {"tetragonal": ((79.0, 79.0, 38.0, 90.0, 90.0, 90.0), "P 43 21 2"),
         "orthorhombic": ((60.0, 85.0, 120.0, 90.0, 90.0, 90.0), "P 21 21 21"),
         "monoclinic": ((150.0, 60.0, 90.0, 90.0, 105.0, 90.0), "C 1 2 1"),
         "small": ((41.3, 52.7, 60.1, 90.0, 90.0, 90.0), "P 21 21 21")}
SIDES = (9, 13, 17, 23, 31, 41, 55)            # shoebox sides and depths the planner gives out
DEPTHS = (3, 5, 9, 17, 33, 65)
VOXELS_MOST = 130e6                            # of one drawn passes case
BOX_VOXELS_MOST = 91e6                         # of one drawn forward-model case


def _sweep(name, nx, ny, frames, block, cell, sigma_m, source, distance=120.0, pixel=0.075, osc=0.1, background=0.2,
           regions=5, parallax=False, adaptive=True, crystal=1):
    named = {} if name is None else dict(name=name)
    return dict(named, kind="sweep", nx=nx, ny=ny, frames=frames, block=block, cell=cell, sigma_m=sigma_m,
                source=source, distance=distance, pixel=pixel, osc=osc, background=background, regions=regions,
                parallax=parallax, adaptive=adaptive, crystal=crystal)


def listed():
    return [
        # a screening wedge on a small detector: what one call costs
        _sweep("sweep-screening", 256, 272, 30, 0, "small", 0.1, "device", distance=80.0, pixel=0.172, osc=0.2,
               background=0.5, regions=3),
        # a 1M-pixel sweep of 100 frames in pinned host memory: frames cross the link inside the call
        _sweep("sweep-1M-host", 1030, 1065, 100, 0, "tetragonal", 0.1, "host", distance=150.0, background=0.5,
               regions=3),
        # a 4M-pixel sweep in HBM as packed bytes, two phi blocks with the widths carried over, deep boxes, a sensor
        # with parallax: the production form of a long sweep, wedge by wedge
        _sweep("sweep-4M-packed", 2068, 2162, 240, 120, "orthorhombic", 0.3, "packed", parallax=True),
        # a 16M-pixel block of raw counts resident in HBM: the large-detector form, hundreds of thousands of boxes
        _sweep("sweep-16M-device", 4148, 4362, 90, 0, "orthorhombic", 0.15, "device"),
        # four 1M-pixel sweeps of different lengths and widths through the batched form (shared persistent launches)
        dict(name="batch-4x1M", kind="batch", sweeps=4, nx=1030, ny=1065, frames=80, sigma_m=0.2),
        # the inner kernel surface on one shoebox shape: small boxes far from the beam's focus (odd count), the common
        # shape of the 16M-pixel detector, and the deep boxes of a mosaic crystal in a crowded lattice
        dict(name="passes-9x9x5", kind="passes", n=40001, side=9, depth=5, neighbours=8, partners=0.05),
        dict(name="passes-31x31x33", kind="passes", n=4096, side=31, depth=33, neighbours=8, partners=0.1),
        dict(name="passes-41x41x65", kind="passes", n=1003, side=41, depth=65, neighbours=16, partners=0.4),
        # the forward model's passes: one chunk of a small window (one term, as the first fit has), and the whole
        # window of a crowded sweep with the halo term
        dict(name="forward-chunk", kind="forward", n=2000, depth=7, side=11, terms=1, frames=16, ny=512, nx=512,
             counts="int32", beta=True),
        dict(name="forward-window", kind="forward", n=60000, depth=9, side=13, terms=2, frames=40, ny=1024, nx=1024,
             counts="int16", beta=False),
        # spot finding: one frame of a 1M-pixel detector (live feedback), and a batch of 16M-pixel frames
        dict(name="spots-1M", kind="spots", frames=1, nx=1030, ny=1065, half=3, extended=True, background=0.5),
        dict(name="spots-16M", kind="spots", frames=4, nx=4148, ny=4362, half=3, extended=True, background=0.2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sweep", "sweep", "batch", "passes", "passes", "forward", "spots"))
    if kind == "sweep":
        nx = _log_int(rng, 256, 4148)
        ny = max(250, min(4362, int(nx * rng.uniform(0.9, 1.1))))
        osc = rng.choice((0.1, 0.2))
        source = rng.choice(("device", "device", "host", "packed", "packed"))
        most = {"device": 50, "packed": 50, "host": 15}[source] * 4148 * 4362 / (nx * ny) * 0.1 / osc
        frames = max(8, min(_log_int(rng, 20, 300), int(most)))
        if source == "packed":                             # packed wedges take frames of a multiple of 4 px
            nx, ny = nx // 2 * 2, ny // 2 * 2
        return _sweep(None, nx, ny, frames, rng.choice((0, max(frames // 2, 10))),
                      rng.choice(("small", "tetragonal", "orthorhombic")) if nx < 2000 else "orthorhombic",
                      round(rng.uniform(0.08, 0.3), 3), source, osc=osc,
                      distance=round(rng.uniform(110.0, 160.0), 1), parallax=rng.random() < 0.3,
                      regions=rng.choice((3, 5)), background=round(rng.uniform(0.1, 1.0), 2),
                      crystal=rng.randint(2, 10 ** 6))
    if kind == "batch":
        return dict(kind="batch", sweeps=rng.randint(2, 5), nx=rng.randint(500, 1100),
                    ny=rng.randint(500, 1100), frames=_log_int(rng, 30, 100), sigma_m=round(rng.uniform(0.08, 0.25), 3))
    if kind == "passes":
        side, depth = rng.choice(SIDES), rng.choice(DEPTHS)
        most = min(40001, VOXELS_MOST / (side * side * depth))
        return dict(kind="passes", n=_log_int(rng, max(16, most / 64), most), side=side, depth=depth,
                    neighbours=rng.choice((4, 8, 12, 16)), partners=round(rng.uniform(0.0, 0.5), 3))
    if kind == "forward":
        depth, side = rng.randint(3, 15), rng.choice((7, 9, 11, 13, 15, 17, 21))
        most = min(60000, BOX_VOXELS_MOST / (depth * side * side))
        return dict(kind="forward", n=_log_int(rng, 500, most), depth=depth, side=side,
                    terms=rng.choice((1, 2)), frames=rng.randint(max(8, depth), 40), ny=_log_int(rng, 256, 1024),
                    nx=_log_int(rng, 256, 1024), counts=rng.choice(("int16", "int32", "float32")),
                    beta=rng.random() < 0.5)
    nx = _log_int(rng, 256, 4148)
    ny = max(256, min(4362, int(nx * rng.uniform(0.8, 1.25))))
    return dict(kind="spots", frames=rng.randint(1, max(1, min(8, int(7.2e7 / (nx * ny))))), nx=nx, ny=ny,
                half=rng.choice((2, 3, 4)), extended=rng.random() < 0.7, background=round(rng.uniform(0.1, 2.0), 2))


# ------------------------------------------------------------------------------------------------------------------
# whole sweeps
# ------------------------------------------------------------------------------------------------------------------

# what the pass kernels compute in float32 and the result table widens to float64: returned as float32 (same values)
F32_COLUMNS = ("bg", "isum", "vsum", "vsum0", "iprf", "vprf", "vprf0", "corr", "xo", "yo", "zo", "p_valid", "p_total",
               "frac_rec", "rho", "m_d", "m_m", "p_fg")


def _spec(case, seed):
    from xpg_b200 import geometry, synth
    cell, group = CELLS[case["cell"]]
    sensor = dict(sensor_thickness=0.45, mu=2.3) if case["parallax"] else {}
    return synth.SweepSpec(name="perf", nx=case["nx"], ny=case["ny"], qx=case["pixel"], distance=case["distance"],
                           wavelength=0.98, osc=case["osc"], nframes=case["frames"], cell=cell, space_group=group,
                           sigma_d=0.03, sigma_m=case["sigma_m"], wilson_b=25.0, mean_i0=50.0,
                           U=geometry.random_orientation(np.random.default_rng(case["crystal"])),
                           background=case["background"], ramp=0.5, seed=1 + int(seed) % 1000003,
                           n_regions_xy=case["regions"], block_frames=case["block"], **sensor)


def _sweep_state(case, seed):
    from xpg_b200 import IntegrationModel, synth
    from xpg_b200 import frames as FR
    spec = _spec(case, seed)
    exp, table = synth.reflection_table(spec)
    if case["source"] == "packed":
        spots = synth.DeviceSpots(spec, table)
        store = FR.pack_generated(lambda k, n, out: spots.render(k + 1, n, out), spec.nframes, spec.ny, spec.nx).to("cuda")
        images = FR.PackedFrames(store, first=1, overload=spec.overload)
    else:
        data = synth.device_frames(spec, table, 1, spec.nframes)
        if case["source"] == "host":
            host = torch.empty(data.shape, dtype=data.dtype, pin_memory=True)
            data = host.copy_(data)
        images = FR.U32Frames(data, first=1, overload=spec.overload)
    edges = spec.block_edges()
    model = IntegrationModel(sigma_d=spec.sigma_d, sigma_m=spec.sigma_m)
    return dict(images=images, blocks=[exp] * (len(edges) - 1), edges=edges, model=model,
                dmin=spec.resolution_limit(), nframes=spec.nframes, regions=spec.n_regions_xy)


def _table(res):
    """The result's reflection table and learnt profiles."""
    out = {k: v.astype(np.float32) if k in F32_COLUMNS else v for k, v in res.refl.items() if isinstance(v, np.ndarray)}
    out["profiles"] = np.stack([res.profiles[b] for b in sorted(res.profiles)])
    return out


def _run_sweep(s):
    import xpg_b200
    res = xpg_b200.integrate(s["images"], s["blocks"], s["edges"], s["model"], s["dmin"], frames=(1, s["nframes"]),
                             n_regions_xy=s["regions"], adaptive=s["adaptive"], verbose=False)
    return _table(res)


def _batch_cases(case):
    """The sweeps of a batched case: lengths from the full one down to a third of it, cells in turn."""
    out = []
    for k in range(case["sweeps"]):
        f = max(12, int(case["frames"] * (1.0 - 0.67 * k / max(case["sweeps"] - 1, 1))))
        out.append(_sweep(None, case["nx"], case["ny"], f, 0, ("orthorhombic", "tetragonal", "monoclinic")[k % 3],
                          round(case["sigma_m"] * (1.0 - 0.1 * k), 4), "device", regions=3, crystal=1 + k))
    return out


def _run_batch(s):
    from xpg_b200.batch import integrate_batch
    return [_batch_rows(r) for r in integrate_batch(s["jobs"])]


def _batch_rows(res):
    """What the batch's user merges: the measurements of every sweep, one array per type."""
    t = _table(res)
    return dict(measured=np.stack([t[k] for k in F32_COLUMNS]),
                counts=np.stack([np.asarray(t[k], np.int64) for k in ("n_over", "n_fg_masked", "isum_raw")]),
                hkl=t["hkl"], profiles=t["profiles"])


def _n_predicted(case):
    """Reflections of a sweep, from its reciprocal volume: a lattice point meets the Ewald sphere twice a turn."""
    spec = _spec(case, 0)
    a, b, c = spec.cell[:3]
    vol = a * b * c * math.sin(math.radians(spec.cell[4]))
    centred = 0.5 if spec.space_group.startswith("C") else 1.0
    return 2.0 * 4.19 * vol * centred / spec.resolution_limit() ** 3 * spec.nframes * spec.osc / 360.0 * 0.6


# ------------------------------------------------------------------------------------------------------------------
# the passes on one shoebox shape
# ------------------------------------------------------------------------------------------------------------------

WAVELENGTH, DISTANCE, PIXEL, OSC = 0.98, 120.0, 0.075, math.radians(0.1)
ORG = (2074.0, 2181.0)
REGIONS = 25
GRID, UMAX = 41, 4.5
GAIN = 1.0


def _wave(x, y):
    """Diffracted wave vector (..., 3) of detector points (pixels), 64 bits."""
    X = torch.stack([(x - ORG[0]) * PIXEL, (y - ORG[1]) * PIXEL, torch.full_like(x, DISTANCE)], -1)
    return X / (X.norm(dim=-1, keepdim=True) * WAVELENGTH)


def _zeta(S):
    s0 = torch.tensor([0.0, 0.0, 1.0 / WAVELENGTH], dtype=torch.float64, device=S.device).expand_as(S)
    e1 = torch.linalg.cross(S, s0)
    return e1[..., 0] / e1.norm(dim=-1)


def _rc_weights():
    w = np.exp(-0.5 * np.linspace(-3.5, 3.5, 21) ** 2 / (1 - 0.25 ** 2))
    return (w / w.sum()).astype(np.float32)


def _passes_inputs(case, seed):
    """Boxes of a 16M-pixel detector's reflections: Wilson intensities, Gaussian spots on a Poisson background, a
    partner's spot beside `partners` of them, neighbours around; some masked columns, overloads, unrecorded frames."""
    n, b, D, K = case["n"], case["side"], case["depth"], case["neighbours"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    f64 = dict(dtype=torch.float64, device="cuda")
    u = lambda *s: torch.rand(*s, generator=gen, **f64)
    x, y = 100.0 + u(4 * n + 64) * 3948.0, 100.0 + u(4 * n + 64) * 4162.0
    ok = torch.nonzero(_zeta(_wave(x, y)).abs() > 0.45)[:n, 0]
    x, y = x[ok], y[ok]
    sigma_px = max((b // 2 - 1) / 5.0, 0.6)
    sd = sigma_px * PIXEL / (1.25 * DISTANCE)
    sm = 0.5 * OSC * max(D - 1, 2) / 9.0
    z = 40.0 + u(n) * 200.0
    phi = z * OSC
    S = _wave(x, y)
    zeta = _zeta(S)
    length = torch.sqrt((x - ORG[0]) ** 2 + (y - ORG[1]) ** 2).mul(PIXEL).square().add(DISTANCE ** 2).sqrt()
    st = length * sd / PIXEL
    sr = st * length / DISTANCE
    sz = sm / zeta.abs() / OSC
    ix0 = (torch.floor(x - 0.5) - b // 2).to(torch.int32)
    iy0 = (torch.floor(y - 0.5) - b // 2).to(torch.int32)
    iz0 = (torch.floor(z) - D // 2).to(torch.int32)
    # neighbours: anywhere within about a box; column 0 is the partner where there is one
    nbx, nby = x[:, None] + (u(n, K) - 0.5) * 4.0 * b, y[:, None] + (u(n, K) - 0.5) * 4.0 * b
    nbz = z[:, None] + (u(n, K) - 0.5) * 4.0 * D
    has_p = u(n) < case["partners"]
    ang = u(n) * 2.0 * math.pi
    nbx[:, 0] = torch.where(has_p, x + 2.5 * st * torch.cos(ang), nbx[:, 0])
    nby[:, 0] = torch.where(has_p, y + 2.5 * st * torch.sin(ang), nby[:, 0])
    nbz[:, 0] = torch.where(has_p, z + (u(n) - 0.5) * sz, nbz[:, 0])
    counts = -torch.log(u(n)) * 400.0
    counts_p = torch.where(has_p, -torch.log(u(n)) * 300.0, torch.zeros_like(counts))
    f32 = lambda t: t.to(torch.float32)
    region = (torch.clamp(y / 4362.0 * 5, 0, 4).long() * 5 + torch.clamp(x / 4148.0 * 5, 0, 4).long()).to(torch.int32)
    rc = dict(S=f32(S), phi=f32(phi), ix0=ix0, iy0=iy0, iz0=iz0, fb=torch.ones(n, device="cuda"), region=region,
              has_p=f32(has_p), pS=f32(_wave(nbx[:, 0], nby[:, 0])), pphi=f32(nbz[:, 0] * OSC))
    nb = dict(x=f32(nbx), y=f32(nby), z=f32(nbz), sx=f32((3.0 * st)[:, None].expand(n, K).contiguous()),
              sz=f32((3.0 * sz)[:, None].expand(n, K).contiguous()))
    sb = torch.empty((n, D, b, b), dtype=torch.float32, device="cuda")
    g32 = torch.arange(b, device="cuda", dtype=torch.float32)
    z32 = torch.arange(D, device="cuda", dtype=torch.float32)
    step = max(1, int(2e7 // (D * b * b)))
    for a in range(0, n, step):
        q = slice(a, min(a + step, n))
        lam = torch.full((sb[q].shape[0], D, b, b), 0.3, device="cuda")
        for cx, cy, cz, c in ((x[q], y[q], z[q], counts[q]), (nbx[q, 0], nby[q, 0], nbz[q, 0], counts_p[q])):
            dx = f32(ix0[q] + 1.0 - cx)[:, None] + g32
            dy = f32(iy0[q] + 1.0 - cy)[:, None] + g32
            rx, ry = f32(cx - ORG[0]), f32(cy - ORG[1])
            rn = torch.sqrt(rx * rx + ry * ry).clamp(min=1e-3)
            rx, ry = (rx / rn)[:, None, None], (ry / rn)[:, None, None]
            ur = dx[:, None, :] * rx + dy[:, :, None] * ry
            ut = dy[:, :, None] * rx - dx[:, None, :] * ry
            s_t, s_r, s_z = f32(st[q])[:, None, None], f32(sr[q])[:, None, None], f32(sz[q])[:, None]
            spot = torch.exp(-0.5 * ((ur / s_r) ** 2 + (ut / s_t) ** 2)) / (2.0 * math.pi * s_r * s_t)
            lo = f32(iz0[q] - cz)[:, None] + z32
            part = 0.5 * (torch.erf((lo + 1.0) / (s_z * 1.41421356)) - torch.erf(lo / (s_z * 1.41421356)))
            lam += (f32(c)[:, None] * part)[:, :, None, None] * spot[:, None]
        sb[q] = torch.poisson(lam, generator=gen)
    bad = u(n)
    sb[bad < 0.03, :, :, b // 3] = -1.0                    # a flagged detector column
    sb[(bad > 0.03) & (bad < 0.04), D // 2, b // 2, b // 2] = -2.0
    sb[bad > 0.98, :max(D // 3, 1)] = -3.0                 # boxes that start before the sweep
    uu = torch.linspace(-UMAX, UMAX, GRID, **f64)
    g2 = uu[None, :] ** 2 + uu[:, None] ** 2
    width = 1.0 + 0.2 * u(REGIONS, 1, 1)
    prof = f32(torch.exp(-0.5 * g2 / width ** 2) / (2.0 * math.pi * width ** 2))
    return dict(sb=sb, rc=rc, nb=nb, prof=prof, sd=sd, sm=sm, rcw=_rc_weights())


def _passes_state(case, seed):
    from xpg_b200 import kernels
    from xpg_b200.geometry import Geometry
    g = Geometry(wavelength=WAVELENGTH, beam=np.array([0.0, 0.0, 1.0]), axis=np.array([1.0, 0.0, 0.0]), orgx=ORG[0],
                 orgy=ORG[1], distance=DISTANCE, ed1=np.array([1.0, 0.0, 0.0]), ed2=np.array([0.0, 1.0, 0.0]),
                 qx=PIXEL, qy=PIXEL, nx=4148, ny=4362, phi0=0.0, osc=math.degrees(OSC))
    s = _passes_inputs(case, seed)
    s["kernels"] = kernels.make_kernels(case["depth"], case["side"], case["side"], REGIONS)
    s["common"] = (kernels.detector_consts(g), g.axis, g.s0, 0.0, OSC, s.pop("sd"), s.pop("sm"), GAIN)
    return s


def _strong(o):
    """The rows that profiles are learnt from, as the integration selects them."""
    return ((o["isum"] > 0) & (o["isum"] / torch.sqrt(o["vsum"].clamp(min=1e-6)) > 10.0) & (o["n_over"] == 0)
            & (o["frac_rec"] > 0.95) & (o["n_fg_nb"] == 0) & (o["n_fg_masked"] == 0))


def _run_passes(s):
    pass1, accumulate_profiles, pass2 = s["kernels"]
    o = pass1(s["sb"], s["rc"], *s["common"], s["prof"], s["nb"], s["rcw"])
    num, den = accumulate_profiles(o["img2"], o["all_valid2"], o["J"], o["u1"], o["u2"], s["rc"]["region"], o["isum"],
                                   _strong(o), o["seff"])
    fit = pass2(s["sb"], s["rc"], *s["common"], s["prof"], o["bg"], o["nbg"], s["nb"], s["rcw"],
                {k: o[k] for k in ("zeta", "J", "u1", "u2", "seff")})
    return dict(moments={k: v for k, v in o.items() if not k.startswith("_")}, num=num, den=den, fit=fit)


# ---- the same in 64 bits, dense over the boxes

def _gradient(f, dim):
    g = torch.empty_like(f)
    n = f.shape[dim]
    at = lambda i: f.narrow(dim, i, 1)
    g.narrow(dim, 1, n - 2).copy_((f.narrow(dim, 2, n - 2) - f.narrow(dim, 0, n - 2)) / 2.0)
    g.narrow(dim, 0, 1).copy_(-1.5 * at(0) + 2.0 * at(1) - 0.5 * at(2))
    g.narrow(dim, n - 1, 1).copy_(0.5 * at(n - 3) - 2.0 * at(n - 2) + 1.5 * at(n - 1))
    return g


def _mapping(S, phi, x, y, lo, hi, sd, sm, rcw):
    """u1, u2, J (rows, y, x), the frames' fractions R (rows, z), zeta and the effective width of reflections S."""
    s0 = torch.tensor([0.0, 0.0, 1.0 / WAVELENGTH], dtype=torch.float64, device=S.device).expand_as(S)
    e1 = torch.linalg.cross(S, s0)
    e1 = e1 / e1.norm(dim=1, keepdim=True)
    e2 = torch.linalg.cross(S, e1)
    e2 = e2 / e2.norm(dim=1, keepdim=True)
    zeta = e1[:, 0]
    side = x.shape[1]
    d = _wave(x[:, None, :].expand(-1, side, -1), y[:, :, None].expand(-1, -1, side)) - S[:, None, None, :]
    norm = S.norm(dim=1)[:, None, None]
    eps1, eps2 = (d * e1[:, None, None, :]).sum(-1) / norm, (d * e2[:, None, None, :]).sum(-1) / norm
    J = (_gradient(eps1, 2) * _gradient(eps2, 1) - _gradient(eps2, 2) * _gradient(eps1, 1)).abs()
    seff = sd * torch.sqrt(1.0 + J[:, side // 2, side // 2] / sd ** 2 / 12.0)
    s = sm / zeta.abs().clamp(min=1e-3)
    sw = (s * 0.25 * math.sqrt(2.0))[:, None, None]
    c = torch.linspace(-3.5, 3.5, 21, dtype=torch.float64, device=S.device) * s[:, None, None]
    part = torch.erf((hi[:, :, None] - phi[:, None, None] - c) / sw) - torch.erf((lo[:, :, None] - phi[:, None, None] - c) / sw)
    R = (0.5 * rcw * part).sum(-1)
    return eps1 / seff[:, None, None], eps2 / seff[:, None, None], J, R, zeta, seff


def _cells(u1, u2):
    f1, f2 = (u1 + UMAX) / 9.0 * (GRID - 1), (u2 + UMAX) / 9.0 * (GRID - 1)
    inside = (f1 >= 0) & (f1 <= GRID - 1) & (f2 >= 0) & (f2 <= GRID - 1)
    f1, f2 = f1.clamp(0, GRID - 1 - 1e-4), f2.clamp(0, GRID - 1 - 1e-4)
    i1, i2 = f1.floor().long(), f2.floor().long()
    t1, t2 = f1 - i1, f2 - i2
    corners = ((i2 * GRID + i1, (1 - t1) * (1 - t2)), (i2 * GRID + i1 + 1, t1 * (1 - t2)),
               ((i2 + 1) * GRID + i1, (1 - t1) * t2), ((i2 + 1) * GRID + i1 + 1, t1 * t2))
    return inside, corners


def _plane(prof, region, u1, u2, J, seff):
    inside, corners = _cells(u1, u2)
    table = prof.double().reshape(REGIONS, -1)[region.long()]
    v = sum(w * table.gather(1, i.flatten(1)).view_as(w) for i, w in corners)
    return torch.where(inside, v, 0.0) * J / (seff ** 2)[:, None, None]


def _in_neighbours(nb, x, y, zz, skip_first):
    m = torch.zeros((x.shape[0], zz.shape[1], y.shape[1], x.shape[1]), dtype=torch.bool, device=x.device)
    for k in range(nb["x"].shape[1]):
        c = {q: v[:, k].double()[:, None] for q, v in nb.items()}
        dx, dy, dz = ((x - c["x"]) / c["sx"]) ** 2, ((y - c["y"]) / c["sx"]) ** 2, ((zz - c["z"]) / c["sz"]) ** 2
        if k == 0 and skip_first is not None:
            dz = torch.where(skip_first[:, None], torch.full_like(dz, 2.0), dz)
        m |= dx[:, None, None, :] + dy[:, None, :, None] + dz[:, :, None, None] < 1.0
    return m


def _exact_rows(s, q):
    """Pass 1, the profile sums and pass 2 of the rows q in 64 bits."""
    rc, nb = {k: v[q] for k, v in s["rc"].items()}, {k: v[q] for k, v in s["nb"].items()}
    c = s["sb"][q].double()
    n, D, b, _ = c.shape
    ar = lambda m: torch.arange(m, dtype=torch.float64, device=c.device)
    x, y = rc["ix0"].double()[:, None] + ar(b) + 1.0, rc["iy0"].double()[:, None] + ar(b) + 1.0
    k0 = rc["iz0"].double()[:, None]
    zz, lo, hi = k0 + ar(D) + 0.5, OSC * (k0 + ar(D)), OSC * (k0 + ar(D) + 1.0)
    rcw = torch.as_tensor(s["rcw"], device=c.device).double()
    S, phi = rc["S"].double(), rc["phi"].double()
    u1, u2, J, R, zeta, seff = _mapping(S, phi, x, y, lo, hi, s["sd"], s["sm"], rcw)
    total = lambda v: v.flatten(1).sum(1)
    col = lambda v: v[:, None, None, None]
    valid, recorded, over = c >= 0, c > -2.5, c == -2.0
    c = torch.where(valid, c, 0.0)
    r2 = u1 ** 2 + u2 ** 2
    fg2 = (r2 <= 9.0)[:, None]
    fgz = (R >= 1e-3 * R.amax(1, keepdim=True) + 1e-6)[:, :, None, None]
    nbm = _in_neighbours(nb, x, y, zz, None)
    clean = valid & ~nbm
    ring = clean & (r2 >= 12.25)[:, None]
    w = ring
    for it in range(5):
        cnt = total(w).double()
        bg = total(torch.where(w, c, 0.0)) / cnt.clamp(min=1e-6)
        if it < 4:
            thr = bg + 3.0 * torch.sqrt(GAIN * bg.clamp(min=0.5)) + 1.0
            w = ring & (c <= col(thr))
    nbg = total(w).double()
    fgv = fg2 & fgz & clean
    net = c - col(bg)
    sums = lambda v: total(torch.where(fgv, v, 0.0))
    nfg, isum, csum = total(fgv).double(), sums(net), sums(c)
    tail = nfg ** 2 * GAIN * bg.clamp(min=1e-3) / nbg.clamp(min=1.0)
    wpos = torch.where(fgv, net.clamp(min=0.0), 0.0)
    sw = total(wpos).clamp(min=1e-6)
    one = dict(bg=bg, nbg=nbg, isum=isum, vsum=GAIN * csum + tail, vsum0=GAIN * nfg * bg + tail,
               xo=total(wpos * x[:, None, None, :]) / sw, yo=total(wpos * y[:, None, :, None]) / sw,
               zo=total(wpos * zz[:, :, None, None]) / sw,
               frac_rec=torch.where(recorded.flatten(2).any(2), R, 0.0).sum(1), nfg=nfg, zeta=zeta, seff=seff, J=J,
               u1=u1, u2=u2, img2=torch.where(fgz & clean, net, 0.0).sum(1),
               fz=torch.where(fg2 & clean, net, 0.0).sum((2, 3)))
    good = _strong(dict(isum=isum, vsum=one["vsum"], frac_rec=one["frac_rec"], n_over=total(over & fg2 & fgz),
                        n_fg_nb=total(fg2 & fgz & nbm), n_fg_masked=total(fg2 & fgz & ~valid & recorded)))
    dens = one["img2"] / isum.clamp(min=1e-6)[:, None, None] / (J / (seff ** 2)[:, None, None]).clamp(min=1e-12)
    inside, corners = _cells(u1, u2)
    take = good[:, None, None] & inside & (clean | ~fgz).all(1)
    base = rc["region"].long()[:, None, None] * GRID * GRID
    num, den = (torch.zeros(REGIONS * GRID * GRID, dtype=torch.float64, device=c.device) for _ in range(2))
    for i, wt in corners:
        num.index_add_(0, (base + i)[take], (wt * dens)[take])
        den.index_add_(0, (base + i)[take], wt[take])
    # pass 2
    has_p = rc["has_p"] > 0.5
    hp = has_p.double()
    p = _plane(s["prof"], rc["region"], u1, u2, J, seff)[:, None] * R[:, :, None, None]
    v1, v2, Jp, Rp, _, seffp = _mapping(rc["pS"].double(), rc["pphi"].double(), x, y, lo, hi, s["sd"], s["sm"], rcw)
    pp = _plane(s["prof"], rc["region"], v1, v2, Jp, seffp)[:, None] * Rp[:, :, None, None] * col(hp)
    del v1, v2, Jp
    nbm = _in_neighbours(nb, x, y, zz, has_p)
    clean = valid & ~nbm
    top, top_p = p.flatten(1).amax(1), pp.flatten(1).amax(1)
    use = clean & ((p > col(0.01 * top)) | (pp > col(0.01 * top_p.clamp(min=1e-12))))
    p_total, p_valid = total(p), total(torch.where(clean, p, 0.0))
    p_fg = total(torch.where(fg2 & fgz, p, 0.0)) / p_total.clamp(min=1e-9)
    p, pp, net = (torch.where(use, v, 0.0) for v in (p, pp, net))
    iv0 = (1.0 / (GAIN * bg.clamp(min=1e-3)))
    a110 = (total(p * p) * iv0).clamp(min=1e-12)
    c0 = total(p) * iv0
    fit = total(net) / (total(p) + total(pp)).clamp(min=1e-6)
    fit_p = fit * hp
    for _ in range(6):
        mu = col(bg) + col(fit.clamp(min=0.0)) * p + col(fit_p.clamp(min=0.0)) * pp
        iv = 1.0 / (GAIN * mu.clamp(min=1e-3))
        a11, b1, a12 = total(p * p * iv), total(p * net * iv), total(p * pp * iv)
        a22 = torch.where(has_p, total(pp * pp * iv), 1.0)
        b2 = total(pp * net * iv)
        det = (a11 * a22 - a12 ** 2).clamp(min=1e-30)
        fit, fit_p = (a22 * b1 - a12 * b2) / det, (a11 * b2 - a12 * b1) / det * hp
    cc = total(torch.where(use, p * iv, 0.0))
    var_b = GAIN * bg.clamp(min=1e-3) / nbg.clamp(min=1.0)
    inv = a22 / det
    two = dict(iprf=fit, vprf=inv + (cc * inv) ** 2 * var_b,
               vprf0=(1.0 / a110 + (c0 / a110) ** 2 * var_b) * (inv * a11).clamp(min=1.0), p_valid=p_valid,
               p_total=p_total, ipartner=fit_p, rho=torch.where(has_p, a12 / torch.sqrt((a11 * a22).clamp(min=1e-30)), 0.0),
               p_fg=p_fg)
    return one, num.view(REGIONS, GRID, GRID), den.view(REGIONS, GRID, GRID), two


def _exact_passes(case, seed):
    s = _passes_inputs(case, seed)
    n = case["n"]
    step = max(1, int(2.5e7 // (case["depth"] * case["side"] ** 2)))
    parts = [_exact_rows(s, slice(a, min(a + step, n))) for a in range(0, n, step)]
    join = lambda k: {q: torch.cat([p[k][q] for p in parts]) for q in parts[0][k]}
    # second moments and the correlation are left out: weak reflections divide by a net sum near zero
    return dict(moments=join(0), num=sum(p[1] for p in parts), den=sum(p[2] for p in parts), fit=join(3))


# ------------------------------------------------------------------------------------------------------------------
# the forward model's passes
# ------------------------------------------------------------------------------------------------------------------

class _Window:
    """The voxels of a window of frames [f0, f1) x detector rectangle, as the forward integrator describes it."""

    def __init__(self, frames, ny, nx):
        self.f0, self.f1, self.y0, self.ny, self.x0, self.nx = 3, 3 + frames, 100, ny, 200, nx


def _forward_state(case, seed):
    """Gaussian spots (and a wider halo) of reflections spread over a window, some of them across its border."""
    n, T, D, b = case["n"], case["terms"], case["depth"], case["side"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    u = lambda *s: torch.rand(*s, generator=gen, device="cuda")
    win = _Window(case["frames"], case["ny"], case["nx"])
    iz0 = win.f0 - D // 2 + (u(n) * (case["frames"] + 1)).long()
    iy0 = win.y0 - b // 2 + (u(n) * (case["ny"] + 1)).long()
    ix0 = win.x0 - b // 2 + (u(n) * (case["nx"] + 1)).long()
    z = torch.arange(D, device="cuda") - D // 2
    xy = torch.arange(b, device="cuda") - b // 2
    R, P = [], []
    for t in range(T):
        sz, sp = D / 7.0 * (1.0 + 0.3 * u(n)), b / 9.0 * (1.0 + 0.2 * u(n)) * (1.0 + t)
        r = torch.exp(-0.5 * ((z + u(n)[:, None] - 0.5) / sz[:, None]) ** 2)
        R.append(r / r.sum(1, keepdim=True))
        gx = torch.exp(-0.5 * ((xy + u(n)[:, None] - 0.5) / sp[:, None]) ** 2)
        gy = torch.exp(-0.5 * ((xy + u(n)[:, None] - 0.5) / sp[:, None]) ** 2)
        p = gy[:, :, None] * gx[:, None, :]
        P.append(p / p.sum((1, 2), keepdim=True) * (0.9 if t == 0 else 0.1))
    I = -torch.log(u(n).clamp(min=1e-6)) * 200.0
    beta = 0.01 * u(n) if case["beta"] else None
    nv = case["frames"] * case["ny"] * case["nx"]
    mu0 = 0.2 + 0.1 * u(nv)
    NS = torch.poisson(mu0 * 1.5, generator=gen)
    NS[u(nv) < 0.02] = -1.0                                # masked voxels
    A, M = NS.clamp(min=0.0), mu0 * (1.0 + u(nv))
    return dict(case=case, win=win, R=torch.stack(R).contiguous(), P=torch.stack(P).contiguous(), I=I, beta=beta,
                iz0=iz0, iy0=iy0, ix0=ix0, rows=torch.randperm(n, generator=gen, device="cuda"), mu0=mu0,
                NS=NS.to(getattr(torch, case["counts"])), A=A, M=M, mu=torch.empty_like(mu0),
                g=torch.zeros((3, n), device="cuda"))


def _run_forward(s):
    """One round of the intensity fit: the model from the intensities, the ratio gradient, the Newton terms."""
    from xpg_b200 import forward
    box = (s["R"], s["P"])
    at = (s["iz0"], s["iy0"], s["ix0"], s["win"])
    s["mu"].copy_(s["mu0"])
    forward.scatter(s["mu"], *box, s["I"], s["beta"], *at)
    s["g"].zero_()
    forward.gather(s["g"][0], None, *box, s["rows"], *at, s["A"], s["M"], s["NS"], 0)
    forward.gather(s["g"][1], s["g"][2], *box, s["rows"], *at, None, s["M"], s["NS"], 1)
    return dict(mu=s["mu"], ratio=s["g"][0], newton=s["g"][1], fisher=s["g"][2])


def _exact_forward(case, seed):
    s = _forward_state(case, seed)
    w, n, D, b = s["win"], case["n"], case["depth"], case["side"]
    mu, M, A = s["mu0"].double(), s["M"].double(), s["A"].double()
    out = torch.zeros((3, n), dtype=torch.float64, device="cuda")
    ar = lambda m: torch.arange(m, device="cuda")
    for a in range(0, n, step := max(1, int(2e7 // (D * b * b)))):
        q = slice(a, min(a + step, n))
        kz, ky, kx = s["iz0"][q, None] - w.f0 + ar(D), s["iy0"][q, None] - w.y0 + ar(b), s["ix0"][q, None] - w.x0 + ar(b)
        inz, iny, inx = (kz >= 0) & (kz < case["frames"]), (ky >= 0) & (ky < w.ny), (kx >= 0) & (kx < w.nx)
        ok = inz[:, :, None, None] & iny[:, None, :, None] & inx[:, None, None, :]
        v = (((kz[:, :, None, None] * w.ny + ky[:, None, :, None]) * w.nx) + kx[:, None, None, :]).where(ok, 0)
        f = torch.einsum("tnz,tnyx->nzyx", s["R"][:, q].double(), s["P"][:, q].double())
        add = f * s["I"][q].double()[:, None, None, None]
        if s["beta"] is not None:
            add = add + s["beta"][q].double()[:, None, None, None]
        mu.index_add_(0, v[ok], add[ok])
        ns = s["NS"][v].double()
        f = torch.where(ok & (ns >= 0), f, 0.0)
        m = M[v]
        at = s["rows"][q]
        out[0].index_add_(0, at, (f * A[v] / m).flatten(1).sum(1))
        out[1].index_add_(0, at, (f * (1.0 - ns.clamp(min=0.0) / m)).flatten(1).sum(1))
        out[2].index_add_(0, at, (f * f / m.clamp(min=1e-6)).flatten(1).sum(1))
    return dict(mu=mu, ratio=out[0], newton=out[1], fisher=out[2])


# ------------------------------------------------------------------------------------------------------------------
# spot finding
# ------------------------------------------------------------------------------------------------------------------

SIGNAL, BACKGROUND, MIN_LOCAL = 3.0, 2.0, 2


def _spots_frames(case, seed):
    """Poisson frames with 3 x 3 px spots (one per 6000 px) and flagged detector columns."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    B, ny, nx = case["frames"], case["ny"], case["nx"]
    img = torch.poisson(torch.full((B, ny, nx), case["background"], device="cuda"), generator=gen)
    k = ny * nx // 6000
    for f in range(B):
        y = torch.randint(5, ny - 5, (k,), generator=gen, device="cuda")
        x = torch.randint(5, nx - 5, (k,), generator=gen, device="cuda")
        c = torch.randint(5, 200, (k,), generator=gen, device="cuda").float()
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                img[f].view(-1).index_add_(0, (y + dy) * nx + x + dx, c)
    img[:, :, ::259] = -1.0
    return img


def _spots_state(case, seed):
    from xpg_b200.spotfind import make_finder
    return dict(img=_spots_frames(case, seed),
                find=make_finder(case["half"], case["half"], SIGNAL, BACKGROUND, MIN_LOCAL, case["extended"]))


def _run_spots(s):
    strong, mean = s["find"](s["img"], 1.0)
    return dict(strong=strong, mean=mean)


def _box_sum(v, h):
    """Sums over the (2h + 1)^2 window, zero outside the frame."""
    k = torch.ones((1, 1, 1, 2 * h + 1), dtype=v.dtype, device=v.device)
    v = torch.nn.functional.conv2d(v[:, None], k, padding=(0, h))
    return torch.nn.functional.conv2d(v, k.transpose(2, 3), padding=(h, 0))[:, 0]


def _exact_spots(case, seed):
    img = _spots_frames(case, seed).double()
    valid = img >= 0
    x = torch.where(valid, img, 0.0)
    n, s1, s2 = _box_sum(valid.double(), case["half"]), _box_sum(x, case["half"]), _box_sum(x * x, case["half"])
    nn = n.clamp(min=2.0)
    mean = s1 / nn
    if not case["extended"]:
        return dict(strong=None, mean=mean)
    var = ((s2 - s1 * mean) / (nn - 1.0)).clamp(min=0.0)
    disp = var > (1.0 + 6.0 * torch.sqrt(2.0 / (nn - 1.0))) * mean.clamp(min=1e-6)
    first = valid & (n >= MIN_LOCAL) & disp & (x - mean > SIGNAL * torch.sqrt(mean.clamp(min=1.0)))
    near = _box_sum(first.double(), 1) > 0.5
    bg = valid & ~near & (img <= mean + BACKGROUND * torch.sqrt(mean.clamp(min=0.5)))
    h = 2 * case["half"] + 1
    return dict(strong=None, mean=_box_sum(torch.where(bg, img, 0.0), h) / _box_sum(bg.double(), h).clamp(min=2.0))


# ------------------------------------------------------------------------------------------------------------------
# the interface
# ------------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        import xpg_b200
        xpg_b200.keep_buffers(True)                        # sweep after sweep on a device of its own
    if kind == "sweep":
        s = _sweep_state(case, seed)
        s["adaptive"] = case["adaptive"]
    elif kind == "batch":
        from xpg_b200.batch import Job
        sweeps = [_sweep_state(c, int(seed) + 7919 * k) for k, c in enumerate(_batch_cases(case))]
        s = dict(jobs=[Job(w["images"], w["blocks"], w["edges"], w["model"], w["dmin"],
                           dict(frames=(1, w["nframes"]), n_regions_xy=w["regions"])) for w in sweeps])
    else:
        s = {"passes": _passes_state, "forward": _forward_state, "spots": _spots_state}[kind](case, seed)
    s["kind"] = kind
    return s


def run(state):
    return {"sweep": _run_sweep, "batch": _run_batch, "passes": _run_passes, "forward": _run_forward,
            "spots": _run_spots}[state["kind"]](state)


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        # every frame read once (a byte a pixel packed, else four), a reflection's 32 results written once
        total = 0.0
        for c in (_batch_cases(case) if kind == "batch" else [case]):
            total += c["nx"] * c["ny"] * c["frames"] * (1.0 if c["source"] == "packed" else 4.0)
            total += 8.0 * 32 * _n_predicted(c)
        return dict(bytes=total, flops=0.0)
    if kind == "passes":
        # a box read once (both passes see the same counts), the per-pixel terms written once, inputs and results;
        # a handful of operations a voxel and pass, six rounds of the fit over about a fifth of the voxels
        n, P, D, K = case["n"], case["side"] ** 2, case["depth"], case["neighbours"]
        return dict(bytes=float(n) * (4 * D * P + 17 * P + 4 * D + 20 * K + 260), flops=float(n) * D * P * (12 + 0.2 * 6 * 10))
    if kind == "forward":
        # the window's model read and written, the counts read, the factors read once by each pass
        nv = case["frames"] * case["ny"] * case["nx"]
        cnt = 2 if case["counts"] == "int16" else 4
        boxes = case["n"] * case["depth"] * case["side"] ** 2
        fac = 4.0 * case["terms"] * case["n"] * (case["depth"] + case["side"] ** 2)
        return dict(bytes=nv * (8.0 + 8.0 + 4.0 + cnt) + 3 * fac + 60.0 * case["n"], flops=boxes * (2.0 * case["terms"] * 3 + 9.0))
    # the frame read once, the mask and the local mean written once
    px = case["frames"] * case["ny"] * case["nx"]
    return dict(bytes=9.0 * px, flops=30.0 * px)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        # profiles and widths are learnt from each block's own reflections and feed the next block: no value of the
        # inputs alone without a second implementation of the whole path, minutes of host time a sweep
        return None
    return {"passes": _exact_passes, "forward": _exact_forward, "spots": _exact_spots}[kind](case, seed)
