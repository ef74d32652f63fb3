"""The work that is timed: what programs that use this library have it do, through its
public entry points, from the smallest calls to the largest frames.

Lenses are the library's seeded prescriptions (a 12-surface double Gauss, a 24-surface
wide angle with two aspheres, an 18-surface decentred and tilted anamorphic with four
cylinders).  Sizes come from the benchmark's workloads, the tests and the defaults of
the configuration classes.  Every random choice comes from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import ghostlight_gb300 as gl
from ghostlight_gb300 import prescriptions as P
from ghostlight_gb300 import starburst as SB
from ghostlight_gb300.flare import filter_ghosts_device

KEYS = ("ghost_r", "ghost_g", "ghost_b", "starburst_r", "starburst_g", "starburst_b", "veil_r", "veil_g", "veil_b")
LENSES = {"dg12": lambda: P.double_gauss_12(seed=1), "wide24": lambda: P.wide_angle_24(seed=2),
          "anam18": lambda: P.anamorphic_18(seed=4)}
N_SURF = {"dg12": 13, "wide24": 24, "anam18": 18}


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # the ghost-pair culler of a new lens: run once per edit in an interactive tool, before a render
        dict(name="cull_wide24", kind="cull", lens="wide24", threshold=1e-6),
        # a batch of single rays along one ghost's path (diagnostics, the survivor scans)
        dict(name="trace_dg12_1m", kind="trace", lens="dg12", rays=1000003, a=2, b=9),
        # the small preview frame: 32^2 pupil samples, 8 wavelengths, 512^2
        dict(name="ghost_dg12_512", kind="ghost", lens="dg12", width=512, height=512, grid=32, adaptive=False,
             spectral=8, sources=1, threshold=0.0, normalize=False, deg=10.0),
        # the full frame the benchmark quotes: adaptive grids 16^2..256^2, 31 wavelengths, 2048^2
        dict(name="ghost_wide24_2048", kind="ghost", lens="wide24", width=2048, height=2048, grid=256, adaptive=True,
             spectral=31, sources=1, threshold=1e-6, normalize=True, deg=15.0),
        # an extended source (five points) at the default 64^2 grid and 16 wavelengths, a video frame
        dict(name="ghost_anam18_5src", kind="ghost", lens="anam18", width=1920, height=1080, grid=64, adaptive=False,
             spectral=16, sources=5, threshold=1e-7, normalize=True, deg=7.0),
        # the starburst precision workload: field form, split-BF16
        dict(name="mdft_split_2048", kind="mdft", form="split_bf16", n=512, kx=2048, ky=2048, spectral=31),
        # the small preview's starburst, on the FP32 form
        dict(name="mdft_fp32_512", kind="mdft", form="fp32", n=256, kx=512, ky=512, spectral=8),
        # the matrix-DFT engine of a flare render: a new source position, its clamped window in the frame
        dict(name="mdft_box_389x301", kind="box", form="split_bf16", grid=1024, fill=0.3, half_x=194, half_y=150,
             width=2048, height=1080, spectral=31),
        # convolution of a frame with a large measured kernel
        dict(name="conv_2048_257", kind="conv", width=2048, height=2048, kw=257, kh=257),
        # the default starburst engine: bake a new pupil's sprite, splat it at a few sources
        dict(name="sprite_2048", kind="sprite", grid=2048, fill=0.3, ds=2, spectral=31, ratio=4.1, width=2048,
             height=2048, sources=3),
        # the default PSF atlas: 8 x 8 tiles of 64^2, Gaussian splat of 4 um
        dict(name="psf_8x8", kind="psf", lens="dg12", nx=8, ny=8, tile=64, grid=64, spectral=16, sigma_um=4.0,
             mono=False, center_mode=0),
        # a whole call: one point source, ghosts + starburst + veil with the default settings, host work included
        dict(name="flare_dg12_1024", kind="flare", lens="dg12", width=1024, height=1024, grid=64, spectral=16,
             engine="sprite", veil=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cull", "trace", "ghost", "ghost", "mdft", "mdft", "box", "conv", "sprite", "psf", "flare"])
    lens = rng.choice(["dg12", "wide24", "anam18"])
    if kind == "cull":
        return dict(kind=kind, lens=lens, threshold=10.0 ** rng.uniform(-8, -5))
    if kind == "trace":
        n = N_SURF[lens]
        a = rng.randrange(0, n - 2)
        b = rng.randrange(a + 1, n)
        if rng.random() < 0.3:
            a = b = -1                                  # primary rays
        return dict(kind=kind, lens=lens, rays=_log(rng, 1, 1000000), a=a, b=b)
    if kind == "ghost":
        w = _log(rng, 160, 2048)
        exact = lens == "dg12" and rng.random() < 0.5
        big = lens == "dg12" or w < 700
        return dict(kind=kind, lens=lens, width=w, height=max(90, int(w * rng.uniform(0.5, 1.0))),
                    grid=_log(rng, 16, 96 if big else 64), adaptive=rng.random() < 0.3, spectral=rng.choice([3, 8, 16, 31]),
                    sources=rng.choice([1, 1, 1, 2, 5]), threshold=0.0 if exact else 10.0 ** rng.uniform(-8, -5),
                    normalize=not exact, deg=rng.uniform(0.0, 18.0))
    if kind == "mdft":
        form = rng.choice(["split_bf16", "split_bf16", "tf32", "fp32"])
        hi = 8 if form == "fp32" else 16
        return dict(kind=kind, form=form, n=128 * rng.randint(1, 3 if form == "fp32" else 4),
                    kx=128 * rng.randint(1, hi), ky=128 * rng.randint(1, hi),
                    spectral=rng.choice([3, 8, 16]) if form == "fp32" else rng.choice([3, 8, 16, 31]))
    if kind == "box":
        return dict(kind=kind, form=rng.choice(["split_bf16", "split_bf16", "tf32", "fp32"]), grid=rng.choice([256, 512, 1024]),
                    fill=rng.choice([0.2, 0.3, 0.45]), half_x=_log(rng, 20, 400), half_y=_log(rng, 20, 300),
                    width=rng.randint(900, 2048), height=rng.randint(700, 1200), spectral=rng.choice([3, 8, 16, 31]))
    if kind == "conv":
        w, h = _log(rng, 100, 2048), _log(rng, 100, 2048)
        return dict(kind=kind, width=w, height=h, kw=2 * _log(rng, 3, 128) + 1, kh=2 * _log(rng, 3, 128) + 1)
    if kind == "sprite":
        n = rng.choice([256, 512, 1024, 2048])
        w = _log(rng, 400, 2048)
        return dict(kind=kind, grid=n, fill=rng.choice([0.3, 0.45]), ds=rng.choice([1, 2, 4]),
                    spectral=rng.choice([3, 8, 16, 31]), ratio=rng.uniform(3.0, 6.0), width=w,
                    height=max(300, int(w * rng.uniform(0.5, 1.0))), sources=rng.randint(1, 8))
    if kind == "psf":
        return dict(kind=kind, lens=rng.choice(["dg12", "wide24"]), nx=rng.randint(1, 8), ny=rng.randint(1, 8),
                    tile=rng.choice([32, 48, 64, 65]), grid=_log(rng, 8, 48), spectral=rng.choice([3, 8, 16]),
                    sigma_um=rng.choice([0.0, 1.5, 4.0, 5.0]), mono=rng.random() < 0.25, center_mode=0)
    w = _log(rng, 256, 1024)
    return dict(kind="flare", lens="dg12", width=w, height=max(200, int(w * rng.uniform(0.5, 1.0))),
                grid=_log(rng, 16, 64), spectral=rng.choice([8, 16]), engine=rng.choice(["sprite", "mdft"]),
                veil=rng.random() < 0.7)


# ---- inputs ------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _lens(name):
    lens = gl.OpticalSystem(LENSES[name](), name=name)
    return lens, gl.calibrate_lens(lens)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 + int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float32)


def _pupil(n, fill, seed, blades=9):
    """(n, n) amplitude in [0, 1]: a bladed stop with an anti-aliased edge and dust discs."""
    r = np.random.default_rng(seed)
    ax = torch.arange(n, device="cuda", dtype=torch.float32) - 0.5 * (n - 1)
    y, x = ax[:, None], ax[None, :]
    rot = float(r.uniform(0.0, 2 * math.pi))
    rad, ang = torch.sqrt(x * x + y * y), torch.atan2(y, x) - rot
    sector = 2 * math.pi / blades
    edge = fill * n * math.cos(math.pi / blades) / torch.cos(torch.remainder(ang, sector) - 0.5 * sector)
    a = torch.clamp((edge - rad) / 2.0 + 0.5, 0.0, 1.0)
    for _ in range(24):
        cx, cy = r.uniform(-fill * n, fill * n, 2)
        d = torch.sqrt((x - float(cx)) ** 2 + (y - float(cy)) ** 2)
        a = torch.minimum(a, torch.clamp(d - float(r.uniform(1.0, 4.0)) + 0.5, 0.0, 1.0))
    return a.contiguous()


def _weights(ns):
    spec, _ = gl.spectral_table(ns)
    return spec


def _mdft_inputs(c, seed):
    """Pupil, scales, centre and weights of a field-form starburst."""
    r = np.random.default_rng(50 + seed)
    spec = _weights(c["spectral"])
    lam = spec[:, 0].astype(np.float64)
    sx, sy = 400.0 / lam / c["kx"], 400.0 / lam / c["ky"]
    w = (spec[:, 1:4].astype(np.float64) * (sx * sy)[:, None]).astype(np.float32)
    centre = (c["kx"] / 2.0 + r.uniform(-0.2, 0.2) * c["kx"], c["ky"] / 2.0 + r.uniform(-0.2, 0.2) * c["ky"])
    return _pupil(c["n"], 0.45, seed), sx, sy, w, centre


def _box_inputs(c, seed):
    """Compact autocorrelation of a pupil, scales, window, centre and tint of one
    source's pixel-integrated starburst (the quantities of mdft_box_starburst_layer)."""
    r = np.random.default_rng(70 + seed)
    N = c["grid"]
    mc = min(int(math.ceil(c["fill"] * N)) + 4, N // 2 - 1)
    n = SB._round128(2 * mc + 1)
    a = _pupil(N, c["fill"] / 2.0, seed).double()
    full = torch.fft.ifft2(torch.fft.fft2(a).abs() ** 2).real
    full = torch.roll(full, (mc, mc), (0, 1))[:2 * mc + 1, :2 * mc + 1] / full[0, 0] / (N * N)
    C = torch.zeros((n, n), device="cuda", dtype=torch.float32)
    C[:2 * mc + 1, :2 * mc + 1] = full.float()
    spec = _weights(c["spectral"])
    lam = spec[:, 0].astype(np.float64)
    sx, sy = 550.0 / lam / (2 * c["half_x"] + 1.3), 550.0 / lam / (2 * c["half_y"] + 1.3)
    w = (spec[:, 1:4] * ((550.0 / lam) ** 2)[:, None]).astype(np.float32)
    px, py = r.uniform(0.1, 0.9) * c["width"], r.uniform(0.1, 0.9) * c["height"]
    x0, x1 = max(0, int(px) - c["half_x"]), min(c["width"], int(px) + c["half_x"] + 1)
    y0, y1 = max(0, int(py) - c["half_y"]), min(c["height"], int(py) + c["half_y"] + 1)
    tint = tuple(float(v) for v in r.uniform(0.5, 1.5, 3))
    K = (SB._round128(min(c["width"], 2 * c["half_x"] + 1)), SB._round128(min(c["height"], 2 * c["half_y"] + 1)))
    return dict(C=C, mc=mc, n=n, sx=sx, sy=sy, w=w, K=K, centre=(px - 0.5 - x0, py - 0.5 - y0), x0=x0, y0=y0,
                ww=x1 - x0, wh=y1 - y0, tint=tint)


def _rays(c, seed):
    """(rays, 7) launches over the front element, a little past its rim, near one field angle, 400..700 nm."""
    lens, _ = _lens(c["lens"])
    g = _gen(seed)
    n = c["rays"]
    R, z = lens.surfaces[0].semi_aperture, lens.surfaces[0].z - 20.0
    u = 2.0 * _rand(g, n, 2) - 1.0
    a = 0.1 * _rand(g, 2)
    d = torch.stack([torch.tan(a[0]).expand(n), torch.tan(a[1]).expand(n), torch.ones(n, device="cuda")], 1)
    o = torch.stack([0.8 * R * u[:, 0] - 20.0 * d[:, 0], 0.8 * R * u[:, 1] - 20.0 * d[:, 1],
                     torch.full((n,), z, device="cuda")], 1)
    d = d / d.norm(dim=1, keepdim=True)
    return torch.cat([o, d, 400.0 + 300.0 * _rand(g, n, 1)], 1).contiguous()


def _ghost_config(c):
    return gl.FlareConfig(ray_grid=c["grid"], spectral_samples=c["spectral"], min_ghost_intensity=c["threshold"],
                          ghost_normalize=c["normalize"], adaptive_grids=c["adaptive"], adaptive_grid_max=max(16, c["grid"]))


def _ghost_sources(c, seed):
    r = np.random.default_rng(90 + seed)
    base = math.radians(c["deg"]) + r.uniform(-0.01, 0.01)
    th = r.uniform(0.0, 0.6)
    src = np.ones((c["sources"], 5), np.float32)
    for i in range(c["sources"]):
        src[i, 0] = base * math.cos(th) + (r.uniform(-0.004, 0.004) if i else 0.0)
        src[i, 1] = base * math.sin(th) + (r.uniform(-0.004, 0.004) if i else 0.0)
        src[i, 2:] = r.uniform(0.5, 1.5, 3)
    return src


def _planes(*shape):
    return [torch.zeros(shape, dtype=torch.float32, device="cuda") for _ in range(3)]


def _sprite_inputs(c, seed):
    r = np.random.default_rng(30 + seed)
    spec = _weights(c["spectral"]).copy()
    spec[:, 1:4] /= spec[:, 1:4].sum(0, keepdims=True)
    M = c["grid"] // c["ds"]
    px = 0.008
    s = px / c["ratio"]
    rx = min(int(math.ceil(0.5 * M * s / px)) + 1, c["width"])
    ry = min(int(math.ceil(0.5 * M * s / px)) + 1, c["height"])
    src = np.stack([[r.uniform(0.1, 0.9) * c["width"], r.uniform(0.1, 0.9) * c["height"], *r.uniform(0.5, 1.5, 3)]
                    for _ in range(c["sources"])]).astype(np.float32)
    return _pupil(c["grid"], c["fill"] / 2.0, seed, 6), spec, M, np.float32(s), np.float32(px), rx, ry, src


def prepare(case, seed):
    c, k = case, case["kind"]
    st = dict(kind=k, case=c)
    if k == "cull":
        lens, cal = gl.OpticalSystem(LENSES[c["lens"]](), name=c["lens"]), _lens(c["lens"])[1]
        lens.surfaces[2].radius *= 1.0 + 0.01 * np.random.default_rng(seed).uniform(-1, 1)     # the edit
        st.update(lens=lens, hw=cal.sensor_half_w, hh=cal.sensor_half_h,
                  config=gl.FlareConfig(min_ghost_intensity=c["threshold"]))
    elif k == "trace":
        st.update(lens=_lens(c["lens"])[0], rays=_rays(c, seed))
    elif k == "ghost":
        lens, cal = _lens(c["lens"])
        st["plan"] = gl.prepare_ghost_render(lens, _ghost_sources(c, seed), c["width"], c["height"], _ghost_config(c),
                                             cal.sensor_half_w, cal.sensor_half_h)
        st["out"] = _planes(c["height"], c["width"])
    elif k == "mdft":
        pupil, sx, sy, w, ctr = _mdft_inputs(c, seed)
        st.update(pupil=pupil, out=_planes(c["ky"], c["kx"]),
                  plan=gl.MdftPlan(c["n"], (c["kx"], c["ky"]), sx, sy, w, c["form"], center_x=ctr[0], center_y=ctr[1]))
    elif k == "box":
        i = _box_inputs(c, seed)
        st.update(inp=i, out=_planes(c["height"], c["width"]),
                  plan=gl.MdftPlan(i["n"], i["K"], i["sx"], i["sy"], i["w"], c["form"], center_x=0.0, center_y=0.0,
                                   box=True, red_center=float(i["mc"])))
    elif k == "conv":
        g = _gen(seed)
        st.update(img=[_rand(g, c["height"], c["width"]) ** 4 for _ in range(3)], out=_planes(c["height"], c["width"]),
                  plan=gl.ConvPlan(c["width"], c["height"], _kernel(c, seed)))
    elif k == "sprite":
        pupil, spec, M, s, px, rx, ry, src = _sprite_inputs(c, seed)
        st.update(pupil=pupil, plan=SB.SpritePlan(c["grid"], spec), s=float(s), px=float(px), rx=rx, ry=ry, src=src,
                  out=_planes(c["height"], c["width"]))
    elif k == "psf":
        lens, cal = _lens(c["lens"])
        r = np.random.default_rng(seed)
        fx, fy = 0.7 * cal.max_half_angle_h, 0.7 * cal.max_half_angle_v
        gx, gy = np.meshgrid(np.linspace(-fx, fx, c["nx"]) if c["nx"] > 1 else [0.3 * fx],
                             np.linspace(-fy, fy, c["ny"]) if c["ny"] > 1 else [0.3 * fy])
        src = np.ones((gx.size, 5), np.float32)
        src[:, 0], src[:, 1] = gx.ravel() + r.uniform(-0.002, 0.002), gy.ravel() + r.uniform(-0.002, 0.002)
        src[:, 2:] = r.uniform(0.5, 1.5, 3)
        st.update(lens=lens, src=src, config=gl.PSFConfig(
            ray_grid=c["grid"], spectral_samples=c["spectral"], grid_nx=c["nx"], grid_ny=c["ny"], tile_w=c["tile"],
            tile_h=c["tile"], monochromatic=c["mono"], splat_sigma_um=c["sigma_um"], center_mode=c["center_mode"]))
    else:
        lens, cal = _lens(c["lens"])
        r = np.random.default_rng(seed)
        dc = gl.DiffractionConfig(starburst=True, veil=c["veil"],
                                  starburst_engine=gl.StarburstEngine.MDFT if c["engine"] == "mdft" else gl.StarburstEngine.SPRITE)
        st.update(lens=lens, cal=cal, config=gl.PointFlareConfig(
            ray_grid=c["grid"], spectral_samples=c["spectral"], source_x=float(r.uniform(0.55, 0.8)),
            source_y=float(r.uniform(0.3, 0.6)), source_g=0.9, source_b=0.8, diffraction=dc))
    return st


def _kernel(c, seed):
    """Seeded smooth radial kernel with noise, unit sum (a measured veil / PSF kernel)."""
    r = np.random.default_rng(200 + seed)
    y, x = np.mgrid[0:c["kh"], 0:c["kw"]].astype(np.float64)
    q = np.hypot((x - c["kw"] // 2) / (0.18 * c["kw"]), (y - c["kh"] // 2) / (0.18 * c["kh"]))
    k = (1.0 / (1.0 + q * q)) ** 1.5 + 0.02 * r.random(q.shape)
    return (k / k.sum()).astype(np.float32)


# ---- one pass ------------------------------------------------------------------
def run(st):
    k, c = st["kind"], st["case"]
    if k == "cull":
        f = filter_ghosts_device(st["lens"], st["hw"], st["hh"], st["config"])
        return {"pairs": f.pairs, "boosts": f.boosts, "footprint": f.footprint_mm}
    if k == "trace":
        return gl.trace_rays(st["lens"], st["rays"], c["a"], c["b"])
    if k == "ghost":
        st["plan"].execute(*st["out"])
        return st["out"]
    if k == "mdft":
        st["plan"].execute(st["pupil"], *st["out"])
        return st["out"]
    if k == "box":
        i = st["inp"]
        st["plan"].set_center(*i["centre"])
        st["plan"].execute_window(i["C"], *st["out"], i["x0"], i["y0"], i["ww"], i["wh"], tint=i["tint"], accumulate=False)
        return st["out"]
    if k == "conv":
        st["plan"].execute(st["img"], st["out"])
        return st["out"]
    if k == "sprite":
        for o in st["out"]:
            o.zero_()
        st["plan"].bake(st["pupil"], c["ds"])
        st["plan"].splat(st["src"], st["s"], st["s"], st["px"], st["px"], st["rx"], st["ry"], 1.0, *st["out"])
        return st["out"]
    if k == "psf":
        o = gl.render_psf(st["src"], st["lens"], st["config"])
        return [o["r"], o["g"], o["b"], o["chief_x_mm"], o["chief_y_mm"], o["status"]]
    o = gl.render_point_flare(c["width"], c["height"], st["lens"], st["cal"], st["config"])
    return {key: o[key] for key in KEYS if key in o}


# ---- what a pass cannot do without -----------------------------------------------
STEP_FLOPS = 60.0     # intersect, clip, bend and weigh one ray at one surface


def work(case):
    c, k = case, case["kind"]
    n = N_SURF.get(c.get("lens"), 0)
    px = 4.0 * c.get("width", 0) * c.get("height", 0)
    if k == "cull":
        return dict(bytes=220.0 * n + 20.0 * n * n / 2, flops=n * n / 2 * 67 * n * STEP_FLOPS)
    if k == "trace":
        steps = n if c["a"] < 0 else n + 2 * (c["b"] - c["a"])
        return dict(bytes=48.0 * c["rays"], flops=0.5 * c["rays"] * steps * STEP_FLOPS)
    if k == "ghost":
        # every pair's own last leg for each pupil sample that the frame keeps; what the legs before
        # it have in common is counted once, which leaves little
        side = c["grid"] * (0.45 if c["adaptive"] else 1.0)
        rays = 0.4 * n * (n - 1) / 2 * c["sources"] * 0.75 * side * side * c["spectral"]
        return dict(bytes=3 * px, flops=rays * (n / 2) * STEP_FLOPS * 0.5)
    if k in ("mdft", "box"):
        if k == "mdft":
            m, kx, ky, out = c["n"], c["kx"], c["ky"], 12.0 * c["kx"] * c["ky"]
            per = 4.0
        else:
            mc = min(int(math.ceil(c["fill"] * c["grid"])) + 4, c["grid"] // 2 - 1)
            m, kx, ky, out = 2 * mc + 1, 2 * c["half_x"] + 1, 2 * c["half_y"] + 1, 3 * px
            per = 2.0
        # even and odd halves about the centre: half of the 2 n^2 K + 4 n K^2 products
        return dict(bytes=4.0 * m * m + out, flops=2.0 * c["spectral"] * 0.5 * (2.0 * m * m * kx + per * m * kx * ky))
    if k == "conv":
        p, q = c["height"] + c["kh"], c["width"] + c["kw"]
        return dict(bytes=6 * px + 8.0 * p * q / 2, flops=2 * 3 * 2.5 * p * q * math.log2(p * q))
    if k == "sprite":
        M = c["grid"] // c["ds"]
        return dict(bytes=4.0 * c["grid"] ** 2 + 12.0 * M * M + 3 * px,
                    flops=10.0 * c["grid"] ** 2 * c["spectral"] + 5.0 * c["grid"] ** 2 * math.log2(c["grid"] ** 2))
    if k == "psf":
        rays = c["nx"] * c["ny"] * 0.75 * c["grid"] ** 2 * (1 if c["mono"] else c["spectral"])
        foot = 4.0 if c["sigma_um"] <= 0 else max(9.0, (5.0 * c["sigma_um"] / (50.0 / c["tile"])) ** 2)
        chan = 1 if c["mono"] else 3
        return dict(bytes=12.0 * c["nx"] * c["ny"] * c["tile"] ** 2, flops=rays * (n * STEP_FLOPS + 2.0 * chan * foot))
    rays = 0.4 * n * (n - 1) / 2 * 0.75 * c["grid"] ** 2 * c["spectral"]
    return dict(bytes=(9 if c["veil"] else 6) * px, flops=rays * (n / 2) * STEP_FLOPS * 0.5)


# ---- the same results in 64 bits ---------------------------------------------------
def exact(case, seed):
    c, k = case, case["kind"]
    if k == "trace" and c["lens"] == "dg12":
        r = _rays(c, seed).double()
        x, y, w, status = _trace64(_lens("dg12")[0], r[:, :3].T, r[:, 3:6].T, r[:, 6], c["a"], c["b"])
        return torch.stack([x, y, torch.zeros_like(x), w, status.double()], 1)
    if k == "ghost" and c["lens"] == "dg12" and not c["normalize"] and c["threshold"] == 0.0 and not c["adaptive"]:
        return _ghost64(c, seed)
    if k == "mdft":
        pupil, sx, sy, w, ctr = _mdft_inputs(c, seed)
        return _mdft64(pupil.double(), (c["n"] - 1) / 2.0, c["kx"], c["ky"], sx, sy, w, ctr, None)
    if k == "box":
        i = _box_inputs(c, seed)
        win = _mdft64(i["C"].double(), float(i["mc"]), i["ww"], i["wh"], i["sx"], i["sy"],
                      i["w"].astype(np.float64) * np.array(i["tint"]), i["centre"], True)
        out = []
        for p in win:
            f = torch.zeros((c["height"], c["width"]), device="cuda", dtype=torch.float64)
            f[i["y0"]:i["y0"] + i["wh"], i["x0"]:i["x0"] + i["ww"]] = p
            out.append(f)
        return out
    if k == "conv":
        g = _gen(seed)
        img = [(_rand(g, c["height"], c["width"]) ** 4).double() for _ in range(3)]
        s = (c["height"] + c["kh"] - 1, c["width"] + c["kw"] - 1)
        K = torch.fft.rfft2(torch.from_numpy(_kernel(c, seed)).cuda().double(), s=s)
        y0, x0 = c["kh"] // 2, c["kw"] // 2
        return [torch.fft.irfft2(torch.fft.rfft2(p, s=s) * K, s=s)[y0:y0 + c["height"], x0:x0 + c["width"]] for p in img]
    if k == "sprite":
        return _sprite64(c, seed)
    # the culler's estimates and the whole call have no closed form; a PSF tile magnifies the rounding of
    # the float32 tile centre to a tenth of a pixel
    return None


def _mdft64(a, cj, kx, ky, sx, sy, w, ctr, box):
    n = a.shape[0]
    out = torch.zeros((3, ky, kx), device="cuda", dtype=torch.float64)
    j = torch.arange(n, device="cuda", dtype=torch.float64) - cj

    def mat(K, s, cen):
        ph = s * torch.outer(torch.arange(K, device="cuda", dtype=torch.float64) - cen, j)
        ph = ph - torch.round(ph)
        m = torch.polar(torch.ones_like(ph), -2 * math.pi * ph)
        return m * torch.sinc(s * j)[None, :] if box else m

    for l in range(len(sx)):
        E = mat(ky, float(sy[l]), ctr[1]) @ (a.to(torch.complex128) @ mat(kx, float(sx[l]), ctr[0]).T)
        I = E.real if box else E.real ** 2 + E.imag ** 2
        for ch in range(3):
            out[ch] += float(w[l][ch]) * I
    return list(out)


def _sprite64(c, seed):
    pupil, spec, M, s, px, rx, ry, src = _sprite_inputs(c, seed)
    N, ds = c["grid"], c["ds"]
    p = torch.fft.fftshift(torch.fft.fft2(pupil.double()).abs() ** 2)
    p = p / p.sum()
    d = torch.arange(N, device="cuda", dtype=torch.float64) - N // 2
    rgb = torch.zeros((3, N, N), device="cuda", dtype=torch.float64)
    for lam, *cmf in spec.astype(np.float64):
        k = 550.0 / lam
        f = N // 2 + d * k
        ok = (f >= 0) & (f < N - 1)
        i0 = f.floor().clamp(0, N - 2).long()
        t = f - i0
        h = p[:, i0] * (1 - t) + p[:, i0 + 1] * t
        v = (h[i0] * (1 - t)[:, None] + h[i0 + 1] * t[:, None]) * (ok[:, None] & ok[None, :]) * k * k
        for ch in range(3):
            rgb[ch] += cmf[ch] * v
    rgb = rgb.reshape(3, M, ds, M, ds).sum((2, 4))
    out = torch.zeros((3, c["height"], c["width"]), device="cuda", dtype=torch.float64)
    s, px = float(s), float(px)
    for sx, sy, *tint in src.astype(np.float64):
        def cover(pos, r, size):
            i = torch.arange(size, device="cuda", dtype=torch.float64)
            lo, hi = (i - pos) * px / s + 0.5 * M, (i + 1 - pos) * px / s + 0.5 * M
            a = torch.arange(M, device="cuda", dtype=torch.float64)
            ov = (torch.minimum(hi[:, None], a + 1) - torch.maximum(lo[:, None], a)).clamp(min=0)
            return ov * ((i - math.floor(pos)).abs() <= r)[:, None]
        for ch in range(3):
            out[ch] += cover(sy, ry, c["height"]) @ rgb[ch] @ cover(sx, rx, c["width"]).T * tint[ch]
    return list(out)


def _ghost64(c, seed):
    lens, cal = _lens("dg12")
    cfg = _ghost_config(c)
    grid = torch.from_numpy(gl.pupil_grid(lens, cfg.ray_grid)).cuda().double()
    spec, corr = gl.spectral_table(max(3, c["spectral"]))
    W, H = c["width"], c["height"]
    acc = torch.zeros((3, H * W), device="cuda", dtype=torch.float64)
    recs = lens.records()
    nd = [1.0] + [float(s.ior) for s in recs]
    pairs = [(a, b) for a in range(len(recs)) for b in range(a + 1, len(recs))
             if abs(nd[a + 1] - nd[a]) >= 1e-3 and abs(nd[b + 1] - nd[b]) >= 1e-3]
    R, z = recs[0].semi_aperture, recs[0].z - 20.0
    for ax, ay, *col in _ghost_sources(c, seed).astype(np.float64):
        bx, by = math.tan(ax), math.tan(ay)
        ln = math.sqrt(bx * bx + by * by + 1.0)
        for lam, *cmf in spec.astype(np.float64):
            o = torch.stack([grid[:, 0] * R - 20.0 * bx, grid[:, 1] * R - 20.0 * by, torch.full_like(grid[:, 0], z)])
            d = torch.tensor([bx / ln, by / ln, 1.0 / ln], device="cuda", dtype=torch.float64)[:, None].expand_as(o)
            lt = torch.full_like(grid[:, 0], lam)
            for a, b in pairs:
                x, y, w, status = _trace64(lens, o, d, lt, a, b)
                px = (x / (2 * cal.sensor_half_w) + 0.5) * W - 0.5
                py = (y / (2 * cal.sensor_half_h) + 0.5) * H - 0.5
                base = w * cfg.flare_gain / len(grid) * (status == 0)
                power = base * sum(u * v for u, v in zip(col, cmf))
                x0, y0 = px.floor(), py.floor()
                for dx in (0, 1):
                    for dy in (0, 1):
                        xi, yi = x0 + dx, y0 + dy
                        wt = (1 - (px - xi).abs()) * (1 - (py - yi).abs())
                        ok = (xi >= 0) & (xi < W) & (yi >= 0) & (yi < H)
                        at = torch.where(ok, yi * W + xi, torch.zeros_like(xi)).long()
                        v = torch.where(ok, power * wt, torch.zeros_like(wt))
                        for ch in range(3):
                            acc[ch].index_add_(0, at, v * cmf[ch])
    if cfg.spectral_correction and c["spectral"] != 3:
        acc = torch.from_numpy(corr).cuda().double() @ acc
    return [acc[ch].reshape(H, W) for ch in range(3)]


def _trace64(lens, o, d, lam, a, b):
    """Rays through spheres and planes with quarter-wave MgF2, along the ghost (a, b) or straight through:
    landing x, y, weight and status (0 landed, 1 missed or clipped, 2 total reflection, 3 away from the sensor)."""
    recs = lens.records()
    ior = []
    for s in recs:
        l2 = (lam * 1e-3) ** 2
        ior.append(torch.sqrt(1.0 + sum(s.sellmeier_B[i] * l2 / (l2 - s.sellmeier_C[i]) for i in range(3)))
                   if s.disp_model == 2 else torch.full_like(lam, float(s.ior)))
    before = [torch.ones_like(lam)] + ior[:-1]
    n = len(recs)
    if b < 0:
        seq = [(i, False, ior[i], None) for i in range(n)]
    else:
        seq = [(i, i == b, ior[i], None) for i in range(b + 1)]
        seq += [(i, i == a, before[i], ior[a]) for i in range(b - 1, a - 1, -1)]
        seq += [(i, False, ior[i], None) for i in range(a + 1, n)]
    o, d = o.clone(), d.clone()
    w, cur = torch.ones_like(lam), torch.ones_like(lam)
    status = torch.full_like(lam, -1.0)                    # -1: still going

    def dead(mask, code):
        nonlocal status
        status = torch.where((status < 0) & mask, torch.full_like(status, code), status)

    for i, reflects, n2, back in seq:
        s = recs[i]
        if not s.is_active:
            continue
        c = 0.0 if abs(s.radius) < 1e-6 else 1.0 / s.radius
        t0 = (s.z - o[2]) / d[2]
        p = o + d * t0
        A, B, Cc = c, c * (p[0] * d[0] + p[1] * d[1]) - d[2], c * (p[0] ** 2 + p[1] ** 2)
        disc = B * B - A * Cc
        den = B + torch.sign(B) * torch.sqrt(disc.clamp(min=0))
        t = t0 - Cc / den
        if c:
            t = torch.where(t > 1e-6, t, t0 - den / A)
        hit = o + d * t
        hx, hy = hit[0] / s.aperture_aspect, hit[1]
        r = torch.sqrt(hx * hx + hy * hy)
        ok = (disc >= 0) & (t > 1e-6) & (r <= s.semi_aperture)
        if s.aperture_shape == 1 and s.aperture_blades >= 3:
            sector = 2 * math.pi / s.aperture_blades
            off = torch.remainder(torch.atan2(hy, hx) - s.aperture_rotation_rad, sector) - 0.5 * sector
            ok = ok & (r <= s.semi_aperture * math.cos(math.pi / s.aperture_blades) / torch.cos(off))
        dead(~ok, 1.0)
        nrm = torch.stack([c * hit[0], c * hit[1], c * (hit[2] - s.z) - 1.0])
        nrm = nrm * -torch.sign((nrm * d).sum(0))
        ci = -(nrm * d).sum(0)
        nr = cur / n2
        s2t = nr * nr * (1 - ci * ci)
        R = _reflectance64(ci, cur, n2, s.ar_layers, lam)
        go = status < 0
        if reflects:
            w = torch.where(go, w * R, w)
            d = d + nrm * (2 * ci)
            cur = cur if back is None else back
        else:
            dead(s2t >= 1, 2.0)
            w = torch.where(status < 0, w * (1 - R), w)
            d = d * nr + nrm * (nr * ci - torch.sqrt((1 - s2t).clamp(min=0)))
            cur = n2
        d = d / d.norm(dim=0)
        o = hit
    ts = -o[2] / d[2]
    dead(~(ts >= 0), 3.0)
    go = status < 0
    zero = torch.zeros_like(w)
    return (torch.where(go, o[0] + d[0] * ts, zero), torch.where(go, o[1] + d[1] * ts, zero), w,
            torch.where(go, zero, status))


def _reflectance64(ci, n1, n2, layers, lam):
    s2t = (n1 / n2) ** 2 * (1 - ci * ci)
    ct = torch.sqrt((1 - s2t).clamp(min=0))
    rs, rp = (n1 * ci - n2 * ct) / (n1 * ci + n2 * ct), (n2 * ci - n1 * ct) / (n2 * ci + n1 * ct)
    bare = torch.where(s2t >= 1, torch.ones_like(ci), 0.5 * (rs * rs + rp * rp))
    if layers <= 0:
        return bare
    nc = 1.38
    s2c = (n1 / nc) ** 2 * (1 - ci * ci)
    cc = torch.sqrt((1 - s2c).clamp(min=0))
    s22 = (nc / n2) ** 2 * (1 - cc * cc)
    c2 = torch.sqrt((1 - s22).clamp(min=0))
    r01, r12 = (n1 * ci - nc * cc) / (n1 * ci + nc * cc), (nc * cc - n2 * c2) / (nc * cc + n2 * c2)
    cd = torch.cos(4 * math.pi * nc * (550.0 / (4 * nc)) * cc / lam)
    film = ((r01 ** 2 + r12 ** 2 + 2 * r01 * r12 * cd) / (1 + (r01 * r12) ** 2 + 2 * r01 * r12 * cd)).clamp(0, 1)
    return torch.where((s2c >= 1) | (s22 >= 1), bare, film * 0.25 ** (layers - 1))
