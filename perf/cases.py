"""The work a program has this library do, as measurable cases.

Each case is one pass through the public entry points (frame renders, lens
sets, the frame server) over the sizes, forms and looks in use: proxies of a
few hundred pixels up to 6144 x 3160 frames, 3 to 31 wavelengths, lenses that
change every frame (cold banks) and lenses that stay (warm banks), the FP32
and the tensor-core / FP16 ("chosen") forms, the Physical and Split looks,
Augment and Preserve energy, scatter, fringe, luma lock, log-encoded sources,
field zones, lens sets and served frames.

`exact` restates the path in 64 bits with torch (discrete decisions, such as
pupil edges and sample positions, in the float32 expressions that define
them) and uses none of the library's code.
"""
import functools
import math

import numpy as np
import torch

from lensdiff_b200 import LensDiffParams
from lensdiff_b200.backend import LensDiffPsfBankCache, image_request
from lensdiff_b200.serving import LensDiffServer

F = np.float32
PI_F = F(3.14159265358979323846)
OUTER = F(0.86)
LUMA = (0.2126, 0.7152, 0.0722)

# RGB weights of the five-bin spectral mode (440..640 nm) and of its
# cyan-magenta style, as a host hands them over.
NATURAL5 = [[0.15863414, 0.0, 0.0, 1.77799344, 1.18257844],
            [0.0, 0.37853149, 1.50904810, 0.53952658, 0.0],
            [2.04875255, 0.45115390, 0.0, 0.0, 0.0]]
STYLE5 = [[0.06493365, 0.05877749, 0.57318610, 1.36540699, 0.51110804],
          [0.17197433, 0.35674790, 1.26974571, 0.60907686, 0.17485593],
          [0.62111682, 0.49386263, 0.68268460, 0.52594876, 0.24511957]]

BASE = {
    "kind": "frame", "width": 1920, "height": 1080, "points": 512, "top": 100.0, "segments": 0,
    "bins": 16,             # wavelengths over 400-700 nm; 1: the Mono mode; 5: the five-bin mode
    "chosen": True,         # the tensor-core / FP16 form, else the FP32 form (the default)
    "cold": True,           # the focus moves every frame, else the lens stays
    "pupil": 512, "radius": 256, "scale_pct": 1.0,
    "blades": 6, "roundness": 0.0, "obstruction": 0.0, "vanes": 0, "rotation": 0.0,
    "noll": 0.0,            # standard deviation of random Noll 2..15 terms, waves
    "chromatic_focus": 0.0,
    "split": False, "preserve": False, "scatter": False, "fringe": False, "style": False, "davinci": False,
    "grid": 0,              # field zones per side (0: none)
}


def _case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    return [
        # Scrubbing a proxy with the plugin's default look: the smallest
        # calls, where launches and host time count.
        _case("proxy_480x270_mono_split_warm", width=480, height=270, points=32, bins=1, chosen=False, cold=False,
              pupil=256, radius=64, scale_pct=24.0, blades=6, roundness=0.5, split=True, preserve=True),
        # A small preview with three wavelengths while the focus is pulled.
        _case("small_1024x576_3wl_cold", width=1024, height=576, points=64, bins=3, pupil=256, radius=128),
        # HD while the focus is pulled: obstructed nine-blade iris, 16
        # wavelengths, streaks and points.
        _case("hd_16wl_cold", segments=16, blades=9, roundness=0.4, obstruction=0.3, vanes=4, noll=0.1),
        # The UHD workload at 31 wavelengths: a new lens every frame, the same
        # lens on every frame (playback), and the default FP32 form.
        _case("uhd_31wl_cold", width=3840, height=2160, points=2048, top=1000.0, bins=31, radius=512,
              chromatic_focus=0.2),
        _case("uhd_31wl_warm", width=3840, height=2160, points=2048, top=1000.0, bins=31, radius=512,
              chromatic_focus=0.2, cold=False),
        _case("uhd_31wl_cold_fp32", width=3840, height=2160, points=2048, top=1000.0, bins=31, radius=512,
              chromatic_focus=0.2, chosen=False),
        # The creative look on a log timeline: five bins, styled with the
        # natural luma kept, Split look, Preserve energy, scatter and fringe.
        _case("hd_styled_split_scatter_cold", bins=5, split=True, preserve=True, scatter=True, fringe=True, style=True,
              davinci=True, radius=216, pupil=256, noll=0.05, roundness=0.3),
        # A ragged crop with aberrations that vary over the field (the
        # reference's 3 x 3 zones), FP32.
        _case("crop_1917x803_zones3_cold_fp32", width=1917, height=803, points=300, bins=9, chosen=False, radius=133,
              pupil=256, grid=3, noll=0.05, blades=7, roundness=0.2),
        # 6K digital cinema, the largest single frame: a kernel radius of 750.
        _case("cinema_6144x3160_31wl_cold", width=6144, height=3160, points=4096, top=1000.0, bins=31, radius=750,
              chromatic_focus=0.2),
        # UHD with an 8 x 8 grid of field zones, each its own bank of 31.
        _case("uhd_zones8_31wl_cold", width=3840, height=2160, points=2048, top=1000.0, bins=31, radius=512,
              chromatic_focus=0.2, grid=8),
        # A contact sheet: the banks of 24 unrelated lenses built together,
        # a thumbnail rendered through each.
        _case("lens_sheet_24", kind="sheet", width=320, height=180, points=24, lenses=24, chromatic_focus=0.2,
              noll=0.1),
        # Served frames of mixed size from host memory, one of them with a
        # lens that changes.
        _case("serve_4_mixed", kind="serve", bins=31, radius=256, chromatic_focus=0.2),
    ]


def _grid_rows(height, radius):
    """The smallest kernel radius from `radius` up whose convolution has a grid:
    the library refuses 649-654 and 1297-1309 rows (frame and kernel reach),
    just above lengths that its transforms have."""
    while 649 <= height + 2 * radius <= 654 or 1297 <= height + 2 * radius <= 1309:
        radius += 1
    return radius


def draw(rng):
    pick = rng.random()
    if pick < 0.1:
        return dict(BASE, kind="sheet", width=rng.randint(160, 400), height=rng.randint(120, 240), points=24,
                    lenses=rng.randint(6, 20), chromatic_focus=0.2, noll=round(rng.uniform(0.02, 0.12), 3))
    height = int(round(math.exp(rng.uniform(math.log(270), math.log(2160)))))
    width = int(round(height * rng.choice([1.333, 1.5, 1.7778, 1.85, 1.896, 2.39]))) + rng.randint(0, 3)
    width = min(width, 4096)
    look = rng.random()
    zones = pick > 0.9
    if zones:
        height, width = min(height, 1080), min(width, 2048)
    short = min(width, height)
    scattered = 0.1 < look < 0.25 and _grid_rows(height, math.ceil(0.015 * short)) == math.ceil(0.015 * short)
    c = dict(BASE, width=width, height=height, points=max(16, width * height // 4096), top=rng.choice([100.0, 1000.0]),
             segments=rng.choice([0, 8]), bins=rng.choice([1, 3, 5, 9, 16, 16, 24, 31, 31]), chosen=rng.random() < 0.6,
             cold=rng.random() < 0.6, pupil=rng.choice([128, 200, 256, 333, 512, 512]),
             radius=_grid_rows(height, max(16, int(short * rng.uniform(0.08, 0.25)))), blades=rng.randint(5, 11),
             roundness=round(rng.random(), 3), obstruction=rng.choice([0.0, 0.0, round(rng.uniform(0.1, 0.4), 3)]),
             vanes=rng.choice([0, 0, 3, 4]), rotation=round(rng.uniform(0.0, 60.0), 2),
             noll=round(rng.uniform(0.0, 0.12), 3), chromatic_focus=rng.choice([0.0, 0.2]),
             preserve=look < 0.35, split=look < 0.2, scatter=scattered, fringe=0.1 < look < 0.3,
             davinci=rng.random() < 0.2, grid=3 if zones else 0)
    if c["bins"] == 5 and rng.random() < 0.5:
        c["style"] = True
    return c


# ---- inputs --------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _frame(width, height, points, top, segments, seed):
    """(H, W, 4) float32: a dim graded background with soft variation, a few
    lamps some pixels wide, point highlights log-uniform in [1, top] and thin
    bright streaks."""
    dev = _device()
    g = torch.Generator(device="cpu").manual_seed(int(seed) * 7919 + 17)
    img = torch.zeros((height, width, 4), dtype=torch.float32, device=dev)
    ramp = torch.linspace(0.0, 0.2, width, device=dev)
    soft = torch.rand((1, 3, 9, 16), generator=g).to(dev) * 0.15
    soft = torch.nn.functional.interpolate(soft, size=(height, width), mode="bilinear", align_corners=True)[0]
    img[..., :3] = ramp[None, :, None] + soft.permute(1, 2, 0)
    img[..., 3] = 1.0
    for _ in range(6):
        cx, cy, r, v = (float(x) for x in torch.rand(4, generator=g))
        cx, cy, r, v = cx * width, cy * height, 1.0 + 0.01 * r * min(width, height), 2.0 + 18.0 * v
        x0, x1 = max(0, int(cx - r)), min(width, int(cx + r) + 1)
        y0, y1 = max(0, int(cy - r)), min(height, int(cy + r) + 1)
        yy = torch.arange(y0, y1, device=dev)[:, None] - cy
        xx = torch.arange(x0, x1, device=dev)[None, :] - cx
        img[y0:y1, x0:x1, :3][(yy * yy + xx * xx) <= r * r] = torch.tensor([v, 0.9 * v, 0.7 * v], device=dev)
    for _ in range(segments):
        x0, y0, x1, y1, v = (float(x) for x in torch.rand(5, generator=g))
        n = 2 * max(width, height)
        t = torch.linspace(0.0, 1.0, n, device=dev)
        px = ((x0 + (x1 - x0) * t) * (width - 1)).long()
        py = ((y0 + (y1 - y0) * t) * (height - 1)).long()
        img[py, px, :3] = 5.0 + 45.0 * v
    xs = torch.randint(0, width, (points,), generator=g)
    ys = torch.randint(0, height, (points,), generator=g)
    # one value per pixel, so that a pixel drawn twice does not depend on the order
    flat, first = np.unique((ys * width + xs).numpy(), return_index=True)
    v = torch.exp(torch.rand(points, generator=g) * math.log(top))[torch.from_numpy(first)].to(dev)
    flat = torch.from_numpy(flat).to(dev)
    tint = 0.7 + 0.3 * torch.rand((flat.numel(), 3), generator=g).to(dev)
    img.view(-1, 4)[flat, :3] = v[:, None] * tint
    return img


def _davinci_encode(x):
    log = (torch.log2(torch.clamp(x, min=0.0) + 0.0075) + 7.0) * 0.07329248
    return torch.where(x <= 0.00262409, x * 10.44426855, log)


def _source(case, seed):
    img = _frame(case["width"], case["height"], case["points"], case["top"], case["segments"], seed)
    if case["davinci"]:
        img[..., :3] = _davinci_encode(img[..., :3].double()).float()
    return img


def _radius_pct(radius, short):
    return (radius - 0.5) * 100.0 / short  # its ceiling in pixels is `radius`


def _lens(case, seed, short):
    """The parameter set of a case as plain values, by the field names of LensDiffParams."""
    rng = np.random.default_rng(int(seed) * 31 + 5)
    b = case["bins"]
    p = dict(lookMode=1 if case["split"] else 0, energyMode=0 if case["preserve"] else 1, effectGain=1.0,
             coreCompensation=0.0, corePreserve=0.1 if case["preserve"] else 0.0, threshold=math.log2(1.0 / 0.18),
             softnessStops=0.5, pointEmphasis=0.0, frameShortSidePx=short, diffractionScalePx=case["scale_pct"],
             phaseMode=1, apertureMode=1, bladeCount=case["blades"], roundness=case["roundness"],
             centralObstruction=case["obstruction"], vaneCount=case["vanes"], vaneThickness=0.02,
             rotationDeg=case["rotation"], pupilResolution=case["pupil"],
             maxKernelRadiusPx=_radius_pct(case["radius"], short), phaseDefocus=0.25 + 0.02 * float(rng.normal()),
             phaseSpherical=0.1 + 0.02 * float(rng.normal()), chromaticFocus=case["chromatic_focus"],
             inputTransfer=1 if case["davinci"] else 0, fftForm=1 if case["chosen"] else 0)
    if case["noll"] > 0.0:
        p["noll"] = [0.0, 0.0] + [float(v) for v in rng.normal(0.0, case["noll"], 14)] + [0.0] * 7
    if b == 1:
        p["spectralMode"] = 0
    elif b == 5:
        p.update(spectralMode=2, rgbMode=0, naturalMatrix=NATURAL5, styleMatrix=STYLE5 if case["style"] else NATURAL5,
                 spectrumForce=0.6 if case["style"] else 0.0, spectrumSaturation=1.1 if case["style"] else 1.0)
    else:
        p.update(spectralMode=3, rgbMode=1, wavelengthsNm=[float(v) for v in np.linspace(400.0, 700.0, b)])
    if case["split"]:
        p.update(coreGain=1.0, structureGain=1.2, coreShoulder=0.0, structureShoulder=40.0)
    if case["scatter"]:
        p.update(scatterAmount=0.3, scatterRadius=1.5)
    if case["fringe"]:
        p.update(creativeFringe=0.2)
    if case["grid"]:
        c = [float(v) for v in rng.normal(0.0, 0.15, 4)]
        p.update(phaseFieldStrength=1.0, phaseFieldComaRadial=c[0], phaseFieldComaTangential=c[1],
                 phaseFieldAstigRadial=c[2], phaseFieldAstigTangential=c[3],
                 fieldGrid=0 if case["grid"] == 3 else case["grid"])
    return p


def _sheet_lenses(case, seed):
    """Unrelated lenses: pupil 128-512, PSF 2-4 times the pupil, 8-31 wavelengths."""
    rng = np.random.default_rng(int(seed) * 101 + 3)
    out = []
    short = min(case["width"], case["height"])
    for _ in range(case["lenses"]):
        pupil = int(rng.integers(128, 513))
        radius = max(8, int(round(float(rng.uniform(2.0, 4.0)) * pupil / 4.0)))
        c = dict(case, pupil=pupil, radius=_grid_rows(case["height"], radius),
                 bins=int(rng.choice([8, 9, 12, 16, 20, 24, 31])), blades=int(rng.integers(5, 10)),
                 roundness=float(rng.uniform(0.0, 1.0)), vanes=int(rng.integers(0, 5)),
                 obstruction=float(rng.choice([0.0, 0.25])), rotation=float(rng.uniform(0.0, 60.0)),
                 scale_pct=100.0 * 12.0 / short)
        out.append(_lens(c, int(rng.integers(0, 1 << 30)), short))
    return out


SERVED = ((1920, 1080), (2048, 1080), (3840, 2160), (1920, 1080))


def _served(case, seed):
    """(frame case, lens) of each served frame: radii 256 px at 1080 rows, 512 at
    2160; the last frame's lens changes from pass to pass."""
    out = []
    for i, (w, h) in enumerate(SERVED):
        c = dict(case, kind="frame", width=w, height=h, points=w * h // 4096, radius=case["radius"] * h // 1080)
        out.append((c, _lens(c, seed + (50 if i == 3 else 0), h)))
    return out


FOCUS_STEP = 1e-3  # waves of defocus per frame of a focus pull


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


def _check(st):
    if not st.ok:
        raise RuntimeError(f"render failed: {st!r}")


def prepare(case, seed):
    if case["kind"] == "serve":
        server = LensDiffServer(0, slots=4)
        jobs = []
        for i, (c, lens) in enumerate(_served(case, seed)):
            src = _source(c, seed + i).cpu().numpy()
            jobs.append([src, LensDiffParams(**lens), np.zeros_like(src)])
        state = {"server": server, "jobs": jobs, "focus": jobs[3][1].phaseDefocus - 4 * FOCUS_STEP, "kind": "serve"}
        for _ in range(4):  # a server renders its sizes once at its start
            run(state)
        return state
    cache = LensDiffPsfBankCache(0)
    src = _source(case, seed)
    stream = _stream()
    if case["kind"] == "sheet":
        lenses = [LensDiffParams(**p) for p in _sheet_lenses(case, seed)]
        dst = torch.zeros((case["lenses"],) + tuple(src.shape), device=src.device)
        torch.cuda.synchronize()
        state = {"kind": "sheet", "cache": cache, "src": src, "dst": dst, "stream": stream, "lenses": lenses,
                 "focus": [p.phaseDefocus - FOCUS_STEP for p in lenses]}
        run(state)
        return state
    params = LensDiffParams(**_lens(case, seed, min(case["width"], case["height"])))
    dst = torch.zeros_like(src)
    torch.cuda.synchronize()
    state = {"kind": "frame", "cache": cache, "src": src, "dst": dst, "stream": stream, "params": params,
             "cold": case["cold"], "focus": params.phaseDefocus}
    if case["cold"]:
        state["focus"] -= FOCUS_STEP
    run(state)  # an instance's first frame: its buffers and calibration
    torch.cuda.synchronize()
    return state


def run(state):
    if state["kind"] == "serve":
        jobs = state["jobs"]
        jobs[3][1].phaseDefocus = state["focus"]
        state["focus"] += FOCUS_STEP
        tickets = [state["server"].submit(src, p, dst)[0] for src, p, dst in jobs]
        for t in tickets:
            _check(state["server"].wait(t)[0])
        return [dst for _, _, dst in jobs]
    cache, src, dst, stream = state["cache"], state["src"], state["dst"], state["stream"]
    if state["kind"] == "sheet":
        for i, p in enumerate(state["lenses"]):
            p.phaseDefocus = state["focus"][i]
            state["focus"][i] += FOCUS_STEP
        _check(cache.build_psf_banks(state["lenses"], stream))
        for i, p in enumerate(state["lenses"]):
            _check(cache.render(image_request(src, dst[i], stream), p))
        return dst
    state["params"].phaseDefocus = state["focus"]
    if state["cold"]:
        state["focus"] += FOCUS_STEP
    _check(cache.render(image_request(src, dst, stream), state["params"]))
    return dst


# ---- what a pass cannot do without ------------------------------------------------
def _lens_sizes(p):
    """(pupil, PSF size, kernel radius) of a parameter set."""
    radius = max(4, math.ceil(p["maxKernelRadiusPx"] * 0.01 * p["frameShortSidePx"]))
    n = min(max(p["pupilResolution"], 64), 1024)
    return n, max(2 * n, 512, 4 * radius), radius


def _wavelengths(p):
    if p["spectralMode"] == 0:
        return [550.0]
    return p.get("wavelengthsNm") or [440.0, 490.0, 540.0, 590.0, 640.0]


def _frame_work(w, h, lens, cold, grid, bank=True):
    """The frame read and written once; for the operations, one transform of
    the driver and one back per output channel on the linear convolution's
    grid and, with a new lens, one PSF transform per wavelength and zone."""
    _, size, radius = _lens_sizes(lens)
    grid_px = (w + 2 * radius) * (h + 2 * radius)
    one = 2.5 * grid_px * math.log2(grid_px)  # a real transform
    parts = 2 if lens["lookMode"] == 1 else 1
    flops = one * (1 + 3 * parts)
    if cold:
        flops += 3 * parts * one
        if bank:
            flops += max(1, grid * grid) * len(_wavelengths(lens)) * 5.0 * size * size * math.log2(size * size)
    return {"bytes": 32.0 * w * h, "flops": flops}


def work(case):
    total = {"bytes": 0.0, "flops": 0.0}
    if case["kind"] == "serve":
        parts = [_frame_work(c["width"], c["height"], lens, i == 3, 0)
                 for i, (c, lens) in enumerate(_served(case, 1))]
    elif case["kind"] == "sheet":
        parts = [_frame_work(case["width"], case["height"], lens, True, 0) for lens in _sheet_lenses(case, 1)]
    else:
        lens = _lens(case, 1, min(case["width"], case["height"]))
        parts = [_frame_work(case["width"], case["height"], lens, case["cold"], case["grid"])]
    for p in parts:
        total = {k: total[k] + p[k] for k in total}
    return total


# ---- the path in 64 bits -------------------------------------------------------
def _coords(n):
    x = ((np.arange(n, dtype=F) + F(0.5)) / F(n) - F(0.5)) * F(2.0)
    nx, ny = np.meshgrid(x, x)
    return nx.astype(F), ny.astype(F)


def _amplitude(p, n, circle):
    nx, ny = _coords(n)
    radius = np.sqrt(nx * nx + ny * ny).astype(F)
    if circle:
        return (radius <= OUTER).astype(np.float64)
    rot = F(p["rotationDeg"] * float(PI_F) / 180.0)
    sides = max(3, p["bladeCount"])
    rnd = F(p["roundness"])
    sector = F(F(2.0) * PI_F / F(sides))
    local = np.fmod((np.arctan2(ny, nx).astype(F) - rot).astype(F), sector).astype(F)
    local = np.where(local < 0, (local + sector).astype(F), local).astype(F)
    local = (local - sector * F(0.5)).astype(F)
    edge = (OUTER * F(np.cos(PI_F / F(sides))) / np.maximum(np.cos(local).astype(F), F(1e-4))).astype(F)
    metric = ((radius / OUTER).astype(F) * rnd + (radius / np.maximum(edge, F(1e-5))).astype(F) * (F(1.0) - rnd)).astype(F)
    keep = (metric <= F(1.0)) & ~(radius < F(F(p["centralObstruction"]) * OUTER))
    thick = F(F(p["vaneThickness"]) * OUTER)
    for i in range(p["vaneCount"]):
        ang = F(rot + F(i) * PI_F / F(p["vaneCount"]))
        cs, sn = F(np.cos(ang)), F(np.sin(ang))
        keep &= ~((np.abs((-nx * sn + ny * cs).astype(F)) <= thick) & (np.abs((nx * cs + ny * sn).astype(F)) <= OUTER))
    return keep.astype(np.float64)


def _phase(p, n, wavelength, zone):
    """Phase in waves: Noll terms on the unit disc of the aperture."""
    c = np.zeros(23)
    c[4] = p["phaseDefocus"] + p["chromaticFocus"] * float((F(wavelength) - F(550.0)) / F(110.0))
    c[11] = p["phaseSpherical"]
    if zone is not None:
        zx, zy = zone
        scale = p["phaseFieldStrength"] * min(1.0, math.hypot(zx, zy) / math.sqrt(2.0))
        ang = math.atan2(zy, zx)
        for rad, tan, jx, jy, m in (("phaseFieldAstigRadial", "phaseFieldAstigTangential", 6, 5, 2),
                                    ("phaseFieldComaRadial", "phaseFieldComaTangential", 8, 7, 1)):
            r, t = p[rad] * scale, p[tan] * scale
            c[jx] += r * math.cos(m * ang) - t * math.sin(m * ang)
            c[jy] += r * math.sin(m * ang) + t * math.cos(m * ang)
    for j, v in enumerate(p.get("noll") or []):
        c[j] += v
    rot = F(p["rotationDeg"] * float(PI_F) / 180.0)
    cs, sn = F(np.cos(-rot)), F(np.sin(-rot))
    nx, ny = _coords(n)
    radius = np.sqrt(nx * nx + ny * ny).astype(F)
    xf = ((nx * cs - ny * sn).astype(F) / OUTER).astype(F)
    yf = ((nx * sn + ny * cs).astype(F) / OUTER).astype(F)
    inside = (radius <= OUTER) & ((xf * xf + yf * yf).astype(F) <= F(1.0))
    x, y = xf.astype(np.float64), yf.astype(np.float64)
    r2, x2, y2 = x * x + y * y, x * x, y * y
    d2 = x2 - y2
    terms = {2: 2 * x, 3: 2 * y, 4: 3 ** 0.5 * (2 * r2 - 1), 5: 6 ** 0.5 * 2 * x * y, 6: 6 ** 0.5 * d2,
             7: 8 ** 0.5 * (3 * r2 - 2) * y, 8: 8 ** 0.5 * (3 * r2 - 2) * x, 9: 8 ** 0.5 * (3 * x2 - y2) * y,
             10: 8 ** 0.5 * (x2 - 3 * y2) * x, 11: 5 ** 0.5 * (6 * r2 * r2 - 6 * r2 + 1),
             12: 10 ** 0.5 * (4 * r2 - 3) * d2, 13: 10 ** 0.5 * (4 * r2 - 3) * 2 * x * y,
             14: 10 ** 0.5 * (x2 * x2 - 6 * x2 * y2 + y2 * y2), 15: 10 ** 0.5 * 4 * x * y * d2}
    out = np.zeros((n, n))
    for j, t in terms.items():
        if c[j] != 0.0:
            out += float(F(c[j])) * t
    return np.where(inside, out, 0.0)


def _psf(amplitude, phase, size, dev):
    """|FFT|^2 of the embedded pupil, centred, of unit sum."""
    n = amplitude.shape[0]
    off = (size - n) // 2
    a = torch.from_numpy(amplitude).to(dev)
    ang = torch.zeros_like(a) if phase is None else torch.from_numpy(phase).to(dev) * (2.0 * math.pi)
    field = torch.zeros((size, size), dtype=torch.complex128, device=dev)
    field[off:off + n, off:off + n] = torch.polar(a, ang)
    spec = torch.view_as_real(torch.fft.fft2(field))
    inten = torch.roll(spec.square().sum(-1), (-(size // 2), -(size // 2)), (0, 1))
    return inten / inten.sum()


def _centre(size):
    return F(size * 0.5) if size % 2 == 0 else F((size - 1) * 0.5)


@functools.lru_cache(maxsize=128)
def _first_zero(n, size):
    """Radius of the first minimum of a clear circle's PSF."""
    dev = _device()
    psf = _psf(_amplitude(None, n, True), None, size, dev)
    top = size // 2
    d = torch.arange(size, dtype=torch.float32, device=dev) - float(_centre(size))
    ring = torch.clamp(torch.floor(torch.sqrt(d[None, :] * d[None, :] + d[:, None] * d[:, None]).double() + 0.5).long(),
                       max=top).view(-1)
    mean = torch.bincount(ring, psf.view(-1), top + 1) / torch.bincount(ring, minlength=top + 1).clamp(min=1)
    prof = mean.cpu().numpy()
    left, right = np.concatenate([prof[:1], prof[:-1]]), np.concatenate([prof[1:], prof[-1:]])
    sm = (left + 2.0 * prof + right) * 0.25

    def refined(i):
        den = sm[i - 1] - 2.0 * sm[i] + sm[i + 1]
        step = 0.0 if abs(den) < 1e-6 else min(max(0.5 * (sm[i - 1] - sm[i + 1]) / den, -0.5), 0.5)
        return max(1.0, i + step)

    best, falls = 1, 1 if sm[1] < sm[0] else 0
    for i in range(2, len(sm) - 1):
        if sm[i] <= sm[i - 1]:
            falls += 1
            best = i if sm[i] < sm[best] else best
        elif falls >= 2:
            return refined(best)
        else:
            best, falls = i, 0
    limit = max(2, min(len(sm) - 1, max(4, size // 8)))
    return refined(1 + int(np.argmin(sm[1:limit + 1])))


def _bilinear(img, x, y):
    lim = img.shape[0] - 1
    bad = (x < 0) | (y < 0) | (x > lim) | (y > lim)
    x, y = torch.where(bad, 0.0, x), torch.where(bad, 0.0, y)
    x0, y0 = torch.floor(x).long(), torch.floor(y).long()
    x1, y1 = torch.clamp(x0 + 1, max=lim), torch.clamp(y0 + 1, max=lim)
    tx, ty = (x - x0.float()).double(), (y - y0.float()).double()
    u = img[y0, x0] + (img[y0, x1] - img[y0, x0]) * tx
    v = img[y1, x0] + (img[y1, x1] - img[y1, x0]) * tx
    return torch.where(bad, 0.0, u + (v - u) * ty)


def _rings(k, dev):
    d = torch.arange(k, dtype=torch.float32, device=dev) - float(F(F(k - 1) * F(0.5)))
    return torch.sqrt(d[None, :] * d[None, :] + d[:, None] * d[:, None])


def _cropped(kernel, radius, rr):
    """The kernel inside `radius` with its boundary taper, of unit sum, on the whole canvas."""
    k = kernel.shape[0]
    c, r = k // 2, min(max(radius, 1), k // 2)
    extent = F(max(1.0, float(r)))
    fade = F(max(F(6.0), min(F(24.0), F(extent * F(0.04)))))
    start = F(max(F(0.0), F(extent - fade)))
    t = torch.clamp((rr - float(start)) / float(fade), 0.0, 1.0)
    s = t * t * (3.0 - 2.0 * t)
    w = torch.where(rr >= float(extent), 0.0, torch.clamp(torch.cos(s * float(F(math.pi * 0.5))), min=0.0)).double()
    box = torch.zeros_like(kernel)
    box[c - r:c + r + 1, c - r:c + r + 1] = (kernel * w)[c - r:c + r + 1, c - r:c + r + 1]
    total = box.sum()
    return box / total if total > 0 else box


def _bank(p, zone, dev):
    """Per wavelength the (full,) or (core, structure) kernels on the canvas."""
    n, size, radius = _lens_sizes(p)
    k = 2 * radius + 1
    r0 = max(1.0, float(F(_first_zero(n, size))))
    base = F(F(max(1.0, p["diffractionScalePx"] * 0.01 * p["frameShortSidePx"])) / F(r0))
    amp = _amplitude(p, n, False)
    rr = _rings(k, dev)
    r_round = torch.clamp(torch.floor(rr.double() + 0.5).long(), max=radius).view(-1)
    r_ceil = torch.clamp(torch.ceil(rr.double()).long(), max=radius).view(-1)
    count = torch.bincount(r_round, minlength=radius + 1)
    d = torch.arange(k, dtype=torch.float32, device=dev) - float(F(F(k - 1) * F(0.5)))
    out = []
    for w in _wavelengths(p):
        psf = _psf(amp, _phase(p, n, w, zone), size, dev)
        inv = F(F(1.0) / max(F(base * F(F(w) / F(550.0))), F(0.05)))
        pos = float(_centre(size)) + d * float(inv)
        sx, sy = pos[None, :].expand(k, k), pos[:, None].expand(k, k)
        if inv <= F(1.0):
            kern = _bilinear(psf, sx, sy)
        else:
            taps = min(max(int(math.ceil(float(inv))), 2), 6)
            step = F(inv / F(taps))
            off = [float(F(F(F(t) + F(0.5)) * step - inv * F(0.5))) for t in range(taps)]
            kern = sum(_bilinear(psf, sx + ox, sy + oy) for oy in off for ox in off) / float(taps * taps)
        kern = kern / kern.sum()
        mean = (torch.bincount(r_round, kern.view(-1), radius + 1) / count.clamp(min=1))[r_round].view(k, k)
        mean = mean / mean.sum()
        # the support that holds the energy and nothing bright outside it
        energy = torch.cumsum(torch.bincount(r_ceil, kern.view(-1), radius + 1), 0).cpu().numpy()
        peak = torch.zeros(radius + 1, dtype=torch.float64, device=dev).scatter_reduce_(
            0, r_ceil, kern.reshape(-1), "amax").cpu().numpy()
        outside = np.concatenate([np.maximum.accumulate(peak[::-1])[::-1][1:], [0.0]])
        ok = (energy / energy[-1] >= float(F(0.9999))) & (outside <= peak.max() * float(F(2e-4)))
        est = max(4, int(np.argmax(ok)) + 1 if ok.any() else radius)
        est += max(6, min(24, int(math.ceil(float(F(F(max(1, est)) * F(0.05)))))))
        support = min(max(est, 4), max(4, radius))
        if p["lookMode"] == 1:
            res = torch.clamp(kern - mean, min=0.0)
            out.append((_cropped(mean, support, rr), _cropped(res / res.sum(), support, rr)))
        else:
            out.append((_cropped(kern, support, rr),))
    return out


def _convolved(planes, kernels):
    """Linear convolutions of planes (n, H, W) with centred kernels (n, K, K), cropped to the plane, not below 0."""
    h, w = planes.shape[-2:]
    k = kernels.shape[-1]
    ph, pw = h + k - 1, w + k - 1
    out = []
    spectra = {}
    for a, b in zip(planes, kernels):
        if a.data_ptr() not in spectra:
            spectra = {a.data_ptr(): torch.fft.rfft2(a, (ph, pw))}
        pad = torch.zeros((ph, pw), dtype=torch.float64, device=a.device)
        pad[:k, :k] = b
        pad = torch.roll(pad, (-(k // 2), -(k // 2)), (0, 1))
        full = torch.fft.irfft2(spectra[a.data_ptr()] * torch.fft.rfft2(pad), (ph, pw))
        out.append(torch.clamp(full[:h, :w], min=0.0))
    return torch.stack(out)


def _mapped(p, planes, kernel_sets):
    """The RGB effect (3, H, W) of one kernel per wavelength: planes is the scalar
    driver (spectral modes) or the three colours (Mono).  The weights are
    applied to the kernels, which the convolution is linear in."""
    dev = planes.device
    lum = torch.tensor(LUMA, dtype=torch.float64, device=dev)
    if p["spectralMode"] == 0:
        return _convolved(planes, kernel_sets[0].expand(3, -1, -1))
    wl = np.array(_wavelengths(p), np.float64)
    if p["rgbMode"] == 1:
        nat = np.stack([np.exp(-0.5 * ((wl - c) / 40.0) ** 2) for c in (600.0, 540.0, 450.0)])
        nat = sty = nat / nat.sum(axis=1, keepdims=True)
    else:
        nat, sty = np.array(p["naturalMatrix"]), np.array(p["styleMatrix"])
    force = float(F(p.get("spectrumForce", 0.0)))
    mix = nat * (1.0 - force) + sty * force
    stack = torch.stack(kernel_sets)
    kern = torch.einsum("cb,bij->cij", torch.from_numpy(mix).to(dev), stack)
    rgb = _convolved(planes[:1].expand(3, -1, -1), kern)
    gray = torch.einsum("c,cij->ij", lum, rgb)
    rgb = gray + (rgb - gray) * float(F(p.get("spectrumSaturation", 1.0)))
    nat_luma = torch.from_numpy(np.array(LUMA) @ nat).to(dev)
    target = _convolved(planes[:1], torch.einsum("b,bij->ij", nat_luma, stack)[None])[0]
    cur = torch.einsum("c,cij->ij", lum, rgb)
    return rgb * torch.where(cur > 1e-6, target / torch.where(cur > 1e-6, cur, 1.0), 1.0)


def _shoulder(v, s):
    return v if s <= 0 else s * (1.0 - torch.exp(-torch.clamp(v, min=0.0) / s))


def _effect(p, planes, zone, dev):
    bank = _bank(p, zone, dev)
    if p["lookMode"] == 1:
        core = _shoulder(_mapped(p, planes, [b[0] for b in bank]), float(F(p["coreShoulder"])))
        struct = _shoulder(_mapped(p, planes, [b[1] for b in bank]), float(F(p["structureShoulder"])))
        return core * p["coreGain"] + struct * p["structureGain"]
    return _mapped(p, planes, [b[0] for b in bank])


def _tent(extent, z, n, dev):
    pos = torch.arange(extent, dtype=torch.float32, device=dev) / float(max(1, extent - 1)) * float(n - 1)
    return torch.clamp(1.0 - (pos - float(z)).abs(), min=0.0).double()


def _clamped(plane, x, y):
    h, w = plane.shape
    x, y = torch.clamp(x, 0.0, w - 1.0), torch.clamp(y, 0.0, h - 1.0)
    x0, y0 = torch.floor(x).long(), torch.floor(y).long()
    x1, y1 = torch.clamp(x0 + 1, max=w - 1), torch.clamp(y0 + 1, max=h - 1)
    tx, ty = (x - x0.float()).double(), (y - y0.float()).double()
    a = plane[y0, x0] * (1.0 - tx) + plane[y0, x1] * tx
    b = plane[y1, x0] * (1.0 - tx) + plane[y1, x1] * tx
    return a * (1.0 - ty) + b * ty


def _rendered(src, p, grid):
    """The whole frame in 64 bits."""
    dev = src.device
    lum = torch.tensor(LUMA, dtype=torch.float64, device=dev)
    h, w = src.shape[:2]
    rgb = src[..., :3].double().permute(2, 0, 1)
    if p["inputTransfer"] == 1:
        rgb = torch.where(rgb <= 0.02740668, rgb / 10.44426855, torch.exp2(rgb / 0.07329248 - 7.0) - 0.0075)
    signal = rgb.amax(0)
    soft, thr = F(p["softnessStops"]), F(p["threshold"])
    e0, e1 = float(F(thr - soft * F(0.5))), float(F(thr + soft * F(0.5)))
    t = torch.clamp((torch.log2(torch.clamp(signal, min=1e-6) / float(F(0.18))) - e0) / max(e1 - e0, 1e-4), 0.0, 1.0)
    mask = torch.where(signal > 0, t * t * (3.0 - 2.0 * t), 0.0)
    keep = float(F(min(max(p["corePreserve"], 0.0), 1.0)))
    rscale = 1.0 - keep
    max_sub = (1.0 - max(0.2, keep)) / rscale
    redist = rgb * (mask * rscale)
    planes = redist if p["spectralMode"] == 0 else (signal * mask * rscale)[None]
    if grid:
        effect = torch.zeros((3, h, w), dtype=torch.float64, device=dev)
        for zy in range(grid):
            for zx in range(grid):
                zone = (2.0 * zx / (grid - 1) - 1.0, 2.0 * zy / (grid - 1) - 1.0)
                weight = _tent(h, zy, grid, dev)[:, None] * _tent(w, zx, grid, dev)[None, :]
                effect += _effect(p, planes, zone, dev) * weight
    else:
        effect = _effect(p, planes, None, dev)
    gain, comp = p["effectGain"], p["coreCompensation"]
    if p["energyMode"] == 0:
        gain = comp = min(max(gain, 0.0), 1.0)
        e_in, e_fx = (float(torch.einsum("c,cij->", lum, v)) for v in (redist, effect))
        effect = effect * (e_in / e_fx) if e_fx > 1e-6 else effect
    short = p["frameShortSidePx"]
    scatter = p.get("scatterRadius", 0.0) * 0.01 * short
    if p.get("scatterAmount", 0.0) > 1e-6 and scatter > 0.25:
        r = F(scatter)
        rad, sigma = max(1, int(math.ceil(max(0.5, float(r))))), max(F(0.5), F(r * F(0.5)))
        a = torch.arange(-rad, rad + 1, device=dev, dtype=torch.float64)
        g = torch.exp(-(a[None, :] ** 2 + a[:, None] ** 2) / float(F(2.0) * sigma * sigma))
        effect = effect + _convolved(effect, (g / g.sum()).expand(3, -1, -1)) * float(F(p["scatterAmount"]))
    fringe = F(p.get("creativeFringe", 0.0) * 0.01 * short)
    if fringe > F(1e-6):
        x = torch.arange(w, dtype=torch.float32, device=dev)[None, :].expand(h, w)
        y = torch.arange(h, dtype=torch.float32, device=dev)[:, None].expand(h, w)
        dx, dy = x - 0.5 * (w - 1), y - 0.5 * (h - 1)
        length = torch.sqrt(dx * dx + dy * dy)
        inv = torch.where(length > 1e-6, 1.0 / length, 0.0)
        shx, shy = dx * inv * float(fringe), dy * inv * float(fringe)
        effect = torch.stack([_clamped(effect[0], x + shx, y + shy), effect[1], _clamped(effect[2], x - shx, y - shy)])
    out = torch.maximum(torch.clamp(rgb - comp * redist + gain * effect, min=0.0),
                        torch.clamp(rgb - redist * max_sub, min=0.0))
    if p["inputTransfer"] == 1:
        out = _davinci_encode(out)
    return torch.cat([out.permute(1, 2, 0), src[..., 3:].double()], dim=-1)


def exact(case, seed):
    if case["kind"] == "serve":
        return [_rendered(_source(c, seed + i), lens, 0).cpu().numpy() for i, (c, lens) in enumerate(_served(case, seed))]
    src = _source(case, seed)
    if case["kind"] == "sheet":
        return torch.stack([_rendered(src, lens, 0) for lens in _sheet_lenses(case, seed)])
    return _rendered(src, _lens(case, seed, min(case["width"], case["height"])), case["grid"])
