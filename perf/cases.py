"""The work that users of the imager have it do, as measurable cases.

Every case goes through the public Python layer (``sarbp.Context``), which is
the C ABI.  The cases cover back-projection of resident range-compressed data
(both storages, both phase forms, corrections, accumulation), the whole
``image`` call from device and from pinned host memory, the weighted
projection, range compression (both storages, single-CTA and split transform
lengths) and the omega-K imager.  Sizes are the repository's own workloads
(config 1, config 2, a config-5 sub-aperture, the RADARSAT-1 scene) and ragged
ones between them.

Inputs are made with torch from the seed alone: point targets on band-limited
clutter, seen along a straight or a curved track.
"""
import functools
import math

import numpy as np
import torch

from sar_cambrianaccelerationcard_gb300 import sarbp, scenes

RADAR = scenes.Radar()          # C band, 100 MHz, fs 120 MHz, 8x upsampling, 5 km
MAX_UPDATES = 4096 ** 3         # config 2: the largest call
EXACT_UPDATES = 12e9            # FP64 back-projection in torch stays within seconds


def listed():
    return [
        # one small tile of a short aperture: a quick-look or one served request; latency
        dict(name="bp_tile", kind="bp", np=256, ns=1024, nx=128, ny=128, spacing=0.25, angle=0.0, fp16=False,
             curved=False, corr=False, accumulate=False),
        # config 2, the headline workload: 4096 pulses onto 4096^2 at 0.25 m
        dict(name="bp_config2", kind="bp", np=4096, ns=8192, nx=4096, ny=4096, spacing=0.25, angle=0.0, fp16=False,
             curved=False, corr=False, accumulate=False),
        # a sub-aperture of config 5 added into a ragged tile: FP16 rows, curved track, 131072 bins per pulse
        dict(name="bp_fp16_subaperture", kind="bp", np=1500, ns=16384, nx=1501, ny=2203, spacing=0.25, angle=0.0,
             fp16=True, curved=True, corr=False, accumulate=True),
        # a coarse, rotated grid (linear-term phase form) with motion-compensation corrections
        dict(name="bp_coarse_corrected", kind="bp", np=1024, ns=8192, nx=1200, ny=1000, spacing=0.75, angle=25.0,
             fp16=False, curved=True, corr=True, accumulate=False),
        # config 1 as one call on device buffers: range compression + back-projection
        dict(name="image_config1", kind="image", np=512, ns=1024, nx=512, ny=512, spacing=0.5, angle=0.0, fp16=False,
             curved=False, host=False),
        # the whole call from and to pinned host memory, FP16 rows (config 3's mode), odd sizes
        dict(name="image_host_fp16", kind="image", np=1111, ns=4000, nx=1000, ny=1030, spacing=0.3, angle=0.0,
             fp16=True, curved=False, host=True),
        # the adjoint that drives autofocus
        dict(name="project", kind="project", np=2048, ns=4096, nx=1024, ny=777, spacing=0.25, angle=0.0, fp16=False,
             curved=True, corr=True),
        # range compression of config 1: a few hundred short pulses
        dict(name="rc_config1", kind="rc", np=512, ns=1024, fp16=False),
        # range compression of config 2: 16384-point transforms, complex64 rows
        dict(name="rc_config2", kind="rc", np=4096, ns=8192, fp16=False),
        # odd pulse and sample counts, 8192-point transforms, FP16 rows and scales
        dict(name="rc_fp16_odd", kind="rc", np=1537, ns=5003, fp16=True),
        # a slice of config 5's range compression: 32768-point transforms, FP16 rows
        dict(name="rc_config5_slice", kind="rc", np=768, ns=16384, fp16=True),
        # the omega-K image of the RADARSAT-1 scene (3072 x 2048 padded to 4096 x 3414)
        dict(name="wk_radarsat1", kind="wk", na=3072, nr=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bp", "bp", "bp", "image", "project", "rc", "rc", "wk"])
    if kind == "rc":
        ns = _log(rng, 700, 16384)
        return dict(kind="rc", np=_log(rng, 64, max(65, min(4096, 4096 * 8192 // ns))), ns=ns,
                    fp16=rng.random() < 0.5)
    if kind == "wk":
        return dict(kind="wk", na=_log(rng, 300, 3072), nr=_log(rng, 200, 2048))
    ns = _log(rng, 1024, 16384)
    ns -= ns % 4 if rng.random() < 0.5 else 0
    n_p = _log(rng, 128, max(129, min(4096, 4096 * 8192 // ns)))
    top = 1024 if kind == "project" else 4096
    nx, ny = _log(rng, 64, top), _log(rng, 64, top)
    if n_p * nx * ny > MAX_UPDATES // 2:
        n_p = max(128, MAX_UPDATES // 2 // (nx * ny))
    c = dict(kind=kind, np=n_p, ns=ns, nx=nx, ny=ny, spacing=round(rng.uniform(0.2, 0.8), 3),
             angle=rng.choice([0.0, 0.0, round(rng.uniform(-60.0, 60.0), 1)]), fp16=rng.random() < 0.4,
             curved=rng.random() < 0.5)
    if kind == "image":
        c["host"] = rng.random() < 0.5
    else:
        c["corr"] = rng.random() < 0.4
    if kind == "bp":
        c["accumulate"] = rng.random() < 0.3
    return c


# ------------------------------------------------------------------ scenes

@functools.cache
def _context():
    """One context for the process, as a program keeps it."""
    return sarbp.Context(0)


def _grid(case):
    a = math.radians(case["angle"])
    ux = case["spacing"] * np.array([math.sin(a), math.cos(a), 0.0])
    uy = case["spacing"] * np.array([math.cos(a), -math.sin(a), 0.0])
    nx, ny = case["nx"], case["ny"]
    origin = np.array([0.0, RADAR.r0, 0.0]) - (nx // 2) * ux - (ny // 2) * uy
    return scenes.Grid(origin=origin, ux=ux, uy=uy, nx=nx, ny=ny)


def _track(case, seed):
    return scenes.curved_track(RADAR, case["np"], seed=seed) if case.get("curved") \
        else scenes.straight_track(RADAR, case["np"])


def _targets(case, seed, n=10):
    if "nx" in case:
        return scenes.random_targets(_grid(case), n, seed)
    rng = np.random.default_rng(seed)  # range compression alone: targets anywhere in the record
    span = 0.4 * case["ns"] / RADAR.fs * RADAR.c / 2.0
    return np.column_stack([rng.uniform(-50, 50, n), RADAR.r0 + rng.uniform(-span, span, n), np.zeros(n),
                            rng.rayleigh(1.0, n)])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _noise(shape, gen):
    """Circular complex normal samples of unit variance."""
    x = torch.randn(*shape, 2, device="cuda", generator=gen)
    return torch.view_as_complex(x.mul_(math.sqrt(0.5)))


def _cis(cycles):
    """exp(2 pi j cycles) in complex64 of FP64 cycles."""
    a = (2.0 * math.pi) * (cycles - torch.round(cycles)).float()
    return torch.complex(torch.cos(a), torch.sin(a))


def _delays(apc, targets):
    a, t = torch.as_tensor(apc, device="cuda"), torch.as_tensor(targets[:, :3], device="cuda")
    return 2.0 * torch.linalg.norm(a[:, None, :] - t[None, :, :], dim=2) / RADAR.c  # [np][targets]


def _record_start(ns):
    return scenes.centred_record_start(RADAR, ns)


def _echo(case, seed):
    """Point-target echo [np][ns] complex64 at 20 dB SNR."""
    n_p, ns = case["np"], case["ns"]
    tg = _targets(case, seed)
    tau = _delays(_track(case, seed), tg)
    t = _record_start(ns) + torch.arange(ns, device="cuda", dtype=torch.float64) / RADAR.fs
    echo = _noise((n_p, ns), _gen(seed)).mul_(0.1)
    step = max(1, (1 << 24) // ns)
    for p in range(0, n_p, step):
        for k in range(len(tg)):
            u = t[None, :] - tau[p:p + step, k, None]
            x = _cis(0.5 * RADAR.kr * (u - RADAR.tp / 2.0) ** 2 - RADAR.fc * tau[p:p + step, k, None])
            echo[p:p + step] += tg[k, 3] * x * ((u >= 0.0) & (u < RADAR.tp))
    return echo


def _rows(case, seed):
    """Range-compressed rows [np][8 ns] complex64 as the matched filter leaves
    them: band-limited target responses on band-limited clutter, upsampled by
    zero insertion; FP16 rows with their power-of-two scales where the case has them."""
    n_p, ns = case["np"], case["ns"]
    lay = scenes.rc_layout(RADAR, ns, _record_start(ns))
    n, up = lay.nfft, RADAR.upsample
    tg = _targets(case, seed)
    tau = _delays(_track(case, seed), tg)
    k = torch.arange(n, device="cuda")
    f = torch.where(k < n // 2, k, k - n).double() * (RADAR.fs / n)
    band = (f.abs() <= RADAR.bandwidth / 2).float()
    gen = _gen(seed)
    rows = torch.empty(n_p, lay.nbins, dtype=torch.complex64, device="cuda")
    scale = torch.ones(n_p, device="cuda")
    half = torch.empty(n_p, lay.nbins, 2, dtype=torch.float16, device="cuda") if case["fp16"] else None
    step = max(1, (1 << 21) // n)
    for p in range(0, n_p, step):
        m = min(step, n_p - p)
        y = _noise((m, n), gen).mul_(0.1 * math.sqrt(n))
        for j in range(len(tg)):
            d = tau[p:p + m, j, None]
            y += float(tg[j, 3]) * _cis(-f[None, :] * (d - lay.t0_bins) - RADAR.fc * d)
        y *= band * (1200.0 / n)
        z = torch.zeros(m, up * n, dtype=torch.complex64, device="cuda")
        z[:, :n // 2] = y[:, :n // 2]
        z[:, up * n - n // 2:] = y[:, n // 2:]
        x = torch.fft.ifft(z, norm="forward")[:, :lay.nbins]
        if half is None:
            rows[p:p + m] = x
        else:
            sc = torch.exp2(torch.ceil(torch.log2(y.abs().sum(1)) - 14.0))
            scale[p:p + m] = sc
            half[p:p + m] = torch.view_as_real(x / sc[:, None]).half()
    return (rows, None, lay) if half is None else (half, scale, lay)


def _corrections(case, seed):
    """Per-pulse range (m) and phase (rad) corrections of a motion-compensation solution."""
    if not case.get("corr"):
        return None, None
    rng = np.random.default_rng(seed + 1)
    p = np.arange(case["np"])
    return 0.2 * np.sin(2 * np.pi * p / 700.0) + rng.normal(0, 0.01, len(p)), rng.normal(0, 0.3, len(p))


def _wk_params():
    return sarbp.WkParams(fr=32317000.0, prf=1256.98, f0=5.3e9, r0=988647.462, kr=-721350000000.0, c=299790000.0,
                          vr=7062.0, f_nc=-6900.0, taps=6)


# --------------------------------------------------------------- the cases

def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "wk":
        s["params"] = _wk_params()
        s["echo"] = _noise((case["na"], case["nr"]), _gen(seed))
        na, nr, _ = ctx.wk_padded_size(case["na"], case["nr"])
        s["image"] = torch.empty(na, nr, dtype=torch.complex64, device="cuda")
        return s
    s["radar"] = sarbp.radar_struct(RADAR, _record_start(case["ns"]))
    if kind == "rc":
        n_p, ns = case["np"], case["ns"]
        s["echo"] = _echo(case, seed)
        if case["fp16"]:
            s["out"] = torch.empty(n_p, RADAR.upsample * ns, 2, dtype=torch.float16, device="cuda")
            s["scale"] = torch.empty(n_p, device="cuda")
        else:
            s["out"] = torch.empty(n_p, RADAR.upsample * ns, dtype=torch.complex64, device="cuda")
        return s
    s["grid"] = sarbp.grid_struct(_grid(case))
    s["mode"] = sarbp.MODE_FP16STORE if case["fp16"] else sarbp.MODE_SPLIT
    apc = _track(case, seed)
    shape = (case["ny"], case["nx"])
    if kind == "image":
        echo = _echo(case, seed)
        s["image"] = torch.empty(shape, dtype=torch.complex64, device="cpu" if case["host"] else "cuda",
                                 pin_memory=case["host"])
        if case["host"]:
            s["echo"], s["apc"] = echo.cpu().pin_memory(), apc
        else:
            s["echo"], s["apc"] = echo, torch.as_tensor(apc, device="cuda")
        return s
    s["apc"] = torch.as_tensor(apc, device="cuda")
    s["rows"], s["scale"], s["lay"] = _rows(case, seed)
    dr, dph = _corrections(case, seed)
    s["dr"], s["dph"] = (None if v is None else torch.as_tensor(v, device="cuda") for v in (dr, dph))
    if kind == "project":
        g = _gen(seed + 2)
        s["weight"] = _noise(shape, g)
        s["out"] = torch.empty(case["np"], dtype=torch.complex128, device="cuda")
    else:
        s["image"] = torch.zeros(shape, dtype=torch.complex64, device="cuda")
        if case["accumulate"]:  # the image of the apertures before this one
            s["before"] = _noise(shape, _gen(seed + 3)).mul_(10.0)
    return s


def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "wk":
        return ctx.wk_image(s["params"], s["echo"], image=s["image"])
    if kind == "rc":
        if case["fp16"]:
            return ctx.range_compress(s["radar"], s["echo"], sarbp.STORE_C32H, out=s["out"], scale=s["scale"])
        return ctx.range_compress(s["radar"], s["echo"], out=s["out"])
    if kind == "image":
        return ctx.image(s["radar"], s["echo"], s["apc"], s["grid"], s["mode"], image=s["image"])
    lay = s["lay"]
    if kind == "project":
        return ctx.project_weighted(s["radar"], s["rows"], s["apc"], s["grid"], s["mode"], lay.t0_bins, lay.bin_rate,
                                    s["weight"], scale=s["scale"], drange=s["dr"], dphase=s["dph"], out=s["out"])
    image, stream = s["image"], None
    if case["accumulate"]:
        # on one stream with the copy that puts the earlier apertures' image there
        own = s.setdefault("stream", torch.cuda.Stream())
        own.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(own):
            image.copy_(s["before"])
        stream = own.cuda_stream
    return ctx.backproject(s["radar"], s["rows"], s["apc"], s["grid"], s["mode"], lay.t0_bins, lay.bin_rate,
                           scale=s["scale"], image=image, accumulate=case["accumulate"], stream=stream,
                           drange=s["dr"], dphase=s["dph"])


def work(case):
    kind = case["kind"]
    if kind == "wk":
        na = case["na"] + 2 * round(case["na"] / 6)
        nr = case["nr"] + 2 * round(case["nr"] / 3)
        return {"bytes": 8 * (case["na"] * case["nr"] + na * nr),
                "flops": na * nr * (10 * math.log2(na * nr) + 40)}
    n_p, ns, up = case["np"], case["ns"], RADAR.upsample
    n = scenes.rc_layout(RADAR, ns, 0.0).nfft
    rc_flops = n_p * (1 + up) * 5 * n * math.log2(n)
    esize = 4 if case["fp16"] else 8
    if kind == "rc":
        return {"bytes": n_p * ns * (8 + up * esize), "flops": rc_flops}
    a = math.radians(case["angle"])
    swath = case["spacing"] * (case["nx"] * abs(math.cos(a)) + case["ny"] * abs(math.sin(a)))
    bins = min(up * ns, swath * 2.0 / RADAR.c * up * RADAR.fs)
    pixels = case["nx"] * case["ny"]
    flops = 28 * n_p * pixels  # range 10, bin 4, interpolation 4, phase 2, complex sum 8
    if kind == "image":
        return {"bytes": 8 * n_p * ns + 8 * pixels, "flops": flops + rc_flops}
    if kind == "project":
        return {"bytes": n_p * bins * esize + 8 * pixels + 16 * n_p, "flops": flops + 2 * n_p * pixels}
    return {"bytes": n_p * bins * esize + 8 * pixels * (2 if case["accumulate"] else 1), "flops": flops}


# ------------------------------------------------------------ 64-bit values

def _exact_spectrum(echo, lay):
    """Matched-filtered spectrum [np][nfft], normalised so that rows are its plain inverse sums."""
    u = torch.arange(lay.nc, device="cuda", dtype=torch.float64) / RADAR.fs
    h = torch.polar(torch.ones_like(u), math.pi * RADAR.kr * (u - RADAR.tp / 2.0) ** 2)
    k = torch.arange(lay.nfft, device="cuda", dtype=torch.float64)
    lag = torch.polar(torch.ones_like(k), -2.0 * math.pi * torch.remainder(k * lay.shift, lay.nfft) / lay.nfft)
    return torch.fft.fft(echo.to(torch.complex128), n=lay.nfft) * torch.fft.fft(h, n=lay.nfft).conj() * lag / lay.nfft


def _exact_upsample(y, lay):
    n, up = lay.nfft, RADAR.upsample
    z = torch.zeros(y.shape[0], up * n, dtype=torch.complex128, device="cuda")
    z[:, :n // 2] = y[:, :n // 2]
    z[:, up * n - n // 2:] = y[:, n // 2:]
    return torch.fft.ifft(z, norm="forward")[:, :lay.nbins]


def _exact_rc(echo, lay, fp16):
    """(rows complex128 before storage, scale float64)"""
    rows = torch.empty(echo.shape[0], lay.nbins, dtype=torch.complex128, device="cuda")
    scale = torch.ones(echo.shape[0], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 23) // (RADAR.upsample * lay.nfft))
    for p in range(0, echo.shape[0], step):
        y = _exact_spectrum(echo[p:p + step], lay)
        rows[p:p + step] = _exact_upsample(y, lay)
        if fp16:
            scale[p:p + step] = torch.exp2(torch.ceil(torch.log2(y.abs().sum(1)) - 14.0))
    return rows, scale


class _Terms:
    """Pulse p's back-projected term at every pixel, in 64 bits."""

    def __init__(self, case, seed, lay):
        g = _grid(case)
        x = torch.arange(g.nx, device="cuda", dtype=torch.float64)[None, :, None]
        y = torch.arange(g.ny, device="cuda", dtype=torch.float64)[:, None, None]
        v = [torch.as_tensor(a, device="cuda") for a in (g.origin, g.ux, g.uy)]
        self.pix = v[0] + x * v[1] + y * v[2]
        self.apc = torch.as_tensor(_track(case, seed), device="cuda")
        self.dr, self.dph = _corrections(case, seed)
        self.lay = lay

    def __call__(self, p, row):
        r = torch.linalg.norm(self.pix - self.apc[p], dim=2)
        ph = 0.0
        if self.dr is not None:
            r, ph = r + float(self.dr[p]), float(self.dph[p])
        tau = 2.0 * r / RADAR.c
        b = (tau - self.lay.t0_bins) * self.lay.bin_rate
        i = torch.floor(b)
        f = b - i
        i = i.long()
        z = torch.cat([torch.zeros(1, dtype=row.dtype, device="cuda"), row, torch.zeros(2, dtype=row.dtype, device="cuda")])
        n = row.numel()
        s0 = z[(i + 1).clamp(0, n + 1)]
        s1 = z[(i + 2).clamp(0, n + 1)]
        cyc = RADAR.fc * tau
        a = 2.0 * math.pi * (cyc - torch.round(cyc)) + ph
        return (s0 + f * (s1 - s0)) * torch.polar(torch.ones_like(a), a)


def _wk_exact(case, seed):
    p = _wk_params()
    echo = _noise((case["na"], case["nr"]), _gen(seed)).to(torch.complex128)
    na, nr, _ = _context().wk_padded_size(case["na"], case["nr"])
    pa, pr = (na - case["na"]) // 2, (nr - case["nr"]) // 2
    dev = dict(device="cuda", dtype=torch.float64)
    m, n = torch.arange(na, **dev), torch.arange(nr, **dev)
    x = torch.zeros(na, nr, dtype=torch.complex128, device="cuda")
    x[pa:pa + case["na"], pr:pr + case["nr"]] = echo
    cyc = -p.f_nc * (m - na // 2) / p.prf
    x *= torch.polar(torch.ones_like(m), 2.0 * math.pi * (cyc - torch.round(cyc)))[:, None]
    x = torch.fft.fft2(x)
    fr = (torch.where(n < nr // 2, n + nr // 2, n - nr // 2) - nr // 2) * (p.fr / nr)
    fa = p.f_nc + (torch.where(m < na // 2, m + na // 2, m - na // 2) - na // 2) * (p.prf / na)
    root = torch.sqrt(torch.clamp((p.f0 + fr)[None, :] ** 2 - p.c ** 2 / (4.0 * p.vr ** 2) * fa[:, None] ** 2, min=0.0))
    theta = 4.0 * math.pi * p.r0 / p.c * root + math.pi * fr[None, :] ** 2 / p.kr
    x *= torch.polar(torch.ones_like(theta), theta)
    centre = n[None, :] - (root - p.f0 - fr[None, :]) * (nr / p.fr)
    out = torch.zeros_like(x)
    for k in range(p.taps):
        i = torch.floor(centre + (k - 0.5 * p.taps)).clamp(0, nr - 1).long()
        out += torch.gather(x, 1, i) * torch.sinc(centre - i)
    return torch.fft.ifft2(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "wk":
        return _wk_exact(case, seed)
    lay = scenes.rc_layout(RADAR, case["ns"], _record_start(case["ns"]))
    if kind == "rc":
        rows, scale = _exact_rc(_echo(case, seed), lay, case["fp16"])
        if case["fp16"]:
            return torch.view_as_real(rows / scale[:, None]), scale
        return rows
    if case["np"] * case["nx"] * case["ny"] > EXACT_UPDATES:
        return None
    if kind == "image":
        rows = _exact_rc(_echo(case, seed), lay, False)[0]
    else:
        rows, scale, _ = _rows(case, seed)
        if case["fp16"]:
            rows = torch.view_as_complex(rows.float()).to(torch.complex128) * scale.double()[:, None]
    term = _Terms(case, seed, lay)
    shape = (case["ny"], case["nx"])
    if kind == "project":
        w = _noise(shape, _gen(seed + 2)).to(torch.complex128).conj()
        return torch.stack([(w * term(p, rows[p].to(torch.complex128))).sum() for p in range(case["np"])])
    image = torch.zeros(shape, dtype=torch.complex128, device="cuda")
    if case.get("accumulate"):
        image += _noise(shape, _gen(seed + 3)).mul_(10.0)
    for p in range(case["np"]):
        image += term(p, rows[p].to(torch.complex128))
    return image
