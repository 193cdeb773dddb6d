"""The migrations that are timed: what a survey processor has the backend do.

Each case is one call of the public backend as a processing program makes it,
with everything but the traces' and tiles' own data decided by the case:

* ``tile``      ``migrate_tile`` / ``_curved_ray`` / ``_vti`` / ``_curved_vti``
                of one output tile on CUDA tensors;
* ``host``      the same with NumPy arrays, copies included, as the reference
                package's executor calls a backend;
* ``bins``      ``migrate_bins``: offset gathers of one tile, an image each;
* ``executor``  ``TiledExecutor``: a small survey grid, tile by tile, on a
                panel in midpoint order;
* ``scatter``   ``migrate_scatter``: a grid in the trace-centric schedule;
* ``variant``   ``migrate_tile_time_variant`` and the resampling back onto the
                uniform time axis;
* ``panel``     ``to_f16_panel``: FP32 traces into scaled FP16 traces.

Traces are band-limited diffraction responses (25 Hz Ricker) with noise at a
tenth of the signal, from sources and receivers spread over the output patch
and, as in a survey, beyond what shallow times can use.  Images are zeroed by
each pass, as a tile's fresh accumulator is.
"""
import math

import numpy as np
import torch

from pstm_b200 import time_variant
from pstm_b200.base import KernelConfig, OutputTile, TraceBlock, VelocitySlice
from pstm_b200.cuda_kernel import Bin, CudaKernel
from pstm_b200.executor import TiledExecutor

DEVICE = "cuda"
KINDS = {"straight": "straight_ray", "curved": "curved_ray", "vti": "anisotropic_vti", "curved_vti": "curved_vti"}
AMPS = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}

BASE = {"form": "tile", "kind": "straight", "precision": "exact", "traces": "f32", "image": "f32",
        "nx": 64, "ny": 64, "nt": 500, "n": 16384, "ns": 500, "dt_ms": 4.0, "dx": 25.0, "start_ms": 0.0,
        "v3d": False, "aa": True, "weights": False, "fold3d": True, "aperture": 5000.0, "dip": 45.0,
        "interp": "linear", "n_bins": 1, "tile": 32}


def _case(name=None, **kw):
    c = {**BASE, **kw}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a quick look at a few traces while picking parameters: the smallest call
        _case("quick_look_8x8", nx=8, ny=8, nt=251, ns=251, n=300, aperture=1000.0, dip=60.0, aa=False),
        # the plain benchmark tile: 64 x 64 bins at 25 m, 2 s at 4 ms, 16,384 traces, constant aperture of 1 km
        _case("plain_64x64x500", aperture=1000.0, dip=60.0, aa=False),
        # one production tile: 3-D velocity, AA, 3 s at 2 ms, the default 5 km aperture, a panel beyond L2's share
        _case("production_64x64x1500", nt=1500, ns=1500, dt_ms=2.0, dx=12.5, v3d=True),
        # the ragged last tile of a survey: odd sizes, unpadded rows, trace weights, recording delay, one fold per pillar
        _case("ragged_37x53x701", nx=37, ny=53, nt=701, ns=777, n=5003, dt_ms=2.0, dx=12.5, start_ms=36.0,
              weights=True, fold3d=False),
        # curved rays through a V(z) gradient, to the reference's accuracy
        _case("curved_48x48x1000", kind="curved", nx=48, ny=48, nt=1000, ns=1000, n=8192, dt_ms=3.0, dx=20.0),
        # a panel put into the precision form's traces once, before its tiles: odd trace length
        _case("panel_40000x1501", form="panel", n=40000, ns=1501, dt_ms=2.0),
        # offset gathers in one call: BF16 traces, VTI, FP32 arithmetic, uneven bins
        _case("bins_vti_bf16", form="bins", kind="vti", precision="fp32", traces="bf16", nx=40, ny=40, nt=1000,
              ns=1000, n=24000, n_bins=6, dt_ms=2.0, dx=12.5, v3d=True),
        # a survey patch tile by tile: scaled FP16 traces, curved rays with VTI, FP32 arithmetic, 1 km aperture
        _case("executor_curved_vti_f16", form="executor", kind="curved_vti", precision="fp32", traces="f16", nx=80,
              ny=80, nt=800, ns=800, n=20000, dt_ms=2.5, dx=12.5, v3d=True, aperture=1000.0),
        # the trace-centric schedule on a whole grid with a narrow aperture
        _case("scatter_96x96x750", form="scatter", nx=96, ny=96, nt=750, ns=750, n=24000, dx=12.5, dt_ms=2.0,
              aperture=500.0),
        # the windowed-sinc interpolator, FP64 throughout, into an FP64 image
        _case("sinc8_40x40x500", image="f64", nx=40, ny=40, n=6000, aperture=1000.0, dip=60.0, interp="sinc8"),
        # the reference executor's call: NumPy in, NumPy out, copies included
        _case("host_32x32x500", form="host", nx=32, ny=32, n=4096, aperture=1000.0, dip=60.0),
        # windows of decreasing rate with depth, resampled onto the uniform axis
        _case("variant_64x64x1001", form="variant", nt=1001, ns=1001, n=12000, dt_ms=2.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# Time of a pair relative to a straight-ray pair, for the size of a drawn case.
COST = {"straight": 1.0, "curved": 3.0, "vti": 2.0, "curved_vti": 4.0}


def draw(rng):
    form = rng.choice(["tile"] * 7 + ["host", "bins", "executor", "scatter", "variant", "interp", "panel"])
    kind = rng.choice(["straight", "straight", "curved", "vti", "curved_vti"])
    if form in ("host", "scatter", "variant", "interp"):
        kind = "straight"
    if form == "panel":
        return _case(form="panel", n=_log(rng, 100, 60000), ns=rng.randint(200, 2000), traces="f32", dt_ms=2.0)
    small = form in ("host", "interp")
    nx, ny = _log(rng, 6, 48 if small else 90), _log(rng, 6, 48 if small else 90)
    nt = _log(rng, 120, 500 if small else 1500)
    n = _log(rng, 200, 6000 if small else 24000)
    limit = (6e9 if form == "interp" else 5e10) / COST[kind]
    n = max(64, min(n, int(limit / (nx * ny * nt))))
    traces = rng.choice(["f32", "f32", "bf16", "f16"]) if form != "host" else "f32"
    precision = rng.choice(["exact", "exact", "fp32"]) if form != "interp" else "exact"
    return _case(form="tile" if form == "interp" else form, kind=kind, precision=precision, traces=traces,
                 image="f64" if form == "interp" else "f32", nx=nx, ny=ny, nt=nt, n=n,
                 ns=nt + rng.randint(0, nt // 4), dt_ms=rng.choice([2.0, 2.0, 3.0, 4.0]),
                 dx=rng.choice([12.5, 20.0, 25.0]), start_ms=rng.choice([0.0, 0.0, 24.0]),
                 v3d=form not in ("host", "variant", "interp") and rng.random() < 0.5, aa=rng.random() < 0.7,
                 weights=rng.random() < 0.3, fold3d=rng.random() < 0.7,
                 aperture=rng.choice([500.0, 1000.0, 2000.0, 5000.0]), dip=rng.choice([45.0, 60.0]),
                 interp=rng.choice(["sinc8", "sinc8", "cubic", "lanczos3", "sinc16"]) if form == "interp" else "linear",
                 n_bins=rng.randint(2, 9) if form == "bins" else 1, tile=rng.choice([24, 32]))


# ------------------------------------------------------------------ inputs
def _panel(c, g, sx, sy, rx, ry, ext):
    """(n, ns) FP32: Ricker responses of six diffractors + a tenth of noise."""
    n, ns = c["n"], c["ns"]
    t = c["start_ms"] / 1000 + torch.arange(ns, device=DEVICE, dtype=torch.float32) * (c["dt_ms"] / 1000)
    tmax = c["nt"] * c["dt_ms"] / 1000
    u = torch.rand((6, 3), generator=g, device=DEVICE, dtype=torch.float64).tolist()
    amps = torch.empty((n, ns), device=DEVICE)
    for b in range(0, n, 16384):
        s = slice(b, min(n, b + 16384))
        acc = torch.zeros((s.stop - b, ns), device=DEVICE)
        for ux, uy, ut in u:
            x, y, t0 = ux * ext[0], uy * ext[1], (0.15 + 0.6 * ut) * tmax
            v = 1500.0 + 2500.0 * t0 / 3.0
            T = sum(torch.sqrt((t0 / 2) ** 2 + ((px[s] - x) ** 2 + (py[s] - y) ** 2) / v ** 2)
                    for px, py in ((sx, sy), (rx, ry)))
            a = (math.pi * 25.0 * (t[None, :] - T.float()[:, None])) ** 2
            acc += (1 - 2 * a) * torch.exp(-a)
        amps[s] = acc
    amps += 0.1 * amps.square().mean().sqrt() * torch.randn((n, ns), generator=g, device=DEVICE)
    return amps


def _inputs(c, seed):
    """Geometry, traces, axes and velocity on the GPU, from the seed alone."""
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))
    n, nx, ny, nt = c["n"], c["nx"], c["ny"], c["nt"]
    rand = lambda *s: torch.rand(s, generator=g, device=DEVICE, dtype=torch.float64)   # noqa: E731
    # midpoints over the patch and a margin of up to half a kilometre, offsets up to 2 km
    ext = (nx * c["dx"], ny * c["dx"])
    margin = min(500.0, c["aperture"] / 2)
    mx, my = (rand(n) * (e + 2 * margin) - margin for e in ext)
    if c["form"] == "bins":   # common-offset gathers, one after another
        which = torch.as_tensor(np.repeat(np.arange(c["n_bins"]), _bin_counts(c)), device=DEVICE)
        off = (which + rand(n)) * 200.0
    else:
        off = rand(n) * 2000.0
    az = rand(n) * 2 * math.pi
    hx, hy = 0.5 * off * torch.cos(az), 0.5 * off * torch.sin(az)
    p = {"sx": mx - hx, "sy": my - hy, "rx": mx + hx, "ry": my + hy, "off": off}
    p["mx"], p["my"] = (p["sx"] + p["rx"]) / 2, (p["sy"] + p["ry"]) / 2
    amps = _panel(c, g, p["sx"], p["sy"], p["rx"], p["ry"], ext)
    p["w"] = 0.5 + rand(n) if c["weights"] else None
    if c["traces"] == "f16" and c["form"] != "panel":   # a power-of-two scale per trace, carried by its weight
        e = torch.floor(torch.log2(amps.abs().amax(1, keepdim=True).double()))
        amps = (amps.double() * torch.exp2(13 - e)).half()
        p["w"] = torch.exp2(e - 13)[:, 0] * (1.0 if p["w"] is None else p["w"])
    elif c["traces"] == "bf16":
        amps = amps.bfloat16()
    p["amps"] = amps
    p["x"] = torch.arange(nx, device=DEVICE, dtype=torch.float64) * c["dx"]
    p["y"] = torch.arange(ny, device=DEVICE, dtype=torch.float64) * c["dx"]
    p["t"] = torch.arange(nt, device=DEVICE, dtype=torch.float64) * c["dt_ms"]
    v = 1500.0 + 2500.0 * p["t"] / 3000.0
    if c["v3d"]:   # a few per cent of smooth lateral variation
        a = (rand(4) * 2 * math.pi).tolist()
        f = torch.sin(p["x"] / 400.0 + a[0])[:, None] * torch.cos(p["y"] / 300.0 + a[1]) + \
            torch.sin((p["x"][:, None] + p["y"]) / 500.0 + a[2])
        v = v * (1 + 0.04 * f)[:, :, None]
    p["v"] = v.contiguous()
    p["eta"] = torch.clamp(0.15 * p["t"] / 3000.0, 0.0, 0.15) if "vti" in c["kind"] else None
    return p


def _bin_counts(c):
    """Traces of each gather: uneven, about n in all."""
    share = np.array([1.0 + (3 * b * b + 5 * b) % 7 for b in range(c["n_bins"])])
    counts = np.floor(c["n"] * share / share.sum()).astype(np.int64)
    counts[0] += c["n"] - counts.sum()
    return counts


def _config(c, p):
    return KernelConfig(max_aperture_m=c["aperture"], max_dip_degrees=c["dip"], aa_enabled=c["aa"],
                        interpolation_method=c["interp"], kernel_type=KINDS[c["kind"]], grid_dx=c["dx"],
                        grid_dy=c["dx"], curved_ray_enabled=c["kind"].startswith("curved"),
                        vti_enabled=p["eta"] is not None,
                        vti_eta_array=p["eta"].cpu().numpy() if c["form"] == "host" and p["eta"] is not None
                        else p["eta"])


def _windows(c):
    return time_variant.compute_time_windows(0.0, (c["nt"] - 1) * c["dt_ms"], c["dt_ms"],
                                             time_variant.FrequencyTimeTable.default())


def prepare(case, seed):
    c = case
    p = _inputs(c, seed)
    if c["form"] == "host":
        p = {k: v.cpu().numpy() if torch.is_tensor(v) else v for k, v in p.items()}
        zeros = lambda s, d: np.zeros(s, {torch.float32: np.float32, torch.int32: np.int32}[d])   # noqa: E731
    else:
        zeros = lambda s, d: torch.zeros(s, dtype=d, device=DEVICE)   # noqa: E731
    cfg = _config(c, p)
    k = CudaKernel(device=0, precision=c["precision"])
    k.initialize(cfg)
    tb = TraceBlock(amplitudes=p["amps"], source_x=p["sx"], source_y=p["sy"], receiver_x=p["rx"], receiver_y=p["ry"],
                    offset=p["off"], midpoint_x=p["mx"], midpoint_y=p["my"], weights=p["w"],
                    sample_rate_ms=c["dt_ms"], start_time_ms=c["start_ms"])
    s = {"case": c, "kernel": k, "cfg": cfg, "traces": tb}
    if c["form"] == "panel":
        return s
    shape = (c["nx"], c["ny"], c["nt"])
    image = torch.float64 if c["image"] == "f64" else torch.float32
    if c["form"] == "executor":
        v = p["v"]
        vel = (lambda a, b, d, e: VelocitySlice(vrms=v[a:b, d:e].contiguous(), is_1d=False)) if c["v3d"] else \
              (lambda a, b, d, e: VelocitySlice(vrms=v, is_1d=True))
        s["executor"] = TiledExecutor(k, tb, p["x"].cpu().numpy(), p["y"].cpu().numpy(), p["t"].cpu().numpy(), vel,
                                      cfg, kernel_type=KINDS[c["kind"]], tile=c["tile"], spatial=True)
    fold = shape if c["fold3d"] else shape[:2]
    s["image"], s["fold"] = zeros(shape, image), zeros(fold, torch.int32)
    s["axes"] = {"x_axis": p["x"], "y_axis": p["y"], "t_axis_ms": p["t"]}
    s["velocity"] = VelocitySlice(vrms=p["v"], is_1d=not c["v3d"])
    if c["form"] == "bins":
        counts = _bin_counts(c)
        s["bins"] = [Bin(int(a), int(m), zeros(shape, image), zeros(fold, torch.int32))
                     for a, m in zip(np.cumsum(counts) - counts, counts)]
    if c["form"] == "variant":
        s["windows"] = _windows(c)
    return s


def run(state):
    s = state
    c, k, cfg, tb = s["case"], s["kernel"], s["cfg"], s["traces"]
    form = c["form"]
    if form == "panel":
        got = k.to_f16_panel(tb)
        return {"traces": got.amplitudes, "weights": got.weights}
    if form == "bins":
        for b in s["bins"]:
            b.image.zero_()
            b.fold.zero_()
        geometry = OutputTile(image=None, fold=None, **s["axes"])
        k.migrate_bins(tb, s["bins"], geometry, s["velocity"], cfg, kernel_type=KINDS[c["kind"]])
        return [{"image": b.image, "fold": b.fold} for b in s["bins"]]
    image, fold = s["image"], s["fold"]
    image[...] = 0
    fold[...] = 0
    if form == "executor":
        s["executor"].run(image, fold)
        return {"image": image, "fold": fold}
    out = OutputTile(image=image, fold=fold, **s["axes"])
    if form == "scatter":
        k.migrate_scatter(tb, out, s["velocity"], cfg, kernel_type=KINDS[c["kind"]])
    elif form == "variant":
        k.migrate_tile_time_variant(tb, out, s["velocity"], cfg, s["windows"])
        image = time_variant.resample_to_uniform(out.image, s["windows"], c["dt_ms"], c["nt"], ctx=k.context)
    else:
        call = {"straight": k.migrate_tile, "curved": k.migrate_tile_curved_ray, "vti": k.migrate_tile_vti,
                "curved_vti": k.migrate_tile_curved_vti}[c["kind"]]
        call(tb, out, s["velocity"], cfg)
    return {"image": image, "fold": fold}


# ------------------------------------------------------------------ floor
TAPS = {"linear": 2, "cubic": 4, "sinc8": 8, "sinc16": 16, "lanczos3": 6}


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    those of one pair inside its time-varying aperture (traveltime, sample
    index, interpolation, weights, accumulation) times the expected number of
    such pairs; a square root, reciprocal or logarithm counts as one."""
    c = case
    elem = 4 if c["traces"] == "f32" else 2
    n, ns = c["n"], c["ns"]
    if c["form"] == "panel":
        return {"bytes": n * ns * 6.0 + n * 8.0, "flops": n * ns * 2.0}
    nx, ny, nt = c["nx"], c["ny"], c["nt"]
    pix = nx * ny * nt
    per_point = 12.0 if c["image"] == "f64" else 8.0
    by = n * ns * elem + n * 48.0 + pix * per_point * c["n_bins"] + (pix * 8.0 if c["v3d"] else 0.0)
    r = np.random.default_rng(1)
    m = 200000
    margin = min(500.0, c["aperture"] / 2)
    d = np.hypot(*(r.random(m) * e * c["dx"] - (r.random(m) * (e * c["dx"] + 2 * margin) - margin) for e in (nx, ny)))
    t0 = r.random(m) * nt * c["dt_ms"] / 1000
    if c["form"] == "variant":
        times = time_variant.window_times(_windows(c)) / 1000
        t0, pix = r.choice(times, m), nx * ny * len(times)
    ap = np.clip((1500 + 2500 * t0 / 3) * t0 / 2 * math.tan(math.radians(c["dip"])), 500.0, c["aperture"])
    inside = float(np.mean((d <= ap) & (t0 * 1000 < ns * c["dt_ms"] + c["start_ms"])))
    per_pair = {"straight": 8, "curved": 12, "vti": 20, "curved_vti": 32}[c["kind"]] + 3 + 5 + \
        (7 if c["aa"] else 0) + (1 if c["weights"] or c["traces"] == "f16" else 0) + \
        (3 if c["interp"] == "linear" else 6 * TAPS[c["interp"]])
    return {"bytes": by, "flops": float(pix) * n * inside * per_pair}


# ------------------------------------------------------------------ in 64 bits
def _time(c, t0, h2, v, eta, v0=1500.0, k=0.5):
    """One leg (source or receiver side) of the traveltime in seconds."""
    th = t0 / 2
    if c["kind"] == "straight":
        return torch.sqrt(th * th + h2 / (v * v))
    if "vti" in c["kind"]:
        den = v * v * (th * th * v * v + (1 + 2 * eta) * h2)
        corr = torch.where(den.abs() > 1e-20, 2 * eta * h2 * h2 / den, torch.zeros_like(h2))
        hyp = th * th + h2 / (v * v)
        if c["kind"] == "vti":
            return torch.where(th > 0, torch.sqrt(torch.clamp(hyp - corr, min=0.0)), 0 * h2)
    vz = v0 * torch.exp(k * th)
    tc = torch.log((vz + torch.sqrt(vz * vz + k * k * h2)) / (v0 + torch.sqrt(v0 * v0 + k * k * h2))) / k
    if c["kind"] == "curved":
        return tc
    return torch.where(th > 0, tc * torch.sqrt(torch.clamp(1 - corr / hyp, min=0.0)), tc)


def _sample(c, amps, row, s):
    """Interpolated amplitudes of rows `row` at fractional samples `s` (0 <= s < ns - 1)."""
    ns, m = c["ns"], c["interp"]
    flat = amps.reshape(-1)
    at = lambda i: flat[row + i]   # noqa: E731
    i0 = s.long()
    f = s - i0
    lin = at(i0) * (1 - f) + at(i0 + 1) * f
    if m == "linear":
        return lin
    if m == "cubic":
        i = i0.clamp(1, ns - 3)
        p0, p1, p2, p3 = (at(i + j) for j in (-1, 0, 1, 2))
        cub = ((((-p0 + 3 * p1 - 3 * p2 + p3) * f + (2 * p0 - 5 * p1 + 4 * p2 - p3)) * f + (p2 - p0)) * f) / 2 + p1
        return torch.where((s >= 1) & (s < ns - 2), cub, lin)
    hw = TAPS[m] // 2
    ic = i0 if m.startswith("lanczos") else (s + 0.5).long()
    acc, norm = torch.zeros_like(s), torch.zeros_like(s)
    for j in range(-hw + 1, hw + 1):
        i = ic + j
        x = s - i
        w = torch.sinc(x) * (torch.sinc(x / hw) if m.startswith("lanczos") else 0.5 * (1 + torch.cos(math.pi * x / hw)))
        w = torch.where((x.abs() < hw) & (i >= 0) & (i < ns), w, torch.zeros_like(w))
        acc += at(i.clamp(0, ns - 1)) * w
        norm += w
    wide = torch.where(norm != 0, acc / norm, torch.zeros_like(acc))
    return torch.where((s < hw) | (s >= ns - hw), lin, wide)


def _exact_image(c, p, t_ms, v, eta, rows):
    """Image and fold of traces `rows` at the times t_ms, all in FP64."""
    nx, ny, nt, ns = len(p["x"]), len(p["y"]), len(t_ms), c["ns"]
    dt, start = c["dt_ms"] / 1000, c["start_ms"] / 1000
    sx, sy, rx, ry, mx, my = (p[k][rows] for k in ("sx", "sy", "rx", "ry", "mx", "my"))
    w = p["w"][rows] if p["w"] is not None else torch.ones_like(sx)
    amps, first = p["amps"].double(), rows.start * ns
    t = t_ms / 1000
    tan = math.tan(math.radians(c["dip"]))
    image = torch.zeros((nx, ny, nt), dtype=torch.float64, device=DEVICE)
    fold = torch.zeros((nx, ny), dtype=torch.int32, device=DEVICE)
    step = 256
    for ix in range(nx):
        for iy in range(ny):
            ddx, ddy = p["x"][ix] - mx, p["y"][iy] - my
            d, order = torch.sort(torch.sqrt(ddx * ddx + ddy * ddy))
            fold[ix, iy] = (d <= c["aperture"]).sum()
            vp = v if v.dim() == 1 else v[ix, iy]
            ap = torch.clamp(vp * t * 0.5 * tan, 500.0, c["aperture"])
            reach = torch.searchsorted(d, torch.stack([ap[b:b + step].max() for b in range(0, nt, step)]), right=True)
            m = torch.maximum(ddx.abs(), ddy.abs())[order]
            ds2 = ((p["x"][ix] - sx) ** 2 + (p["y"][iy] - sy) ** 2)[order]
            dr2 = ((p["x"][ix] - rx) ** 2 + (p["y"][iy] - ry) ** 2)[order]
            base, wo = first + order * ns, w[order]
            for q, r in enumerate(reach.tolist()):
                b = q * step
                if r == 0:
                    continue
                t0, vv, aa = t[b:b + step, None], vp[b:b + step, None], ap[b:b + step, None]
                et = eta[b:b + step, None] if eta is not None else None
                T = _time(c, t0, ds2[None, :r], vv, et) + _time(c, t0, dr2[None, :r], vv, et)
                s = (T - start) / dt
                ok = (s >= 0) & (s < ns - 1) & (d[None, :r] <= aa)
                g = _sample(c, amps, base[None, :r], torch.where(ok, s, torch.zeros_like(s))) * wo[:r]
                x = (d[None, :r] - 0.9 * aa) / (0.1 * aa)
                g *= torch.where(x > 0, 0.5 * (1 + torch.cos(math.pi * x)), torch.ones_like(x))
                vw = 1500.0 * torch.exp(0.5 * t0 / 2) if c["kind"].startswith("curved") else vv
                late = T > 0.001
                if c["aa"]:
                    sn = torch.clamp(m[None, :r] / (vw * T), max=1.0)
                    fmax = torch.clamp(vw / (4 * c["dx"] * sn), max=500.0)
                    g *= torch.where((T >= 0.001) & (sn >= 0.01), torch.clamp(1 - 30.0 / fmax, min=0.0),
                                     torch.ones_like(T))
                g *= torch.where(late, t0 / (vw * T * T), torch.ones_like(T))
                image[ix, iy, b:b + step] = torch.where(ok, g, torch.zeros_like(g)).sum(1)
    if c["fold3d"]:
        fold = fold[:, :, None].expand(nx, ny, nt).contiguous()
    return {"image": image, "fold": fold}


def exact(case, seed):
    c = case
    p = _inputs(c, seed)
    if c["form"] == "panel":
        a = p["amps"].double()
        e = torch.floor(torch.log2(a.abs().amax(1, keepdim=True)))
        w = torch.exp2(e - 13)[:, 0] * (1.0 if p["w"] is None else p["w"])
        return {"traces": a * torch.exp2(13 - e), "weights": w}
    if c["nx"] * c["ny"] * (c["nt"] // 256 + 1) * c["n_bins"] > 50000:   # over about 20 seconds
        return None
    everything = slice(0, c["n"])
    if c["form"] == "bins":
        counts = _bin_counts(c)
        return [_exact_image(c, p, p["t"], p["v"], p["eta"], slice(int(e - m), int(e)))
                for e, m in zip(np.cumsum(counts), counts)]
    if c["form"] != "variant":
        return _exact_image(c, p, p["t"], p["v"], p["eta"], everything)
    tv = time_variant.window_times(_windows(c))
    v = torch.as_tensor(np.interp(tv, p["t"].cpu().numpy(), p["v"].cpu().numpy()), device=DEVICE)
    tt = torch.as_tensor(tv, device=DEVICE)
    got = _exact_image({**c, "fold3d": False}, p, tt, v, None, everything)
    # linear onto the uniform axis, the edge values beyond it
    u = torch.clamp(p["t"], float(tv[0]), float(tv[-1]))
    i = torch.clamp(torch.searchsorted(tt, u, right=True) - 1, 0, len(tv) - 2)
    f = (u - tt[i]) / (tt[i + 1] - tt[i])
    got["image"] = got["image"][:, :, i] * (1 - f) + got["image"][:, :, i + 1] * f
    if c["fold3d"]:
        got["fold"] = got["fold"][:, :, None].expand(c["nx"], c["ny"], c["nt"]).contiguous()
    return got
