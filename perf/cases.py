"""Timed cases of the library's public entry points.

Each case is a dict of plain values whose "kind" names the entry point:

  image       one device-resident image (Context.run_jobs with one job)
  batch       images of uneven size in one call (Context.run_jobs)
  plan        such a batch captured once and replayed (Context.plan)
  host        the reference's operator on host arrays (Context.backprojection_cuda)
  accumulate  one image formed from pulse chunks (Accumulator)
  profiles    range compression alone (Context.range_compress_device)
  output      dB and u8 images of a complex image
  resize      resampling of a recorded phase history (sarbp_resize_device)

Phase histories are those of point scatterers in complex Gaussian noise on a
circular aperture, made on the GPU from the seed.  A phase history of S
samples in steps of df has the range resolution c / (2 S df); "pixel" is the
pixel spacing in units of it.  The image plane is the reference's, turned
with the aperture by "az" degrees.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "halide-sar-app_b200"))
import sarbp_b200 as sb  # noqa: E402
from sarbp_b200._lib import check, lib  # noqa: E402

C = 299792458.0
GPU = "cuda"
_context = []


def context():
    """The process's library context (a program makes one per device)."""
    if not _context:
        _context.append(sb.Context(0))
    return _context[0]


# ---- the cases ----

def _image(name, kind="image", **kw):
    base = dict(name=name, kind=kind, nu=512, nv=512, pulses=469, samples=424, upsample=2, f0=9.29e9, df=1.5e6,
                R0=10e3, dep=30.0, span=4.0, az=0.0, pixel=0.41, taylor=17, precise=False, locs=False, u8=False)
    base.update(kw)
    return base


def listed():
    return [
        # the smallest images a serving job asks for: launches and latency
        _image("image_256", nu=256, nv=256, pulses=300, samples=256, df=1.0e6, R0=8e3, dep=35.0, span=3.0,
               pixel=0.5, taylor=20),
        # the bench's plain_small, a one-pass AFRL-sized image with its u8 image
        _image("image_512", u8=True),
        # sizes that divide nothing, pixel positions as the reference passes
        # them (an array), coarse pixels, a plane turned off the axes
        _image("image_ragged", nu=1000, nv=731, pulses=777, samples=600, df=1.1e6, R0=6e3, dep=40.0, span=3.5,
               az=35.0, pixel=0.6, taylor=25, locs=True),
        # the bench's plain_large, the headline workload
        _image("image_2048", nu=2048, nv=2048, pulses=1999, samples=1024, f0=16.7e9, df=0.59e6, R0=8e3, dep=45.0,
               span=3.0, pixel=0.1968, taylor=30),
        # f64 positions at 20 km (the bench's precision study), half its pulses
        _image("image_precise_4096", nu=4096, nv=4096, pulses=2000, samples=2048, f0=16.7e9, df=0.59e6, R0=20e3,
               dep=45.0, span=3.0, pixel=0.197, taylor=30, precise=True),
        # a served mix of uneven jobs, f64 positions and u8 images
        dict(name="batch_12", kind="batch", jobs=12, mix=7, nmin=256, nmax=1024, precise=True, u8=True),
        # a fixed set of small jobs replayed as its data changes
        dict(name="plan_small", kind="plan", jobs=6, mix=3, nmin=256, nmax=512, precise=False, u8=False),
        # the drop-in call: numpy arrays in, numpy image out
        _image("host_768", kind="host", nu=768, nv=768, pulses=800, samples=512, df=1.2e6, R0=9e3, dep=35.0,
               span=3.0, az=12.0, pixel=0.4),
        # a phase history that arrives in chunks
        _image("accumulate_1024", kind="accumulate", nu=1024, nv=1024, pulses=1200, samples=700, f0=12e9, df=0.8e6,
               R0=12e3, dep=30.0, span=3.0, az=-20.0, pixel=0.45, taylor=22, precise=True, chunk=200),
        # range profiles of a long-swath collection (8192 samples: N_fft 32768)
        _image("profiles_8192", kind="profiles", pulses=1024, samples=8192, f0=16.7e9, df=0.07375e6, R0=8e3,
               dep=45.0, span=3.0, taylor=30),
        # display and measurement images of a formed image
        dict(name="output_2048", kind="output", nu=2048, nv=2048, lo=-45.0, hi=0.0),
        # a recorded phase history brought to fewer pulses and samples
        dict(name="resize_half", kind="resize", rows=1999, cols=1800, out_rows=999, out_cols=900, double=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["image"] * 5 + ["batch", "plan", "host", "accumulate", "profiles", "output", "resize"])
    if kind in ("batch", "plan"):
        return dict(kind=kind, jobs=rng.randint(2, 12), mix=rng.randrange(1 << 20), nmin=rng.choice([64, 128, 256]),
                    nmax=rng.choice([512, 1024]), precise=rng.random() < 0.5, u8=rng.random() < 0.5)
    if kind == "output":
        return dict(kind=kind, nu=_log(rng, 64, 4096), nv=_log(rng, 64, 4096), lo=rng.choice([-60.0, -45.0, -30.0]),
                    hi=0.0)
    if kind == "resize":
        r, c = _log(rng, 64, 3000), _log(rng, 64, 3000)
        f, g = rng.choice([0.25, 0.5, 0.8, 1.0, 1.5, 2.0]), rng.choice([0.25, 0.5, 0.8, 1.0, 1.5, 2.0])
        return dict(kind=kind, rows=r, cols=c, out_rows=max(1, int(r * f)), out_cols=max(1, int(c * g)),
                    double=rng.random() < 0.7)
    n = _log(rng, 64, 2048)
    c = _image(None, kind=kind, nu=n, nv=max(32, min(2048, int(n * rng.uniform(0.6, 1.4)))),
               pulses=_log(rng, 48, 2000), samples=_log(rng, 100, 2048), upsample=rng.choice([1, 2, 2, 2, 6]),
               f0=rng.uniform(9e9, 17e9), df=rng.uniform(0.5e6, 1.5e6), R0=rng.uniform(5e3, 20e3),
               dep=rng.uniform(20.0, 50.0), span=rng.uniform(2.0, 4.0), az=rng.choice([0.0, rng.uniform(-60.0, 60.0)]),
               pixel=rng.uniform(0.2, 0.7), taylor=rng.randint(17, 30), precise=rng.random() < 0.4,
               locs=rng.random() < 0.4, u8=rng.random() < 0.4)
    del c["name"]
    if kind == "host":
        c["nu"], c["nv"] = min(c["nu"], 1024), min(c["nv"], 1024)
    if kind == "accumulate":
        c["chunk"] = rng.randint(16, max(17, c["pulses"] // 2))
    if kind == "profiles":
        c["pulses"], c["samples"] = _log(rng, 48, 2000), _log(rng, 100, 8192)
        c["df"] *= min(1.0, 1024 / c["samples"])
        c["upsample"] = rng.choice([1, 2])
    return c


def _mix(case):
    """The jobs of a batch or plan: sizes as the bench's uneven batch draws them."""
    rng = np.random.default_rng(case["mix"])
    sizes = [n for n in (64, 128, 256, 512, 1024) if case["nmin"] <= n <= case["nmax"]]
    jobs = []
    for _ in range(case["jobs"]):
        n = int(rng.choice(sizes))
        jobs.append(_image(None, nu=n, nv=n, pulses=int(rng.integers(128, 1001)),
                           samples=int(rng.choice([256, 512, 1024])), f0=float(rng.uniform(9e9, 17e9)),
                           df=float(rng.uniform(0.5e6, 1.5e6)), R0=float(rng.uniform(5e3, 15e3)),
                           dep=float(rng.uniform(20.0, 50.0)), span=float(rng.uniform(2.0, 4.0)), pixel=0.5,
                           taylor=int(rng.integers(17, 31)), precise=case["precise"], u8=case["u8"]))
    return jobs


# ---- inputs ----

def _rng(seed):
    g = torch.Generator(device=GPU)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _aperture(c, seed, scatterers=16):
    """Phase history and geometry of a case, on the GPU."""
    P, S = c["pulses"], c["samples"]
    delta_r = C / (2.0 * S * c["df"])
    az = torch.deg2rad(torch.linspace(-c["span"] / 2, c["span"] / 2, P, dtype=torch.float64) + c["az"])
    dep = math.radians(c["dep"])
    pos = torch.stack([c["R0"] * math.cos(dep) * torch.cos(az), c["R0"] * math.cos(dep) * torch.sin(az),
                       torch.full_like(az, c["R0"] * math.sin(dep))], 1).to(GPU)
    k_r = (4.0 * math.pi / C) * (c["f0"] + c["df"] * torch.arange(S, dtype=torch.float64, device=GPU))
    g = _rng(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device=GPU, dtype=torch.float64)  # noqa: E731
    d = c["pixel"] * delta_r
    xy = (rand(scatterers, 2) - 0.5) * torch.tensor([0.8 * c["nu"] * d, 0.8 * c["nv"] * d], device=GPU)
    amp = torch.complex(*(torch.randn(2, scatterers, generator=g, device=GPU, dtype=torch.float64) / math.sqrt(2.0)))
    phs = torch.zeros(P, S, dtype=torch.complex128, device=GPU)
    norm = pos.norm(dim=1)
    ca, sa = math.cos(math.radians(c["az"])), math.sin(math.radians(c["az"]))
    for i in range(scatterers):
        x = torch.stack([ca * xy[i, 0] - sa * xy[i, 1], sa * xy[i, 0] + ca * xy[i, 1], torch.zeros_like(xy[i, 0])])
        ph = (norm - (pos - x).norm(dim=1))[:, None] * k_r[None, :]
        phs += amp[i] * torch.polar(torch.ones_like(ph), ph)
    noise = torch.randn(2, P, S, generator=g, device=GPU, dtype=torch.float32)
    phs += 0.1 * math.sqrt(scatterers / 2.0) * torch.complex(noise[0], noise[1])
    # the image plane's axes (the reference's, from the mid-aperture position)
    ip = sb.img_plane_create(S, P, delta_r, pos[P // 2].float().cpu().numpy(), upsample=False, with_pixel_locs=False)
    axis = lambda n: (torch.arange(n, dtype=torch.float64, device=GPU) - n // 2) * d  # noqa: E731
    return dict(phs=phs.to(torch.complex64), pos=pos, k_r=k_r, delta_r=delta_r, u=axis(c["nu"]), v=axis(c["nv"]),
                u_hat=ip["u_hat"], v_hat=ip["v_hat"], n_fft=sb.n_fft_for(S, c["upsample"]))


def _locs(a):
    """Pixel positions [3, nu * nv], pixel i at u[i % nu], v[i // nu]."""
    uh, vh = [torch.as_tensor(np.asarray(x), device=GPU) for x in (a["u_hat"], a["v_hat"])]
    return ((uh[:, None, None] * a["u"][None, None, :]) + (vh[:, None, None] * a["v"][None, :, None])).reshape(3, -1)


def _job(c, seed):
    """A device-resident job: its arrays, and the Job that points to them."""
    a = _aperture(c, seed)
    a["out"] = torch.zeros(c["nv"], c["nu"], dtype=torch.complex128, device=GPU)
    a["u8"] = torch.zeros(c["nv"], c["nu"], dtype=torch.uint8, device=GPU) if c["u8"] else None
    a["r"] = _locs(a).contiguous() if c["locs"] else None
    a["k32"], a["pos32"] = a["k_r"].float(), a["pos"].float()
    at = lambda t: t.data_ptr() if t is not None else 0  # noqa: E731
    a["job"] = sb.make_job(c["samples"], c["pulses"], a["n_fft"], c["taylor"], c["nu"], c["nv"], a["delta_r"],
                           at(a["phs"]), at(a["k32"]), at(a["pos32"]), at(a["out"]), r=at(a["r"]), u=at(a["u"]),
                           v=at(a["v"]), u_hat=a["u_hat"], v_hat=a["v_hat"],
                           k_r64=at(a["k_r"]) if c["precise"] else 0, pos64=at(a["pos"]) if c["precise"] else 0,
                           out_u8=at(a["u8"]), dB_min=-40.0, dB_max=0.0,
                           precision=sb.PREC_PRECISE if c["precise"] else sb.PREC_COMPAT)
    return a


def _images(arrays):
    return [[a["out"], a["u8"]] if a["u8"] is not None else [a["out"]] for a in arrays]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "output":
        # speckle with a few bright points, as a formed image has
        g = _rng(seed)
        z = torch.randn(2, case["nv"], case["nu"], generator=g, device=GPU, dtype=torch.float64)
        img = torch.complex(z[0], z[1]).reshape(-1)
        at = torch.randint(0, img.numel(), (64,), generator=g, device=GPU)
        img[at] *= 10.0 ** (3.0 * torch.rand(64, generator=g, device=GPU, dtype=torch.float64))
        return dict(case=case, img=img.reshape(case["nv"], case["nu"]).contiguous(),
                    dB=torch.empty(case["nv"], case["nu"], dtype=torch.float64, device=GPU),
                    u8=torch.empty(case["nv"], case["nu"], dtype=torch.uint8, device=GPU))
    if kind == "resize":
        t = torch.float64 if case["double"] else torch.float32
        src = torch.randn(case["rows"], case["cols"], 2, generator=_rng(seed), device=GPU, dtype=t)
        return dict(case=case, src=src, out=torch.empty(case["out_rows"], case["out_cols"], 2, device=GPU, dtype=t))
    if kind in ("batch", "plan"):
        arrays = [_job(c, seed * 100 + i) for i, c in enumerate(_mix(case))]
        s = dict(case=case, arrays=arrays, jobs=[a["job"] for a in arrays])
        if kind == "plan":
            torch.cuda.synchronize()
            s["plan"] = context().plan(s["jobs"])
        return s
    if kind == "host":
        a = _aperture(case, seed)
        pos, k_r = (a["pos"], a["k_r"]) if case["precise"] else (a["pos"].float(), a["k_r"].float())
        host = dict(phs=a["phs"], k_r=k_r, pos=pos, u=a["u"], v=a["v"], r=_locs(a))
        return dict(case=case, n_fft=a["n_fft"], delta_r=a["delta_r"],
                    **{k: v.cpu().numpy() for k, v in host.items()})
    if kind == "profiles":
        a = _job(dict(case, nu=1, nv=1), seed)
        a["q"] = torch.empty(case["pulses"], a["n_fft"], dtype=torch.complex64, device=GPU)
        return dict(case=case, arrays=[a])
    a = _job(case, seed)
    s = dict(case=case, arrays=[a], jobs=[a["job"]])
    if kind == "accumulate":
        torch.cuda.synchronize()
        s["acc"] = sb.Accumulator(context(), a["job"], case["chunk"], a["job"].precision)
    return s


def run(s):
    case, ctx = s["case"], context()
    kind = case["kind"]
    if kind in ("image", "batch"):
        ctx.run_jobs(s["jobs"])
        return _images(s["arrays"])
    if kind == "plan":
        s["plan"].launch(lib().sarbp_ctx_stream(ctx.handle))
        return _images(s["arrays"])
    if kind == "host":
        return ctx.backprojection_cuda(s["phs"], s["k_r"], case["taylor"], s["n_fft"], s["delta_r"], s["u"], s["v"],
                                       s["pos"], s["r"])
    if kind == "accumulate":
        acc, a, P, n = s["acc"], s["arrays"][0], case["pulses"], case["chunk"]
        acc.reset()
        row = case["samples"] * 8
        for p in range(0, P, n):
            acc.add_device(p, min(n, P - p), a["phs"].data_ptr() + p * row)
        acc.finalize()
        return _images(s["arrays"])
    if kind == "profiles":
        a = s["arrays"][0]
        ctx.range_compress_device(a["job"], a["q"].data_ptr(), a["job"].precision)
        return a["q"]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    if kind == "output":
        nu, nv = case["nu"], case["nv"]
        check(lib().sarbp_img_output_to_dB_device(ctx.handle, p(s["img"]), nu, nv, p(s["dB"])))
        ctx.img_output_u8_from_img_device(s["img"].data_ptr(), nu, nv, case["lo"], case["hi"], s["u8"].data_ptr())
        return [s["dB"], s["u8"]]
    check(lib().sarbp_resize_device(ctx.handle, 8 if case["double"] else 4, 2, p(s["src"]), case["rows"],
                                    case["cols"], case["out_rows"], case["out_cols"], p(s["out"])))
    return s["out"]


def work(case):
    kind = case["kind"]
    if kind in ("batch", "plan"):
        parts = [work(c) for c in _mix(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "output":
        n = case["nu"] * case["nv"]
        return {"bytes": n * (16 + 8 + 1), "flops": n * 20}
    if kind == "resize":
        e = 16 if case["double"] else 8
        n_in, n_out = case["rows"] * case["cols"], case["out_rows"] * case["out_cols"]
        return {"bytes": e * (n_in + n_out), "flops": 2 * 11 * n_out}
    P, S, px = case["pulses"], case["samples"], case["nu"] * case["nv"]
    N = sb.n_fft_for(S, case["upsample"])
    wide = 2 if case["precise"] else 1
    inputs = 8 * P * S + wide * 4 * (S + 3 * P)
    fft = P * (5 * N * math.log2(N) + 6 * S)
    if kind == "profiles":
        return {"bytes": inputs + 8 * P * N, "flops": fft}
    # a pixel and pulse: 18 single-precision instructions (most of them
    # fused multiply-adds) and 3 special functions
    pixels = 24 * px if case["locs"] or kind == "host" else 8 * (case["nu"] + case["nv"])
    return {"bytes": inputs + pixels + 16 * px + (px if case["u8"] else 0), "flops": fft + 39 * px * P}


# ---- the same in 64 bits, plain torch ----

def _taylor(n, level):
    """The reference's Taylor window (signal.h:14-51) up to 30 dB."""
    p10 = np.float32(10.0) ** np.float32(level / 20)
    A2 = (float(np.log(p10 + np.sqrt(p10 * p10 - np.float32(1)))) / math.pi) ** 2
    nbar = int(2 * A2 + 0.5) + 1
    sp2 = nbar ** 2 / (A2 + (nbar - 0.5) ** 2)
    xi = torch.linspace(-0.5, 0.5, n, dtype=torch.float64, device=GPU)
    w = torch.ones_like(xi)
    for m in range(1, nbar):
        num = den = 1.0
        for r in range(1, nbar):
            num *= (-1.0) ** (m + 1) * (1.0 - m * m / sp2 / (A2 + (r - 0.5) ** 2))
            if r != m:
                den *= 1.0 - float((m * m) // (r * r))
        w += num / den * torch.cos(2 * math.pi * m * xi)
    return w / w.max()


def _profiles64(c, a):
    """Windowed, filtered, padded, shifted and transformed rows, in pulse order."""
    P, S, N = c["pulses"], c["samples"], a["n_fft"]
    k = a["k_r"] if c["precise"] else a["k_r"].float().double()
    x = a["phs"].to(torch.complex128) * (k.abs() * _taylor(S, c["taylor"]))[None, :] * _taylor(P, c["taylor"])[:, None]
    x = x.roll(-(2 * (P // 2 + P % 2)) % P, 0)
    pad = torch.zeros(P, N, dtype=torch.complex128, device=GPU)
    at = (N - S) // 2
    lo, hi = max(0, -at), min(S, N - at)
    pad[:, lo + at:hi + at] = x[:, lo:hi]
    return torch.fft.fft(pad.roll(-(N // 2), 1), dim=1).roll(-(N // 2), 1)


def _image64(c, a):
    P, S, N = c["pulses"], c["samples"], a["n_fft"]
    Q = _profiles64(c, a)
    pos = a["pos"] if c["precise"] else a["pos"].float().double()
    k_c = float(a["k_r"][S // 2] if c["precise"] else a["k_r"][S // 2].float())
    if c["precise"]:
        norm = pos.norm(dim=1)
    else:  # the reference's |pos| is a single-precision value
        f = a["pos"].float()
        norm = torch.sqrt(f[:, 0] * f[:, 0] + f[:, 1] * f[:, 1] + f[:, 2] * f[:, 2]).double()
    lsa, lsb = math.floor(-S * a["delta_r"] / 2), math.floor(S * a["delta_r"] / 2)
    inv = (N - 1) / (lsb - lsa)
    r = _locs(a)
    img = torch.zeros(r.shape[1], dtype=torch.complex128, device=GPU)
    phasor = lambda ph: torch.polar(torch.ones_like(ph), ph)  # noqa: E731
    dist = lambda p: norm[p] - ((r - pos[p][:, None]) ** 2).sum(0).sqrt()  # noqa: E731
    for p in range(P):
        dr = dist(p)
        t = (dr - lsa) * inv
        low = t.floor()
        q = Q[p]
        i = low.long()
        q0, q1 = q[i.clamp(0, N - 1)], q[(i + 1).clamp(0, N - 1)]
        img += (q0 + (q1 - q0) * (t - low)) * phasor(dr * -k_c)
    img *= phasor(dist(P // 2) * k_c)
    return img.reshape(c["nv"], c["nu"]).flip(0)


def _resize64(case, src):
    x = src.double()
    shape, out = (case["rows"], case["cols"]), (case["out_rows"], case["out_cols"])
    lo, hi = x.amin((0, 1)), x.amax((0, 1))

    def mirror(i, n):
        if n == 1:
            return torch.zeros_like(i)
        i = i.abs() % (2 * n - 2)
        return torch.where(i >= n, 2 * n - 2 - i, i)

    shrinks = any(o < n for n, o in zip(shape, out))
    for ax in (0, 1):
        sigma = (shape[ax] / out[ax] - 1) / 2
        if shrinks and sigma > 1e-15:
            rad = int(4 * sigma + 0.5)
            w = torch.exp(-0.5 / sigma ** 2 * torch.arange(-rad, rad + 1, dtype=torch.float64) ** 2)
            w /= w.sum()
            i = torch.arange(shape[ax], device=GPU)
            x = sum(float(w[j + rad]) * x.index_select(ax, mirror(i + j, shape[ax])) for j in range(-rad, rad + 1))
    for ax in (0, 1):
        n = shape[ax]
        cc = (torch.arange(out[ax], dtype=torch.float64, device=GPU) + 0.5) * (n / out[ax]) - 0.5
        if n == 1:
            cc = torch.zeros_like(cc)
        cc = cc.abs()
        cc = torch.where(cc > n - 1, 2 * (n - 1) - cc, cc)
        f = cc.floor()
        i, t = f.long(), cc - f
        t = t[:, None, None] if ax == 0 else t[None, :, None]
        x = x.index_select(ax, mirror(i, n)) * (1 - t) + x.index_select(ax, mirror(i + 1, n)) * t
    return torch.minimum(torch.maximum(x, lo), hi)


def exact(case, seed):
    kind = case["kind"]
    if kind == "output":
        img = prepare(case, seed)["img"]
        a = img.abs()
        return [10.0 * torch.log(a / a.max()) / float(np.log(np.float32(10.0))), None]
    if kind == "resize":
        return _resize64(case, prepare(case, seed)["src"])
    if kind == "profiles":
        return _profiles64(case, _aperture(dict(case, nu=1, nv=1), seed))
    pair = lambda c, z: [z, None] if c["u8"] else [z]  # noqa: E731
    if kind in ("batch", "plan"):
        return [pair(c, _image64(c, _aperture(c, seed * 100 + i))) for i, c in enumerate(_mix(case))]
    if case["nu"] * case["nv"] * case["pulses"] > 1 << 34:
        return None
    z = _image64(case, _aperture(case, seed))
    return z if kind == "host" else [pair(case, z)]
