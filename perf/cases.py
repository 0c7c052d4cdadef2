"""The engine's workloads for performance measurement.

Every case is a dict of plain values.  Its "call" names the public entry
point that run() makes one pass through:

  focus       Plan.focus, device arrays: range compression + backprojection
  focus_host  Plan.focus, numpy arrays: the same with the copies in and out
  hypotheses  Plan.backproject_hypotheses: images of H antenna tracks from one
              set of range profiles
  autofocus   one step of a gradient autofocus: autograd.backproject, image
              entropy, backward to the 12 cubic track coefficients and the
              per-pulse slant-range offsets
  batch       Batch.focus: uneven scenes in one launch
  mf          Plan.matched_filter

Scenes are the synthetic stepped-frequency apertures of scenes.py (point
scatterers, circular track, complex Gaussian noise at 20 dB), made on the GPU
from the seed.  The track is jittered by a centimetre and the slant range is
its distance to the scene centre, as a measured aperture has it.
"""
import math

import numpy as np
import torch

from uncc_sar_focusing_b200 import autograd, focusing, scenes

C = 299792458.0
TAU = 2.0 * math.pi

# the point-target configuration's geometry (scenes.point_target_scene)
POINT = dict(fc=9.6e9, bw=600e6, radius=10e3, el=30.0, span=4.0, spacing=0.08, window="hamming")


def listed():
    p = POINT
    return [
        # a preview chip from a short sub-aperture: latency and launches count
        dict(name="focus_chip", call="focus", precision="mixed", K=64, pulses=48, nfft=512, nx=32, ny=32, nz=1,
             targets=3, **p),
        # the point-target configuration: 424 is not a power of two
        dict(name="focus_points", call="focus", precision="mixed", K=424, pulses=512, nfft=3392, nx=256, ny=256, nz=1,
             targets=5, **p),
        # the same through host buffers, as the reference's callers hold them
        dict(name="focus_points_host", call="focus_host", precision="mixed", K=424, pulses=512, nfft=3392, nx=256,
             ny=256, nz=1, targets=5, **p),
        # an aperture and a grid as a user happens to have them, untapered
        dict(name="focus_ragged", call="focus", precision="mixed", K=501, pulses=777, nfft=4008, nx=333, ny=517, nz=1,
             targets=40, **{**p, "window": "none"}),
        # the large configuration
        dict(name="focus_large", call="focus", precision="mixed", K=1024, pulses=2048, nfft=8192, nx=1024, ny=1024,
             nz=1, targets=200, fc=9.6e9, bw=640e6, radius=8e3, el=45.0, span=30.0, spacing=100.0 / 1023,
             window="hamming"),
        # full-circle volume, a stack of z-slices
        dict(name="focus_volume", call="focus", precision="mixed", K=512, pulses=2048, nfft=4096, nx=128, ny=128,
             nz=16, targets=100, fc=9.6e9, bw=600e6, radius=10e3, el=30.0, span=360.0, spacing=10.0 / 127,
             window="hamming"),
        # all-FP64 path: the point-target configuration, and the autofocus grid
        dict(name="focus_points_fp64", call="focus", precision="fp64", K=424, pulses=512, nfft=3392, nx=256, ny=256,
             nz=1, targets=5, **p),
        dict(name="focus_wide_fp64", call="focus", precision="fp64", K=512, pulses=1024, nfft=4096, nx=512, ny=512,
             nz=1, targets=5, **p),
        # a grid-search batch of motion hypotheses
        dict(name="hypotheses_24", call="hypotheses", precision="mixed", K=512, pulses=1024, nfft=4096, nx=256, ny=256,
             nz=1, tracks=24, targets=5, **p),
        # one descent step of the autofocus configuration (forward and backward)
        dict(name="autofocus_step", call="autofocus", precision="mixed", K=512, pulses=1024, nfft=4096, nx=512, ny=512,
             nz=1, targets=5, **p),
        # independent scenes of uneven sizes in one launch
        dict(name="batch_uneven", call="batch", precision="mixed", K=512, pulses=1024, nfft=4096, nx=512, ny=512, nz=1,
             scenes=10, targets=20, **p),
        # the matched-filter image of a small scene
        dict(name="matched_filter", call="mf", precision="mixed", K=256, pulses=128, nfft=2048, nx=96, ny=96, nz=1,
             targets=5, **p),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# pixel-pulses (matched filter: sample-pixel-pulses) of the largest drawn case
_MOST = {"focus": 2.0e9, "focus64": 2.2e8, "focus_host": 1.0e8, "hypotheses": 2.0e9, "autofocus": 4.0e8,
         "batch": 1.5e9, "mf": 5.0e8}


def draw(rng):
    call = rng.choice(["focus", "focus", "focus", "focus64", "focus_host", "hypotheses", "autofocus", "batch", "mf"])
    K = rng.choice([_log_int(rng, 48, 1024), 256, 512, 1024])
    if call == "mf":
        K = _log_int(rng, 48, 400)
    up = rng.choice([4, 8, 8])
    pulses = _log_int(rng, 40, 2048)
    nx, ny, nz = _log_int(rng, 24, 1024), _log_int(rng, 24, 1024), 1
    if call == "focus" and rng.random() < 0.25:
        nz = rng.randint(2, 16)
    case = dict(call="focus" if call == "focus64" else call, precision="fp64" if call == "focus64" else "mixed", K=K,
                targets=rng.randint(2, 60))
    case.update(POINT, span=rng.choice([4.0, 30.0, 360.0]), radius=rng.choice([8e3, 10e3]),
                el=rng.choice([30.0, 45.0]), spacing=rng.uniform(0.05, 0.12), window=rng.choice(["hamming", "none"]))
    # an image stays inside the unambiguous swath
    reach = max(24, int(0.7 * _swath(case) / case["spacing"]))
    nx, ny = min(nx, reach), min(ny, reach)
    many = 1
    if call == "hypotheses":
        case["tracks"] = many = rng.randint(3, 48)
    if call == "batch":
        case["scenes"] = many = rng.randint(3, 16)
    work = lambda: nx * ny * nz * pulses * many * (K if call == "mf" else 1)  # noqa: E731
    while work() > _MOST[call]:
        nx, ny, nz, pulses = max(24, int(nx * 0.85)), max(24, int(ny * 0.85)), max(1, nz - 1), max(24, int(pulses * 0.95))
    case.update(pulses=pulses, nx=nx, ny=ny, nz=nz, nfft=up * K)
    return case


# ---- inputs ----------------------------------------------------------------

def _delta_freq(c):
    return c["bw"] / (c["K"] - 1)


def _grid(c):
    d = c["spacing"]
    return scenes.Grid(nx=c["nx"], ny=c["ny"], nz=c["nz"], wx=d * (c["nx"] - 1), wy=d * (c["ny"] - 1),
                       wz=d * (c["nz"] - 1))


def _swath(c):
    return C / (2.0 * _delta_freq(c))


def _aperture(c, rng):
    """(phase history, ant_x, ant_y, ant_z, slant_range, start_freq) on the GPU."""
    n, K, df = c["pulses"], c["K"], _delta_freq(c)
    ax, ay, az = scenes.circular_track(n, c["radius"], c["el"], rng.uniform(-180.0, 180.0), c["span"])
    ant = np.stack([ax, ay, az], 1) + rng.normal(0.0, 0.01, (n, 3))
    r0 = np.sqrt((ant * ant).sum(1))
    f0 = np.full(n, c["fc"] - c["bw"] / 2.0)
    # scatterers over the image, inside the unambiguous swath
    T = c["targets"]
    half = np.array([c["nx"] - 1, c["ny"] - 1, c["nz"] - 1]) * c["spacing"] / 2.0
    pos = rng.uniform(-1.0, 1.0, (T, 3)) * np.minimum(half, 0.2 * _swath(c))
    amp = rng.rayleigh(1.0, T) * np.exp(1j * rng.uniform(0.0, TAU, T))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    a, r, x, g = dev(ant), dev(r0), dev(pos), dev(amp)
    f = f0[0] + df * torch.arange(K, dtype=torch.float64, device="cuda")
    ph = torch.zeros((n, K), dtype=torch.complex64, device="cuda")
    step = max(1, (1 << 25) // (n * K))
    for t in range(0, T, step):
        dR = (a[:, None, :] - x[None, t:t + step, :]).square().sum(-1).sqrt() - r[:, None]
        rev = dR[:, :, None] * (f * (-2.0 / C))
        ang = ((rev - rev.round()) * TAU).float()
        ph += (torch.polar(torch.ones_like(ang), ang) * g[None, t:t + step, None].to(torch.complex64)).sum(1)
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 30)))
    noise = torch.randn((n, K, 2), generator=gen, device="cuda")
    sigma = (ph.abs().square().mean() * 10.0 ** -2.0 / 2.0).sqrt()
    ph = (ph + torch.view_as_complex(noise) * sigma).contiguous()
    return (ph, a[:, 0].contiguous(), a[:, 1].contiguous(), a[:, 2].contiguous(), r, dev(f0))


def _plan(c):
    return focusing.Plan(c["K"], c["pulses"], c["nfft"], _swath(c), _grid(c), precision=c["precision"],
                         window=c["window"])


def _batch_cases(c):
    """The scenes of a batch: sizes around the case's, spread by a factor of about two either way."""
    rng = np.random.default_rng(c["scenes"] * 1009 + c["nx"])
    out = []
    for _ in range(c["scenes"]):
        s = dict(c)
        size = lambda v: max(16, int(v * math.exp(rng.uniform(-0.9, 0.3))))  # noqa: E731
        s.update(nx=size(c["nx"]), ny=size(c["ny"]), pulses=size(c["pulses"]))
        out.append(s)
    return out


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 17])
    call = case["call"]
    st = {"case": case}
    if call == "batch":
        subs = _batch_cases(case)
        st["apertures"] = [_aperture(s, rng) for s in subs]
        sc = [scenes.Scene("scene", ap[0], ap[1], ap[2], ap[3], ap[4], ap[5], _delta_freq(s), s["nfft"], _grid(s),
                           window=s["window"]) for s, ap in zip(subs, st["apertures"])]
        st["batch"] = focusing.Batch(sc)
        st["images"] = st["batch"].new_images()
        return st
    ap = _aperture(case, rng)
    st["plan"] = plan = _plan(case)
    if call == "focus_host":
        st["aperture"] = [v.cpu().numpy() for v in ap]
        return st
    st["aperture"] = ap
    if call == "hypotheses":
        H, n = case["tracks"], case["pulses"]
        tau = scenes.slow_time(n)
        err = np.stack([scenes.cubic_track_error(rng.uniform(-0.1, 0.1, (3, 4)), tau) for _ in range(H)])  # [H, 3, n]
        e = torch.as_tensor(err).cuda()
        st["tracks"] = [(ap[1 + i][None, :] + e[:, i, :]).contiguous() for i in range(3)] + [
            v[None, :].expand(H, n).contiguous() for v in (ap[4], ap[5])]
        plan.range_compress(ap[0])
    if call == "autofocus":
        # the measured track is off by a cubic of a few centimetres; the
        # corrections are FP32 parameters on top of the FP64 track
        n = case["pulses"]
        tau = scenes.slow_time(n)
        e = torch.as_tensor(scenes.cubic_track_error(rng.uniform(-0.03, 0.03, (3, 4)), tau)).cuda()
        st["track"] = torch.stack(ap[1:4]) + e
        st["powers"] = torch.as_tensor(np.stack([tau ** k for k in range(4)])).cuda()
        st["theta"] = torch.zeros((3, 4), device="cuda", requires_grad=True)
        st["offset"] = torch.zeros(n, device="cuda", requires_grad=True)
        plan.range_compress(ap[0])
    return st


def run(st):
    call = st["case"]["call"]
    if call == "batch":
        st["batch"].focus(st["apertures"], st["images"])
        return st["images"]
    plan = st["plan"]
    if call in ("focus", "focus_host"):
        return plan.focus(*st["aperture"])
    if call == "mf":
        return plan.matched_filter(*st["aperture"])
    if call == "hypotheses":
        return plan.backproject_hypotheses(*st["tracks"])
    theta, offset = st["theta"], st["offset"]
    theta.grad = offset.grad = None
    a = st["track"] + theta.double() @ st["powers"]
    img = autograd.backproject(plan, a[0].contiguous(), a[1].contiguous(), a[2].contiguous(),
                               st["aperture"][4] + offset.double(), st["aperture"][5])
    e = autograd.image_entropy(img)
    e.backward()
    return {"entropy": e.detach(), "image": img.detach(), "theta_grad": theta.grad, "offset_grad": offset.grad}


# ---- what a pass cannot do without ---------------------------------------

def work(case):
    """Inputs read once, outputs written once; 26 flops per pixel-pulse of
    backprojection (10 of range geometry, 16 of interpolation and rotation),
    twice that again for the adjoint, 8 per sample of the matched filter and
    5 N log2 N per range profile."""
    if case["call"] == "batch":
        parts = [work({**s, "call": "focus"}) for s in _batch_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    esz = 16 if case["precision"] == "fp64" else 8
    n, K, npix = case["pulses"], case["K"], case["nx"] * case["ny"] * case["nz"]
    profiles = n * case["nfft"]
    compress = 5.0 * profiles * math.log2(case["nfft"])
    if case["call"] == "mf":
        return {"bytes": 8.0 * n * K + 40.0 * n + esz * npix, "flops": 8.0 * npix * n * K}
    if case["call"] == "hypotheses":
        H = case["tracks"]
        return {"bytes": float(esz * profiles + H * (40 * n + esz * npix)), "flops": 26.0 * npix * n * H}
    if case["call"] == "autofocus":
        return {"bytes": float(esz * profiles + 40 * n + 3 * esz * npix + 4 * n), "flops": 78.0 * npix * n}
    return {"bytes": float(8 * n * K + 40 * n + esz * npix), "flops": 26.0 * npix * n + compress}


# ---- the same in 64 bits, torch alone ---------------------------------------

def _taper(c):
    K = c["K"]
    if c["window"] == "none":
        return torch.ones(K, dtype=torch.float64, device="cuda")
    k = torch.arange(K, dtype=torch.float64, device="cuda")
    return 0.54 - 0.46 * torch.cos(TAU * k / (K - 1))


def _profiles64(c, ph):
    x = ph.to(torch.complex128) * _taper(c)
    return torch.fft.fftshift(torch.fft.ifft(x, n=c["nfft"], dim=1), dim=1)


def _pixels(c):
    ax = []
    for n in (c["nz"], c["nx"], c["ny"]):
        w = c["spacing"] * (n - 1)
        ax.append(-0.5 * w + torch.arange(n, dtype=torch.float64, device="cuda") * c["spacing"])
    z, x, y = torch.meshgrid(*ax, indexing="ij")
    return x.reshape(-1), y.reshape(-1), z.reshape(-1)


def _chunks(c, ap, rc, x, y, z):
    """Per group of pulses: (pulse slice, unit vector parts, profile sample, its slope per metre, rotation)."""
    npix, n, N = x.numel(), c["pulses"], c["nfft"]
    lam = N / _swath(c)
    step = max(1, (1 << 24) // npix)
    for p in range(0, n, step):
        q = slice(p, min(n, p + step))
        d = [v[q, None] - u[None, :] for v, u in zip(ap[1:4], (x, y, z))]
        R = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt()
        dR = R - ap[4][q, None]
        b = dR * lam + 0.5 * N
        ok = (b > 0) & (b < N - 1)
        i = torch.where(ok, b.floor(), torch.zeros_like(b)).long()
        v0, v1 = torch.gather(rc[q], 1, i), torch.gather(rc[q], 1, i + 1)
        rev = dR * (ap[5][q, None] * (2.0 / C))
        ang = (rev - rev.round()) * TAU
        slope = torch.where(ok, v1 - v0, torch.zeros_like(v0))
        val = torch.where(ok, v0, torch.zeros_like(v0)) + slope * (b - i)
        yield q, [u / R for u in d], val, slope * lam, torch.polar(torch.ones_like(ang), ang)


def _image64(c, ap, rc):
    x, y, z = _pixels(c)
    img = torch.zeros(x.numel(), dtype=torch.complex128, device="cuda")
    for _, _, val, _, rot in _chunks(c, ap, rc, x, y, z):
        img += (val * rot).sum(0)
    return img.reshape(c["nz"], c["nx"], c["ny"])


def _matched64(c, ap):
    x, y, z = _pixels(c)
    w, K = _taper(c), c["K"]
    k = torch.arange(K, dtype=torch.float64, device="cuda")
    img = torch.zeros(x.numel(), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 24) // K)
    for p in range(c["pulses"]):
        s = ap[0][p].to(torch.complex128) * w
        f = (ap[5][p] + k * _delta_freq(c)) * (2.0 / C)
        for q in range(0, x.numel(), step):
            o = slice(q, q + step)
            dR = ((ap[1][p] - x[o]).square() + (ap[2][p] - y[o]).square() + (ap[3][p] - z[o]).square()).sqrt() - ap[4][p]
            rev = dR[:, None] * f[None, :]
            ang = (rev - rev.round()) * TAU
            img[o] += torch.polar(torch.ones_like(ang), ang) @ s
    return img.reshape(c["nz"], c["nx"], c["ny"])


def _autofocus64(c, st):
    ap = (st["aperture"][0], *st["track"], st["aperture"][4], st["aperture"][5])
    rc = _profiles64(c, ap[0])
    img = _image64(c, ap, rc)
    w = img.abs().square()
    S = w.sum()
    logp = torch.log((w / S).clamp_min(1e-30))
    E = -(w / S * logp).sum()
    G = (-2.0 * img * (logp + E) / S).reshape(-1)
    x, y, z = _pixels(c)
    ga = torch.zeros((3, c["pulses"]), dtype=torch.float64, device="cuda")
    gr = torch.zeros(c["pulses"], dtype=torch.float64, device="cuda")
    for q, u, val, slope, rot in _chunks(c, ap, rc, x, y, z):
        kr = TAU * ap[5][q, None] * (2.0 / C)
        s = ((slope + 1j * kr * val) * rot * G.conj()[None, :]).real
        for i in range(3):
            ga[i, q] = (s * u[i]).sum(1)
        gr[q] = -s.sum(1)
    return {"entropy": E, "image": img, "theta_grad": ga @ st["powers"].T, "offset_grad": gr}


def exact(case, seed):
    call = case["call"]
    if call in ("batch", "focus", "focus_host", "mf"):
        rng = np.random.default_rng([int(seed), 17])
        if call == "batch":
            subs = _batch_cases(case)
            aps = [_aperture(s, rng) for s in subs]
            return [_image64(s, ap, _profiles64(s, ap[0])) for s, ap in zip(subs, aps)]
        ap = _aperture(case, rng)
        if call == "mf":
            return _matched64(case, ap)
        img = _image64(case, ap, _profiles64(case, ap[0]))
        return img.cpu().numpy() if call == "focus_host" else img
    st = prepare(case, seed)
    if call == "autofocus":
        return _autofocus64(case, st)
    rc = _profiles64(case, st["aperture"][0])
    imgs = [_image64(case, (None, *[v[h] for v in st["tracks"]]), rc) for h in range(case["tracks"])]
    return torch.stack(imgs)
