"""The measured workloads of the focusing engine: fixed-point and float frames, split-precision frames,
autofocus gradients and the display scaling, each through the public entry points of ``pfa_b200``.

A case is a dict of plain values.  ``kind`` names the entry point:

* ``fixed``      ``FixedPlan.form`` / ``FixedPlan.form_iq16`` (uint16 image)
* ``float``      ``FloatPlan.form`` (FP32, ``detect`` "mag", "power" or "complex")
* ``mixed``      ``FloatPlan(mixed=True).form``
* ``autofocus``  ``autofocus.entropy_grad`` (entropy and its gradient, i.e. forward and backward)
* ``display``    ``geocode.display_u8`` of a detected image

``m`` pulses by ``n`` samples; ``grid`` is the fixed-point raster; ``rs`` / ``az`` choose the 32-tap sinc for
the range and the cross pass (otherwise the 2-tap lerp); ``jitter`` displaces the pulse angles by that
fraction of their spacing, so that the sort of tan(phi) is a real permutation.
"""
import math
import os
import sys
from fractions import Fraction

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpfs250t-sar-ifp_b200"))
from pfa_b200 import autofocus, engine, geocode, geometry, synth  # noqa: E402

C = 299_792_458.0
FC = 9.6e9                     # X band, as the Umbra collects
HALF_APERTURE = math.radians(1.5)
TARGETS = 32


def listed():
    return [
        # the smallest frame a host forms: latency, launches
        dict(name="fixed_256x240_sinc", kind="fixed", m=256, n=240, grid=256, rs=True, az=True, iq=False, bw=600e6, jitter=0.3),
        # the emulator's default interpolators on a decimated scene
        dict(name="fixed_1000x937_lerp", kind="fixed", m=1000, n=937, grid=1024, rs=False, az=False, iq=False, bw=600e6, jitter=0.0),
        # a scene whose signal arrives as the board's int16 I/Q
        dict(name="fixed_2962x3755_iq16_sinc", kind="fixed", m=2962, n=3755, grid=4096, rs=True, az=True, iq=True, bw=300e6, jitter=0.1),
        # the production fixed-point frame (Centerfield shape, --range-sinc --az-sinc)
        dict(name="fixed_5634x4319_sinc", kind="fixed", m=5634, n=4319, grid=8192, rs=True, az=True, iq=False, bw=113.6e6, jitter=0.0),
        # the small float scene
        dict(name="float_1024_lerp", kind="float", m=1024, n=1024, rs=False, az=False, detect="mag", bw=600e6, jitter=0.0),
        # an uneven scene of the batch whose complex image goes on to further processing
        dict(name="float_2326x2054_sinc_complex", kind="float", m=2326, n=2054, rs=True, az=True, detect="complex", bw=600e6, jitter=0.1),
        # the production float frame (NDSU shape), both interpolators
        dict(name="float_8167x8192_lerp", kind="float", m=8167, n=8192, rs=False, az=False, detect="mag", bw=600e6, jitter=0.0),
        dict(name="float_8167x8192_sinc", kind="float", m=8167, n=8192, rs=True, az=True, detect="mag", bw=600e6, jitter=0.0),
        # the tensor-core mode on an uneven scene
        dict(name="mixed_4133x3001_lerp", kind="mixed", m=4133, n=3001, rs=False, az=False, detect="mag", bw=600e6, jitter=0.1),
        # the autofocus scene, and an uneven one through the sinc passes
        dict(name="autofocus_4096_lerp", kind="autofocus", m=4096, n=4096, rs=False, az=False, bw=600e6, jitter=0.0),
        dict(name="autofocus_1379x2755_sinc", kind="autofocus", m=1379, n=2755, rs=True, az=True, bw=600e6, jitter=0.1),
        # the map product of the production frame
        dict(name="display_8192x8192", kind="display", m=8192, n=8192),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fixed", "fixed", "float", "float", "mixed", "autofocus", "display"])
    if kind == "display":
        return dict(kind=kind, m=_size(rng, 64, 8192), n=_size(rng, 64, 8192))
    lo, hi = {"fixed": (200, 5634), "float": (200, 8167), "mixed": (1025, 4133), "autofocus": (200, 3000)}[kind]
    c = dict(kind=kind, m=_size(rng, lo, hi), n=_size(rng, lo, hi), rs=rng.random() < 0.6, az=rng.random() < 0.6,
             bw=rng.choice([113.6e6, 300e6, 600e6]), jitter=rng.choice([0.0, 0.1, 0.3]))
    if kind == "fixed":
        c["grid"] = geometry.pow2(max(c["m"], c["n"]))
        c["iq"] = rng.random() < 0.3
    elif kind in ("float", "mixed"):
        c["detect"] = rng.choice(["mag", "mag", "power", "complex"])
    return c


# ------------------------------------------------------------------------------------------ inputs
def _scene(case, seed):
    """Pulse positions and frequencies of a spotlight collect (float64 host arrays), SRP at the origin."""
    m, n, bw = case["m"], case["n"], case["bw"]
    rng = np.random.default_rng(seed)
    th = np.linspace(-HALF_APERTURE, HALF_APERTURE, m)
    th = th + rng.uniform(-1.0, 1.0, m) * case["jitter"] * (2 * HALF_APERTURE / max(m - 1, 1))
    apc = np.stack([10_000.0 * np.cos(th), 10_000.0 * np.sin(th), np.full(m, 3_000.0)], axis=1)
    sc = synth.Scene(signal=None, tx=apc.copy(), rcv=apc.copy(), srp=np.zeros((m, 3)), sc0=np.full(m, FC - bw / 2),
                     scss=np.full(m, bw / n), mn=(m, n))
    return sc, rng


def _look(sc):
    los = sc.srp - 0.5 * (sc.tx + sc.rcv)
    u = los / np.linalg.norm(los, axis=1, keepdims=True)
    return u @ sc.uiax, u @ sc.uiay


def _signal(case, sc, rng, seed):
    """Point targets plus clutter 10 dB below them: (m, n) complex64 on the GPU."""
    m, n, bw = case["m"], case["n"], case["bw"]
    ax, ay = _look(sc)
    half = 0.35 * min((n - 1) * C / (2 * bw), (m - 1) * (C / FC) / (4 * HALF_APERTURE))
    tgt = rng.uniform(-half, half, (TARGETS, 2))
    amp = (rng.standard_normal(TARGETS) + 1j * rng.standard_normal(TARGETS)) / math.sqrt(2.0)
    d = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    proj = d(ax)[:, None] * d(tgt[:, 0])[None, :] + d(ay)[:, None] * d(tgt[:, 1])[None, :]          # (m, P)
    ph0, dph = (4 * math.pi / C) * d(sc.sc0)[:, None] * proj, (4 * math.pi / C) * d(sc.scss)[:, None] * proj
    blk = 64
    q = torch.arange(-(-n // blk), device="cuda", dtype=torch.float64) * blk
    r = torch.arange(blk, device="cuda", dtype=torch.float64)
    out = torch.empty((m, n), dtype=torch.complex64, device="cuda")
    for i in range(0, m, 512):
        pa, pb = ph0[i:i + 512, None, :] + q[None, :, None] * dph[i:i + 512, None, :], dph[i:i + 512, :, None] * r
        a = (torch.polar(torch.ones_like(pa), pa) * d(amp)).to(torch.complex64)
        b = torch.polar(torch.ones_like(pb), pb).to(torch.complex64)
        out[i:i + 512] = torch.bmm(a, b).reshape(a.shape[0], -1)[:, :n]
    g = torch.Generator(device="cuda").manual_seed(seed + 17)
    level = float(out.abs().square().mean()) * 0.1
    noise = torch.randn((m, n, 2), generator=g, device="cuda") * math.sqrt(level / 2)
    return out + torch.view_as_complex(noise)


def _theta(case, rng):
    """Quadratic phase error with 3 rad at the aperture edges plus a random walk."""
    u = np.linspace(-1.0, 1.0, case["m"])
    return (3.0 * u * u + np.cumsum(rng.normal(0.0, 0.05, case["m"]))).astype(np.float32)


def _image(case, seed):
    """A detected image: Rayleigh speckle with bright responses."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.randn((case["m"], case["n"], 2), generator=g, device="cuda")
    mag = z.square().sum(-1).sqrt()
    bright = torch.randint(0, case["m"] * case["n"], (case["m"] * case["n"] // 512 + 1,), generator=g, device="cuda")
    mag.view(-1)[bright] *= 40.0
    return mag * 1234.5


def _iq16(sig):
    """The board's sig.bin: int16 I/Q on a block exponent."""
    x = torch.view_as_real(sig)
    e = math.ceil(math.log2(float(x.abs().max()) / 32767.0))
    return torch.floor(x * 2.0 ** -e).clamp(-32768, 32767).to(torch.int16).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "display":
        return dict(case=case, mag=_image(case, seed))
    sc, rng = _scene(case, seed)
    sig = _signal(case, sc, rng, seed)
    tables = geometry.prepare_tables_from_scene_fast(sc)
    st = dict(case=case)
    if kind == "fixed":
        st["plan"] = engine.FixedPlan(case["m"], case["n"], case["grid"], case["rs"], case["az"])
        st["sig"] = _iq16(sig) if case["iq"] else sig
        st["img"] = torch.empty((case["grid"], case["grid"]), dtype=torch.uint16, device="cuda")
    else:
        p = st["plan"] = engine.FloatPlan(case["m"], case["n"], case["rs"], case["az"], mixed=kind == "mixed")
        st["sig"] = sig
        if kind == "autofocus":
            st["theta"] = torch.from_numpy(_theta(case, rng)).cuda()
            st["dtheta"] = torch.empty_like(st["theta"])
            st["entropy"] = torch.empty((), dtype=torch.float64, device="cuda")
        else:
            dt = torch.complex64 if case["detect"] == "complex" else torch.float32
            st["img"] = torch.empty((p.m2, p.n2), dtype=dt, device="cuda")
    st["plan"].set_tables(tables)
    return st


def run(st):
    c = st["case"]
    if c["kind"] == "display":
        out, hi = geocode.display_u8(st["mag"])
        return {"display": out, "hi": hi}
    if c["kind"] == "fixed":
        img = st["plan"].form_iq16(st["sig"], out=st["img"]) if c["iq"] else st["plan"].form(st["sig"], out=st["img"])
        return img.view(torch.int16)               # the same bits, in a type that every torch operation takes
    if c["kind"] == "autofocus":
        ent, g = autofocus.entropy_grad(st["plan"], st["sig"], st["theta"], st["dtheta"], st["entropy"])
        return {"entropy": ent, "dtheta": g}
    return st["plan"].form(st["sig"], out=st["img"], detect=c["detect"])


# ------------------------------------------------------------------------------------------ work
def work(case):
    m, n, kind = case["m"], case["n"], case["kind"]
    if kind == "display":
        return {"bytes": 5 * m * n, "flops": 3 * m * n}
    tap = {False: 2, True: 32}
    fft = lambda lines, size: 5.0 * lines * size * math.log2(size)  # noqa: E731
    if kind == "fixed":
        g = case["grid"]
        flops = m * n * 4.0 * (tap[case["rs"]] + tap[case["az"]]) + fft(n + g, g)
        return {"bytes": (4 if case["iq"] else 8) * m * n + 2 * g * g, "flops": flops}
    m2, n2 = geometry.pow2(m), geometry.pow2(n)
    flops = m * n * 4.0 * (tap[case["rs"]] + tap[case["az"]]) + fft(n, m2) + fft(m2, n2)
    if kind == "autofocus":
        return {"bytes": 8 * m * n + 8 * m, "flops": 2 * flops}
    return {"bytes": 8 * m * n + (8 if case["detect"] == "complex" else 4) * m2 * n2, "flops": flops}


# ------------------------------------------------------------------------------------------ exact
def _sinc_table():
    """The 256-phase, 32-tap Q15 sinc that defines the sinc interpolator, as float64 taps."""
    pi, tab = Fraction(math.pi), np.zeros((256, 32))
    for ph in range(256):
        d = [Fraction(ph, 256) + 15 - t for t in range(32)]
        w = [Fraction(1) if x == 0 else Fraction(math.sin(math.pi * float(x))) / (pi * x) for x in d]
        s = sum(w)
        q = [min(32767, max(-32768, math.floor(x * 32768 / s + Fraction(1, 2)))) for x in w]
        left = 32768 - sum(q)
        for t in sorted(range(32), key=lambda i: (-abs(q[i]), i)):
            add = max(min(left, 32767 - q[t]), -32768 - q[t])
            q[t] += add
            left -= add
        tab[ph] = q
    return torch.from_numpy(tab / 32768.0).cuda()


def _resample(x, xp, f, tab):
    """Rows of complex128 ``f`` on ascending sources ``xp`` at the ascending queries ``x`` (every row's), zero
    outside the sources' span; the 32-tap sinc where ``tab`` is given and all its taps exist, else the lerp."""
    n = xp.shape[1]
    k = torch.searchsorted(xp, x.expand(xp.shape[0], -1).contiguous(), right=True) - 1
    live = (x >= xp[:, :1]) & (x <= xp[:, -1:])
    k.clamp_(0, n - 2)
    a = xp.gather(1, k)
    frac = (x - a) / (xp.gather(1, k + 1) - a)
    g = f.gather(1, k)
    out = g + frac * (f.gather(1, k + 1) - g)
    if tab is not None:
        ph = (torch.round(frac * 32768.0).clamp(0, 32767).long() >> 7) * 32
        inner = (k >= 15) & (k <= n - 17)
        base = torch.where(inner, k - 15, 0)
        acc = 0
        for t in range(32):
            acc = acc + tab.view(-1)[ph + t] * f.gather(1, base + t)
        out = torch.where(inner, acc, out)
    return torch.where(live, out, 0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "fixed":
        return None                                # whole numbers
    if kind == "display":
        s = _image(case, seed).double().view(-1).sort().values
        at = (s.numel() - 1) * 0.997
        k = math.floor(at)
        return {"display": None, "hi": s[k] + (at - k) * (s[min(k + 1, s.numel() - 1)] - s[k])}
    m, n = case["m"], case["n"]
    sc, rng = _scene(case, seed)
    sig = _signal(case, sc, rng, seed).to(torch.complex128)
    theta = torch.from_numpy(_theta(case, rng)).cuda().double().requires_grad_() if kind == "autofocus" else None
    tab = _sinc_table() if case["rs"] or case["az"] else None
    ax, ay = _look(sc)
    dx, dy = ax.mean() / np.hypot(ax.mean(), ay.mean()), ay.mean() / np.hypot(ax.mean(), ay.mean())
    pr, pc = ax * dx + ay * dy, ay * dx - ax * dy
    freq = sc.sc0[:, None] + np.arange(n)[None, :] * sc.scss[:, None]
    kr = (2.0 * freq / C) * pr[:, None]
    lo, hi = kr[:, -1].min(), kr[:, 0].max()
    if lo > hi:
        lo, hi = kr.min(), kr.max()                # the reference's grid: the union of the pulses' spans
    KR = np.linspace(lo, hi, n)
    tan = pc / pr
    order = np.argsort(tan)
    kc = np.abs(KR).max() * np.abs(tan).max()
    KC = np.linspace(-kc, kc, m)
    d = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    p1 = _resample(d(KR), d(kr), sig, tab if case["rs"] else None)
    del sig
    if theta is not None:
        p1 = p1 * torch.polar(torch.ones_like(theta), -theta)[:, None]
    p1 = p1[d(order)].T.contiguous()                                                     # (n, m) range-bin rows
    g2 = _resample(d(KC), d(KR)[:, None] * d(tan[order])[None, :], p1, tab if case["az"] else None)
    del p1
    g2 = (g2 * d(np.hamming(n))[:, None] * d(np.hamming(m))[None, :]).T
    m2, n2 = 1 << (m - 1).bit_length(), 1 << (n - 1).bit_length()
    pad = torch.nn.functional.pad(torch.view_as_real(g2.contiguous()), (0, 0, 0, n2 - n, 0, m2 - m))
    pad = torch.view_as_complex(pad.contiguous())
    if kind == "autofocus":
        p = torch.fft.fft2(pad).abs().square()
        p = p / p.sum()
        ent = -torch.xlogy(p, p).sum()
        ent.backward()
        return {"entropy": ent.detach(), "dtheta": theta.grad}
    z = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(pad)))
    return z if case["detect"] == "complex" else z.abs().square() if case["detect"] == "power" else z.abs()
