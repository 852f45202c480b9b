"""Measured calls of the reconstruction path, through the package's public entry points.

Each case is one call (or, for the operators, one forward and one adjoint) as
a user's program makes it: a context created once for the acquisition's
geometry, buffers allocated once, then a call per stack.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs and context
    run(state)           one pass; returns its outputs whole
    work(case)           compulsory bytes and operations of one pass
    exact(case, seed)    the same outputs in 64 bits, in plain torch

Ranges: holograms of 256 to 2048 pixels a side, 8 or 16 bits, 1 to 600 of
them; fields of 64 to 512 pixels a side (powers of two, and the 250 of the
shipped configuration); volumes of 128 to 1024 voxels a side; Born and Rytov;
Volkov and Herraez unwrapping; device and page-locked host buffers.

Inputs are synthetic: Gaussian bodies whose analytic transform is sampled on
each illumination's Ewald cap, tilts on a spiral out to 0.9 NXMAX, and for
holograms an off-axis reference, shot noise, read noise and 12-bit (or 8-bit)
samples.  The aberration mask is background everywhere but the bodies and a
margin along the frame, where the extraction's window leaves no light and the
phase is noise.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mtd_transmission_gb300 import Context, Geometry

MEAN_E, REF_FRACTION, READ_SIGMA = 2000.0, 0.7, 3.0


def listed():
    return [
        # one camera frame checked while the user aligns the microscope: the smallest call
        dict(name="extract-frame", kind="extract", H=512, F=128, D=256, bits=8, n=1, born=1, volkov=1),
        # a whole acquisition's extraction, its spectra kept for later processing
        dict(name="extract-stack", kind="extract", H=1024, F=256, D=512, bits=16, n=400, born=0, volkov=1),
        # field formation of a small Born stack (unwrapping, aberration fits)
        dict(name="fields-born", kind="fields", H=512, F=128, D=256, bits=16, n=100, born=1, volkov=1),
        # field formation of a Rytov stack, large phase excursions
        dict(name="fields-rytov", kind="fields", H=1024, F=256, D=512, bits=16, n=200, born=0, volkov=1),
        # the configuration's other unwrapping method (VOLKOV 0) on part of a stack
        dict(name="fields-herraez", kind="fields", H=1024, F=256, D=512, bits=16, n=48, born=0, volkov=0),
        # volume from the fields of the shipped configuration (NXMAX 125), every output asked for
        dict(name="reconstruct-config", kind="reconstruct", H=1024, F=250, D=512, bits=16, n=500, born=0, volkov=1),
        # a quick look during an acquisition: few small frames to a small volume, latency counts
        dict(name="pipeline-preview", kind="pipeline", H=256, F=64, D=128, bits=8, n=8, born=1, volkov=1, host=0),
        # holograms on the device to the volume: 600 x 1024^2 to 512^3, Rytov
        dict(name="pipeline-rytov", kind="pipeline", H=1024, F=256, D=512, bits=16, n=600, born=0, volkov=1, host=0),
        # page-locked host holograms in, host volumes out: 100 x 512^2 to 256^3
        dict(name="pipeline-host", kind="pipeline", H=512, F=128, D=256, bits=16, n=100, born=0, volkov=1, host=1),
        # large frames and the largest volume: 64 x 2048^2 to 1024^3
        dict(name="pipeline-large", kind="pipeline", H=2048, F=512, D=1024, bits=16, n=64, born=0, volkov=1, host=0),
        # forward operator and adjoint of a user's own gradient method: 256^3, 400 caps
        dict(name="operators", kind="operators", H=512, F=128, D=256, bits=16, n=400, born=1, volkov=1),
        # regularised reconstruction, a few iterations between two looks at the result
        dict(name="tv", kind="tv", H=512, F=128, D=256, bits=16, n=400, born=1, volkov=1, iterations=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["extract", "fields", "fields", "reconstruct", "pipeline", "pipeline", "operators", "tv"])
    F = rng.choice([64, 128, 128, 250, 256, 512])
    if kind in ("operators", "tv"):
        F = rng.choice([64, 128])
    H = rng.choice([h for h in (256, 512, 1024, 2048) if 2 * F <= h])
    D = rng.choice([d for d in (128, 256, 512, 1024) if 2 * F <= d <= 4 * F + 24])
    if kind in ("operators", "tv"):
        D = 2 * F
    born = rng.choice([0, 1])
    volkov = 1
    if kind == "fields" and F <= 256 and rng.random() < 0.25:
        volkov = 0
    most = max(2, min(600, int(600 * (1024 / H) ** 2 * (256 / F) ** 0.5)))
    if D == 1024:
        most = min(most, 64)
    if not volkov:
        most = min(most, 48)
    c = dict(kind=kind, H=H, F=F, D=D, bits=rng.choice([8, 16, 16]), n=_log(rng, 1, most), born=born, volkov=volkov)
    if kind == "pipeline":
        # Born at the smallest fields only: in a weak object's volume the rounding of the phase along the
        # frame's dark edge, which the unwrapping spreads, outweighs every other difference at larger ones
        # (relative error 1e-4 against 64 bits, 2e-6 to 5e-6 for Rytov); Born fields are drawn by "fields"
        c["born"] = c["born"] if F == 64 else 0
        c["host"] = int(D <= 512 and rng.random() < 0.3)
    if kind == "tv":
        c["n"] = _log(rng, 20, 400)
        c["iterations"] = rng.randint(2, 8)
    if kind == "operators":
        c["n"] = _log(rng, 4, 500)
    return c


# ---------------------------------------------------------------- geometry
def _keys(c):
    H, F = c["H"], c["F"]
    g = dict(ccd_roix=H, nxmax=F // 2, circle_cx=H // 4, circle_cy=H // 4, dim_final=c["D"], born=c["born"], c_aber=1,
             deroul=1, volkov=c["volkov"], na=1.40, n0=1.515, lambda0=633e-9, f_tube=0.2, f_obj=0.002, tpcam=1e-5,
             rf=1.0, coef_na_obj_limit=1.0)
    if F == 250:  # the shipped configuration's carrier and optics
        g.update(circle_cx=H // 4 - 9 if H >= 1024 else H // 4, circle_cy=H - H // 4 + 9 if H >= 1024 else H // 4,
                 lambda0=632e-9, f_tube=0.15, tpcam=5.5e-6, rf=0.75)
    for k in ("na", "n0", "lambda0", "f_tube", "f_obj", "tpcam", "rf", "coef_na_obj_limit"):
        g[k] = float(np.float32(g[k]))  # the configuration reader's values are floats
    return g


def _rayon(g):
    return float(np.round(g["nxmax"] * g["n0"] / g["na"]))


def _tilts(n, N):
    k = np.arange(n, dtype=np.float64)
    r = 0.9 * N * np.sqrt((k + 0.5) / n)
    th = k * (math.pi * (3.0 - math.sqrt(5.0)))
    return np.stack([np.round(r * np.cos(th)), np.round(r * np.sin(th))], 1).astype(np.int64)


# ---------------------------------------------------------------- inputs
def _bodies(seed, born):
    r = np.random.default_rng(seed)
    out = []
    for _ in range(3):
        ax = r.uniform(0.05, 0.09, 3) if born else r.uniform(0.12, 0.2, 3)
        out.append((r.uniform(-0.06, 0.06, 3), ax, float(r.uniform(0.01, 0.05)), float(r.uniform(0.0, 0.004))))
    return out


def _ratio_fields(c, seed, tilts):
    """Object / background field ratio (n x F x F complex64), and the support of the bodies."""
    g = _keys(c)
    N, F, r = g["nxmax"], 2 * g["nxmax"], _rayon(g)
    f = torch.arange(-N, N, device="cuda", dtype=torch.float32)
    fy, fx = torch.meshgrid(f, f, indexing="ij")
    inside = fx * fx + fy * fy < N * N
    s = torch.sqrt(torch.clamp(r * r - fx * fx - fy * fy, min=1.0))
    bodies = _bodies(seed, c["born"])

    def cap(t):
        t = torch.as_tensor(t, device="cuda", dtype=torch.float32).reshape(-1, 2, 1, 1)
        qx, qy = fx - t[:, 0], fy - t[:, 1]
        qz = s - torch.sqrt(torch.clamp(r * r - t[:, 0] ** 2 - t[:, 1] ** 2, min=0.0))
        v = 0
        for ctr, ax, dn, kappa in bodies:
            w = torch.exp(-0.5 * math.pi ** 2 * ((ax[0] * qx) ** 2 + (ax[1] * qy) ** 2 + (ax[2] * qz) ** 2))
            ph = -2 * math.pi * (qx * ctr[0] + qy * ctr[1] + qz * ctr[2])
            v = v + complex(dn, kappa) * float(np.prod(ax)) * torch.polar(w, ph)
        v = torch.where(inside, 1j * v * (r / s), torch.zeros((), device="cuda", dtype=torch.complex64))
        return torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(v, dim=(-2, -1))), dim=(-2, -1))

    u0 = cap(np.zeros((1, 2)))[0]
    peak = 0.5 if c["born"] else 40.0 * F / 256  # rad
    im = peak / float(u0.imag.abs().max())
    out = torch.empty((len(tilts), F, F), dtype=torch.complex64, device="cuda")
    for a in range(0, len(tilts), 64):
        u = cap(tilts[a:a + 64])
        u = torch.complex(torch.clamp(u.real * im, -0.1, 0.1), u.imag * im)
        out[a:a + 64] = 1 + u if c["born"] else torch.exp(u)
    return out, u0.imag.abs() > 0.05 * float(u0.imag.abs().max())


def _mask(support):
    """Aberration mask (F x F uint8): background but for the bodies and the frame's margin."""
    F = support.shape[0]
    k = max(1, F // 32)
    grown = torch.nn.functional.max_pool2d(support.float()[None, None], 2 * k + 1, 1, k)[0, 0] > 0
    m = torch.full((F, F), 255, dtype=torch.uint8, device="cuda")
    m[grown] = 0
    e = max(3, F // 16)
    m[:e], m[-e:], m[:, :e], m[:, -e:] = 0, 0, 0, 0
    return m.cpu().numpy()


def _holograms(c, seed):
    g = _keys(c)
    H, F, n = c["H"], c["F"], c["n"]
    tilts = _tilts(n, g["nxmax"])
    ratio, support = _ratio_fields(c, seed, tilts)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = torch.uint16 if c["bits"] == 16 else torch.uint8
    gain, top = (1.0, 4095) if c["bits"] == 16 else (255 / 4095, 255)
    out = torch.empty((n, H, H), dtype=dtype, device="cuda")
    ar, ao = math.sqrt(MEAN_E * REF_FRACTION), math.sqrt(MEAN_E * (1 - REF_FRACTION))
    pad, step = (H - F) // 2, max(1, (1 << 25) // (H * H))
    x = torch.arange(H, device="cuda", dtype=torch.float64)
    for a in range(0, n, step):
        r = ratio[a:a + step]
        spec = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(r, dim=(-2, -1))), dim=(-2, -1))
        big = torch.zeros((len(r), H, H), dtype=torch.complex64, device="cuda")
        big[:, pad:pad + F, pad:pad + F] = spec
        o = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(big, dim=(-2, -1))), dim=(-2, -1)) * (H / F) ** 2
        t = torch.as_tensor(tilts[a:a + step], device="cuda", dtype=torch.float64)
        px = 2 * math.pi / H * ((g["circle_cx"] - H // 2 + t[:, 0:1]) * x % H)
        py = 2 * math.pi / H * ((g["circle_cy"] - H // 2 + t[:, 1:2]) * x % H)
        car = torch.polar(torch.ones_like(px), px).to(torch.complex64)[:, None, :] * \
            torch.polar(torch.ones_like(py), py).to(torch.complex64)[:, :, None]
        e = ar * ar + ao * ao * o.abs() ** 2 + 2 * ar * ao * (car * o).real
        e = torch.poisson(torch.clamp(e, min=0.0), generator=gen)
        e += READ_SIGMA * torch.randn(e.shape, generator=gen, device="cuda")
        out[a:a + step] = torch.clamp(torch.round(e * gain), 0, top).to(torch.int32).to(dtype)
    return out, _mask(support)


def _spectra(c, seed):
    """Crop spectra of evenly lit fields with smooth aberrations and noise (n x F x F complex64)."""
    g = _keys(c)
    F, n = c["F"], c["n"]
    tilts = _tilts(n, g["nxmax"])
    ratio, support = _ratio_fields(c, seed, tilts)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    v = torch.linspace(-1, 1, F, device="cuda")
    k = torch.randn((n, 6, 1, 1), generator=gen, device="cuda")
    y, x = v[:, None], v[None, :]
    ph = 0.8 * (k[:, 0] * x + k[:, 1] * y + k[:, 2] * x * y + k[:, 3] * x * x + k[:, 4] * y * y)
    amp = 700.0 * (1 + 0.05 * (x * x - y * y) + 0.02 * k[:, 5] * x)
    u = ratio * torch.polar(amp, ph)
    u += 2.0 * torch.randn(u.shape, generator=gen, device="cuda", dtype=torch.complex64)
    spec = torch.fft.fft2(torch.fft.ifftshift(u, dim=(-2, -1))) / (F * F)
    for a, (tx, ty) in enumerate(tilts):  # the specular peak at the crop position of the tilt
        spec[a] = torch.roll(spec[a], (F // 2 + int(ty), F // 2 + int(tx)), dims=(0, 1))
    return spec.contiguous(), _mask(support)


def _positions(c):
    t = _tilts(c["n"], c["F"] // 2) + c["F"] // 2
    return torch.as_tensor(np.concatenate([t[:, 0], t[:, 1]]).astype(np.int32), device="cuda")


def _fields(c, seed):
    """Born or Rytov fields at the tilts' positions, with a little noise (n x F x F complex64)."""
    F, n = c["F"], c["n"]
    ratio, _ = _ratio_fields(c, seed, _tilts(n, F // 2))
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    noise = 0.003 * torch.randn(ratio.shape, generator=gen, device="cuda", dtype=torch.complex64)
    if c["born"]:
        return ratio - 1 + noise
    # log of the ratio with the phase unwrapped: the bodies' phase never wraps along a row here
    ph = torch.angle(ratio)
    for d in (1, 2):
        first = ph.narrow(d, 0, 1)
        step = torch.diff(ph, dim=d)
        step -= 2 * math.pi * torch.round(step / (2 * math.pi))
        ph = torch.cat([first, first + torch.cumsum(step, d)], d)
    return torch.complex(torch.log(ratio.abs()), ph) + noise


def _volume(c, seed):
    D = c["D"]
    v = torch.linspace(-0.5, 0.5, D, device="cuda")
    z, y, x = v[:, None, None], v[None, :, None], v[None, None, :]
    idx = torch.zeros((D, D, D), device="cuda")
    ab = torch.zeros((D, D, D), device="cuda")
    for ctr, ax, dn, kappa in _bodies(seed, 1):
        w = torch.exp(-2 * (((x - ctr[0]) / ax[0]) ** 2 + ((y - ctr[1]) / ax[1]) ** 2 + ((z - ctr[2]) / ax[2]) ** 2))
        idx += dn * w
        ab += kappa * w
    return idx, ab


def _caps(c, seed):
    """Cap values (n x F x F complex64) of a known volume, with noise on the cells."""
    cells, n = _Cells(c), c["n"]
    idx, ab = _volume(c, seed)
    V = cells.spectrum(torch.complex(idx.to(F64), ab.to(F64))).reshape(-1)
    pos = _positions(c).reshape(2, n).T.to(torch.int64)
    out = torch.zeros((n, c["F"], c["F"]), dtype=torch.complex64, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    noise = 1e-5 * float(V.abs().max())
    for a in range(0, n, 64):
        cell = cells(pos[a:a + 64])[0]
        v = V[cell.clamp(min=0)].to(torch.complex64)
        v += noise * torch.randn(v.shape, generator=gen, device="cuda", dtype=torch.complex64)
        out[a:a + 64] = torch.where(cell >= 0, v, 0)
    return out


def prepare(case, seed):
    kind, n, F, D = case["kind"], case["n"], case["F"], case["D"]
    ctx = Context(Geometry(**_keys(case)), n)
    st = {"kind": kind, "ctx": ctx, "n": n}

    def vol(host=False, dtype=torch.float32):
        return torch.zeros((D, D, D), dtype=dtype, pin_memory=True) if host else \
            torch.zeros((D, D, D), dtype=dtype, device="cuda")

    if kind in ("extract", "pipeline"):
        holos, mask = _holograms(case, seed)
        ctx.set_mask(mask)
        host = bool(case.get("host"))
        st["holos"] = holos.cpu().pin_memory() if host else holos
        if kind == "extract":
            st["spectra"] = torch.zeros((n, F, F), dtype=torch.complex64, device="cuda")
        else:
            st["index"], st["absorption"] = vol(host), vol(host)
    elif kind == "fields":
        st["spectra"], mask = _spectra(case, seed)
        ctx.set_mask(mask)
        st["fields"] = torch.zeros((n, F, F), dtype=torch.complex64, device="cuda")
        st["pos"] = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    elif kind == "reconstruct":
        st["fields"], st["pos"] = _fields(case, seed), _positions(case)
        st["index"], st["absorption"] = vol(), vol()
        st["otf"], st["counts"] = vol(dtype=torch.uint8), vol(dtype=torch.int32)
    elif kind == "operators":
        st["index"], st["absorption"] = _volume(case, seed)
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        st["caps_in"] = torch.randn((n, F, F), generator=gen, device="cuda", dtype=torch.complex64)
        st["pos"] = _positions(case)
        st["caps"] = torch.zeros((n, F, F), dtype=torch.complex64, device="cuda")
        st["grad_index"], st["grad_absorption"] = vol(), vol()
    else:  # tv: cap values of a known volume, with noise
        st["pos"], st["caps"] = _positions(case), _caps(case, seed)
        st["index"], st["absorption"] = vol(), vol()
        st["iterations"] = case["iterations"]
    return st


def run(st):
    ctx, kind, n = st["ctx"], st["kind"], st["n"]
    if kind == "extract":
        ctx.extract(st["holos"], spectra_out=st["spectra"])
        return {"spectra": st["spectra"]}
    if kind == "fields":
        ctx.fields(st["spectra"], fields_out=st["fields"], posspec_out=st["pos"])
        return {"fields": st["fields"], "pos": st["pos"]}
    if kind == "reconstruct":
        ctx.reconstruct(st["fields"], st["pos"], indice=st["index"], absorption=st["absorption"], otf=st["otf"],
                        counts=st["counts"])
        return {k: st[k] for k in ("index", "absorption", "otf", "counts")}
    if kind == "pipeline":
        ctx.pipeline(st["holos"], indice=st["index"], absorption=st["absorption"])
        return {k: st[k] for k in ("index", "absorption")}
    if kind == "operators":
        ctx.forward(st["index"], st["absorption"], n=n, posspec=st["pos"], caps_out=st["caps"])
        ctx.adjoint(st["caps_in"], n=n, posspec=st["pos"], index_out=st["grad_index"],
                    absorption_out=st["grad_absorption"])
        return {k: st[k] for k in ("caps", "grad_index", "grad_absorption")}
    rep = ctx.tv_reconstruct(st["index"], st["absorption"], caps=st["caps"], n=n, posspec=st["pos"],
                             iterations=st["iterations"], init=1, tv_eps=2e-3, index_max=0.1, absorption_max=0.02)
    return {"index": st["index"], "absorption": st["absorption"], "misfit_first": rep["misfit_first"],
            "misfit_last": rep["misfit_last"]}


def work(case):
    n, H, F, D, kind = case["n"], case["H"], case["F"], case["D"], case["kind"]
    lg = math.log2
    holo_in = n * H * H * (case["bits"] // 8)
    # a real H x H transform pruned to the crop: H real rows, then F complex columns
    extract = n * (2.5 * H * H * lg(H) + 5 * F * H * lg(H))
    # field (2 x F transforms), Volkov (3.5 x F more with the mirror's symmetries used)
    fields = n * 5 * F * F * lg(F) * (2 + (3.5 if case["volkov"] else 0))
    caps = n * 5 * F * F * lg(F) * 2
    fft3 = 5 * D ** 3 * 3 * lg(D)
    if kind == "extract":
        return {"bytes": holo_in + n * F * F * 8, "flops": extract}
    if kind == "fields":
        return {"bytes": 2 * n * F * F * 8, "flops": fields}
    if kind == "reconstruct":
        return {"bytes": n * F * F * 8 + D ** 3 * 13, "flops": caps + fft3}
    if kind == "pipeline":
        return {"bytes": holo_in + D ** 3 * 8, "flops": extract + fields + caps + fft3}
    if kind == "operators":
        return {"bytes": 2 * (n * F * F * 8 + D ** 3 * 8), "flops": 2 * fft3}
    it = case["iterations"]
    return {"bytes": n * F * F * 8 + D ** 3 * 8 + it * D ** 3 * 16, "flops": (2 * it + 1) * fft3}


# ---------------------------------------------------------------- the same in 64 bits
F64, C128 = torch.float64, torch.complex128


def _tukey(n, alpha):
    """The window's 1D factor as the method defines it: single-precision arguments, 3.1415."""
    f = np.float32
    al = f(alpha)
    b1 = int(math.floor(float(al * f(n - 1) / f(2)) + 0.5))
    b2 = int(math.floor(float(f(n - 1) * (f(1) - al / f(2))) + 0.5))
    t = np.ones(n)
    for i in range(n):
        if i <= b1:
            t[i] = 0.5 * (1 + math.cos(3.1415 * float(f(2 * i) / (al * f(n - 1)) - f(1))))
        elif i > b2:
            t[i] = 0.5 * (1 + math.cos(3.1415 * float(f(2 * i) / (al * f(n - 1)) - f(2) / al + f(1))))
    return torch.as_tensor(t, device="cuda", dtype=F64)


def _sign(n):
    s = torch.ones(n, device="cuda", dtype=F64)
    s[1::2] = -1
    return s


def _x_extract(c, holos):
    g = _keys(c)
    H, N, F = c["H"], g["nxmax"], c["F"]
    w = _tukey(H, 0.05) * _sign(H)
    h = holos.to(torch.int32).to(F64) * w[:, None] * w[None, :]
    y0, x0 = g["circle_cy"] - N, g["circle_cx"] - N
    z = torch.fft.fft2(h)[:, y0:y0 + F, x0:x0 + F] / (H * H)
    ky, kx = torch.arange(y0, y0 + F, device="cuda"), torch.arange(x0, x0 + F, device="cuda")
    return z * (1.0 - 2.0 * ((ky[:, None] + kx[None, :]) % 2))


def _x_unwrap(ph):
    F = ph.shape[-1]
    m = torch.cat([torch.arange(F - 1, -1, -1, device="cuda"), torch.arange(F, device="cuda")])
    s = ph[:, m][:, :, m]
    k = torch.fft.fftfreq(2 * F, device="cuda", dtype=F64)
    kx, ky = k[None, None, :], k[None, :, None]
    z = torch.polar(torch.ones_like(s), s)
    zf, sf = torch.fft.fft2(z), torch.fft.fft2(s.to(C128))
    gx = ((-1j * torch.fft.ifft2(2j * math.pi * kx * zf) / z).real - torch.fft.ifft2(2j * math.pi * kx * sf).real)
    gy = ((-1j * torch.fft.ifft2(2j * math.pi * ky * zf) / z).real - torch.fft.ifft2(2j * math.pi * ky * sf).real)
    k2 = kx * kx + ky * ky
    k2[:, 0, 0] = 1
    p = -1j * (kx * torch.fft.fft2(gx.to(C128)) + ky * torch.fft.fft2(gy.to(C128))) / (2 * math.pi * k2)
    p[:, 0, 0] = 0
    return ph + torch.fft.ifft2(p).real[:, F:, F:]


def _x_fields(c, spec, mask):
    """Fields and specular positions (x, y) of crop spectra."""
    F, n = c["F"], len(spec)
    bi = spec.abs().reshape(n, -1).argmax(1)
    px, py = bi % F, bi // F
    ar = torch.arange(F, device="cuda")
    yy, xx = (ar[None] + py[:, None]) % F, (ar[None] + px[:, None]) % F
    r = spec[torch.arange(n, device="cuda")[:, None, None], yy[:, :, None], xx[:, None, :]]
    u = torch.fft.fftshift(torch.fft.ifft2(r) * (F * F), dim=(-2, -1))
    unw, amp = _x_unwrap(torch.angle(u)), u.abs()
    v = (ar.to(F64) - 0.5 * (F - 1)) / (0.5 * (F - 1))
    X, Y = v[None, :].expand(F, F), v[:, None].expand(F, F)
    basis = torch.stack([X ** a * Y ** b for a in range(5) for b in range(5 - a)], -1)
    on = torch.zeros((F, F), dtype=torch.bool, device="cuda")
    on[::5, ::5] = torch.as_tensor(mask, device="cuda")[::5, ::5] > 45
    q, rr = torch.linalg.qr(basis[on])

    def fit(img):
        return (basis @ torch.linalg.solve_triangular(rr, q.T @ img[:, on].T, upper=True)).permute(2, 0, 1)

    ph = unw - fit(unw)
    af = amp / (fit(amp) + 1e-8)
    af = torch.where(af.abs() > 10, torch.ones_like(af), af).abs()
    f = torch.polar(af, ph) - 1 if c["born"] else torch.complex(torch.log(af), ph)
    return f, torch.stack([px, py], 1)


class _Cells:
    """Ewald-cap cells: for angles at positions (x, y), each bin's volume cell (flat index) or -1."""

    def __init__(self, c):
        self.c, g = c, _keys(c)
        self.N, self.F, self.D, self.r = g["nxmax"], c["F"], c["D"], _rayon(g)
        kv = np.float32(2 * 3.14159 / g["lambda0"])
        k0 = float(np.float32(kv * np.float32(g["n0"])))
        self.cap_scale = (k0 / 3.14159) * (-2 * 3.14159)
        pix = g["tpcam"] / ((g["f_tube"] / g["f_obj"]) / g["rf"])
        self.dx = pix * g["ccd_roix"] / (2 * g["nxmax"])
        df = 1 / (self.dx * 2 * g["nxmax"])
        kk = 2 * math.pi / g["lambda0"]
        self.out_scale = df ** 3 * (-1 / (2 * g["n0"] * kk * kk))

    def __call__(self, pos):
        """(cell index or -1, weight of the bin's spectrum value) for pos (m x 2)."""
        N, F, D, r = self.N, self.F, self.D, self.r
        k = torch.arange(F, device="cuda")
        fx, fy = (k[None] + pos[:, 0:1]) % F - N, (k[None] + pos[:, 1:2]) % F - N
        fd2 = (fx * fx)[:, None, :] + (fy * fy)[:, :, None]
        h = torch.sqrt(torch.clamp(r * r - fd2.to(F64), min=0.0))
        c0 = (r * r - ((pos - N) ** 2).sum(1)).to(F64)
        fz = torch.sqrt(torch.clamp(c0, min=0.0))[:, None, None]
        on = (fd2 < N * N) & (c0 >= 0)[:, None, None]
        z = torch.floor(h - fz + 0.5).to(torch.int64) + D // 2
        X, Y = D // 2 + fx + N - pos[:, 0:1], D // 2 + fy + N - pos[:, 1:2]
        idx = (z * D + Y[:, :, None]) * D + X[:, None, :]
        sg = 1.0 - 2.0 * ((k[:, None] + k[None, :]) % 2)
        return torch.where(on, idx, -1), self.cap_scale * (h / r) * self.dx ** 2 * sg

    def parity(self):
        p = torch.arange(self.D, device="cuda") % 2
        return 1.0 - 2.0 * ((p[:, None, None] + p[None, :, None] + p[None, None, :]) % 2)

    def to_volume(self, V, scale):
        """scale (-1)^m IFFT3((-1)^k V), unnormalised, in place."""
        s = self.parity()
        V *= s
        V = torch.fft.ifftn(V)
        V *= s * (scale * float(self.D) ** 3)
        return V

    def spectrum(self, x):
        s = self.parity()
        return s * torch.fft.fftn(s * x) / (self.out_scale * float(self.D) ** 3)


def _x_reconstruct(cells, fields, pos, step=32):
    """Volume (complex), OTF, counts from FP64 fields; fields(a, b) gives those of angles [a, b)."""
    D = cells.D
    V = torch.zeros(D ** 3, dtype=C128, device="cuda")
    cnt = torch.zeros(D ** 3, dtype=torch.int32, device="cuda")
    w = _tukey(cells.F, 0.1)
    for a in range(0, cells.c["n"], step):
        f, p = fields(a, min(a + step, cells.c["n"])), pos(a, min(a + step, cells.c["n"]))
        idx, wt = cells(p)
        v = 1j * wt * torch.fft.fft2(f * w[:, None] * w[None, :])
        on = idx >= 0
        torch.view_as_real(V).index_add_(0, idx[on], torch.view_as_real(v[on]))
        cnt.index_add_(0, idx[on], torch.ones((), dtype=torch.int32, device="cuda").expand(int(on.sum())))
    V /= torch.clamp(cnt, min=1)
    otf = (V.real.to(torch.float32) != 0).to(torch.uint8).reshape(D, D, D)
    return cells.to_volume(V.reshape(D, D, D), cells.out_scale), otf, cnt.reshape(D, D, D)


def _tv_grad(x, eps):
    def diff(d):
        return torch.nn.functional.pad(torch.diff(x, dim=d), [0, 1 if d == 2 else 0, 0, 1 if d == 1 else 0, 0,
                                                              1 if d == 0 else 0])
    g = [diff(d) for d in range(3)]
    inv = 1 / torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2 + eps ** 2)
    out = -(g[0] + g[1] + g[2]) * inv
    for d in range(3):
        out.narrow(d, 1, x.shape[d] - 1).add_((g[d] * inv).narrow(d, 0, x.shape[d] - 1))
    return out


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if not case["volkov"]:
        return None  # the group merging's decisions are those of the single-precision wrapped phase
    if kind == "extract":
        holos, _ = _holograms(case, seed)
        return {"spectra": torch.cat([_x_extract(case, holos[a:a + 16]) for a in range(0, n, 16)])}
    if kind == "fields":
        spec, mask = _spectra(case, seed)
        f = torch.cat([_x_fields(case, spec[a:a + 16].to(C128), mask)[0] for a in range(0, n, 16)])
        return {"fields": f, "pos": None}
    cells = _Cells(case)
    if kind == "reconstruct":
        f = _fields(case, seed)
        p = _positions(case).reshape(2, n).T.to(torch.int64)
        v, _, _ = _x_reconstruct(cells, lambda a, b: f[a:b].to(C128), lambda a, b: p[a:b])
        return {"index": v.real, "absorption": v.imag, "otf": None, "counts": None}
    if kind == "pipeline":
        holos, mask = _holograms(case, seed)
        step, fs, ps = 16, [], []
        for a in range(0, n, step):
            f, p = _x_fields(case, _x_extract(case, holos[a:a + step]), mask)
            fs.append(f)
            ps.append(p)
        f, p = torch.cat(fs), torch.cat(ps)
        del holos, fs
        v, _, _ = _x_reconstruct(cells, lambda a, b: f[a:b], lambda a, b: p[a:b], 16)
        return {"index": v.real, "absorption": v.imag}
    pos = _positions(case).reshape(2, n).T.to(torch.int64)
    idx = torch.cat([cells(pos[a:a + 64])[0] for a in range(0, n, 64)])
    on = idx >= 0

    def scatter(v):
        V = torch.zeros((case["D"] ** 3, 2), dtype=F64, device="cuda")
        V.index_add_(0, idx[on], torch.view_as_real(v[on].contiguous()))
        return torch.view_as_complex(V)

    def sample(x):
        return torch.where(on, cells.spectrum(x).reshape(-1)[idx.clamp(min=0)], 0)

    shape = (case["D"],) * 3
    if kind == "operators":
        i, ab = _volume(case, seed)
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        caps_in = torch.randn(idx.shape, generator=gen, device="cuda", dtype=torch.complex64).to(C128)
        g = cells.to_volume(scatter(caps_in).reshape(shape), 1 / (cells.out_scale * float(case["D"]) ** 3))
        return {"caps": sample(torch.complex(i.to(F64), ab.to(F64))), "grad_index": g.real, "grad_absorption": g.imag}
    data = _caps(case, seed).to(C128)
    cnt = torch.zeros(case["D"] ** 3, dtype=F64, device="cuda")
    cnt.index_add_(0, idx[on], torch.ones(int(on.sum()), dtype=F64, device="cuda"))
    cnt = cnt.clamp(min=1)
    x = cells.to_volume((scatter(data) / cnt).reshape(shape), cells.out_scale)
    first = last = 0.0
    for it in range(case["iterations"]):
        r = torch.where(on, sample(x) - data, 0)
        last = float((r.real ** 2 + r.imag ** 2).sum())
        first = last if it == 0 else first
        g = cells.to_volume((scatter(r) / cnt).reshape(shape), cells.out_scale)
        re = x.real - g.real - 1e-3 * 0.1 * _tv_grad(x.real.contiguous(), 2e-3)
        im = x.imag - g.imag - 1e-3 * 0.02 * _tv_grad(x.imag.contiguous(), 2e-3)
        x = torch.complex(re.clamp(0, 0.1), im.clamp(0, 0.02))
    return {"index": x.real, "absorption": x.imag, "misfit_first": first, "misfit_last": last}
