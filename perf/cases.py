"""Workloads that stand for the use of this framework, for timing and comparing it.

A case is a dict of plain values.  ``prepare(case, seed)`` makes the inputs on
the GPU (host arrays for the engine class), ``run(state)`` makes one pass
through the public entry points, ``work(case)`` counts what the path cannot do
without, and ``exact(case, seed)`` computes the outputs of ``run`` in 64 bits
with plain torch.

Scans are circular: seeded ellipsoids seen as line integrals (with detector
noise) or as Poisson counts, sizes from the repository's configurations and
benchmark or generic ones.
"""
import math

import numpy as np
import torch

from tomokvas_gb300 import _lib, device
from tomokvas_gb300.batch import Batch
from tomokvas_gb300.fbp import FilteredBackProjection, VolumeSink
from tomokvas_gb300.geometry import FDKGeometry

I0 = 50000.0
TAU = 0.02  # cm; the virtual pixel pitch (it scales the filter, nothing else)


def listed():
    return [
        # the smallest call: a preview volume while a scan is being set up (latency and launches count)
        {"name": "fdk_preview_f32", "kind": "fdk", "W": 64, "N": 96, "H": 64, "X": 64, "Y": 64, "Z": 48, "D": 312.5,
         "scale": 1.25, "shift": 0.0, "flips": 0, "precision": "f32", "input": "f32", "layout": "sinogram",
         "window": "ramlak", "maps": False},
        # an ordinary reconstruction with every default: FP32 storage, the reference's sinogram order and filter
        {"name": "fdk_256_f32", "kind": "fdk", "W": 256, "N": 180, "H": 256, "X": 256, "Y": 256, "Z": 256,
         "D": 2500.0, "scale": 1.0, "shift": 0.0, "flips": 0, "precision": "f32", "input": "f32",
         "layout": "sinogram", "window": "ramlak", "maps": False},
        # the largest: a full-resolution scan from raw detector frames, FP16 storage
        {"name": "fdk_1024_f16_u16", "kind": "fdk", "W": 1024, "N": 720, "H": 1024, "X": 1024, "Y": 1024, "Z": 1024,
         "D": 6000.0, "scale": 1.0, "shift": 0.0, "flips": 0, "precision": "f16", "input": "u16",
         "layout": "projection", "window": "ramlak", "maps": False},
        # a region of interest off the axis with ragged sizes, flips, dark and flat maps, BF16 storage
        {"name": "fdk_region_bf16_u16", "kind": "fdk", "W": 500, "N": 301, "H": 389, "X": 333, "Y": 290, "Z": 201,
         "D": 1700.0, "scale": 1.1, "shift": 7.3, "flips": 5, "precision": "bf16", "input": "u16",
         "layout": "projection", "window": "hann", "maps": True},
        # the filter alone on frames as they arrive during a scan
        {"name": "filter_frames_f16_u16", "kind": "filter", "W": 1024, "N": 90, "H": 1024, "D": 6000.0,
         "precision": "f16", "input": "u16", "layout": "projection", "window": "shepp_logan"},
        # the filter alone on a wide odd-sized FP32 sinogram
        {"name": "filter_rows_f32", "kind": "filter", "W": 1501, "N": 300, "H": 411, "D": 4100.0,
         "precision": "f32", "input": "f32", "layout": "sinogram", "window": "hann"},
        # one Z slab of a larger volume, added to what is there: FP32 coefficient images
        {"name": "slab_f32c", "kind": "slab", "W": 768, "N": 240, "H": 512, "X": 640, "Y": 640, "nz": 48, "z0": -30.0,
         "D": 3900.0, "scale": 1.1, "shift": 0.0, "precision": "f32c"},
        # the gradient of a volume loss with respect to the projections (training, data consistency)
        {"name": "backward_512", "kind": "backward", "W": 768, "N": 360, "H": 768, "X": 512, "Y": 512, "Z": 512,
         "D": 4000.0, "scale": 1.5, "shift": 0.0, "layout": "sinogram", "window": "ramlak"},
        # data-consistency steps on a reconstructed volume, checkpoint in FP16, loss watched
        {"name": "refine_256", "kind": "refine", "W": 320, "N": 240, "H": 272, "X": 256, "Y": 256, "Z": 224,
         "D": 1300.0, "scale": 1.2, "shift": 0.0, "steps": 2, "half": True},
        # a server's batch of small uneven scans, planned once and replayed on new data
        {"name": "batch_uneven_f16", "kind": "batch", "items": 8, "small": 96, "large": 288, "sizes": 11,
         "precision": "f16"},
        # the drop-in engine class, host sinogram to host volume, block by block
        {"name": "engine_256", "kind": "engine", "W": 256, "N": 180, "H": 256, "X": 256, "Z": 256, "D": 2500.0,
         "scale": 1.0, "zb": 32, "precision": "f32"},
        # completion of an offset-detector scan before its reconstruction
        {"name": "complete_half_fan", "kind": "rebin", "op": "full", "W": 520, "N": 720, "rows": 256, "am": 21,
         "D": 2300.0, "flip": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cap(c):
    """Drawn sizes stay below the largest listed case's work (a third of it)."""
    while work(c)["flops"] > 0.3 * 1.1e13:
        for k in ("N", "Z", "X", "Y"):
            if k in c:
                c[k] = max(16, int(c[k] * 0.8))
    return c


def draw(rng):
    kind = rng.choice(["fdk"] * 4 + ["filter"] * 2 + ["slab", "backward", "refine", "batch", "engine", "rebin"])
    window = rng.choice(["ramlak", "shepp_logan", "hann"])
    layout = rng.choice(["sinogram", "projection"])
    if kind == "fdk":
        n = _log(rng, 48, 640)
        square = rng.random() < 0.5  # a centred square volume over a full turn of 4k angles, or any other
        W = max(16, int(n * rng.uniform(0.8, 1.5)))
        scale = round(rng.uniform(0.6, 1.0) * min(1.5, 1.2 * W / n), 3)
        N = _log(rng, 60, 900)
        if square:
            n, N = max(32, n // 32 * 32), N // 4 * 4
        inp = rng.choice(["f32", "u16"])
        return _cap({"kind": "fdk", "W": W, "N": N, "H": max(16, int(W * rng.uniform(0.6, 1.1))), "X": n,
                     "Y": n if square else max(16, int(n * rng.uniform(0.7, 1.2))),
                     "Z": max(8, int(n * rng.uniform(0.4, 1.1))), "D": round(W * rng.uniform(3.0, 10.0), 2),
                     "scale": scale, "shift": 0.0 if square else round(rng.uniform(-0.1, 0.1) * n, 2),
                     "flips": 0 if square else rng.randrange(8),
                     "precision": rng.choice(["f32", "f16", "f16", "bf16", "f32c"]), "input": inp, "layout": layout,
                     "window": window, "maps": inp == "u16" and rng.random() < 0.5})
    if kind == "filter":
        W = _log(rng, 60, 2048)
        return {"kind": "filter", "W": W, "N": _log(rng, 16, 400), "H": max(16, min(900, int(W * rng.uniform(0.3, 1.0)))),
                "D": round(W * rng.uniform(3.0, 10.0), 2), "precision": rng.choice(["f32", "f16", "bf16", "f32c"]),
                "input": rng.choice(["f32", "u16"]), "layout": layout, "window": window}
    if kind == "slab":
        n = _log(rng, 64, 800)
        W = max(32, int(n * rng.uniform(0.9, 1.4)))
        return _cap({"kind": "slab", "W": W, "N": _log(rng, 60, 600), "H": max(32, int(W * rng.uniform(0.5, 1.0))),
                     "X": n, "Y": max(32, int(n * rng.uniform(0.8, 1.0))), "nz": rng.randrange(5, 97),
                     "z0": round(rng.uniform(-0.4, 0.1) * n, 1), "D": round(W * rng.uniform(3.0, 10.0), 2),
                     "scale": round(rng.uniform(0.7, 1.2), 3), "shift": round(rng.uniform(-0.05, 0.05) * n, 2),
                     "precision": rng.choice(["f32", "f16", "bf16", "f32c"])})
    if kind == "backward":
        n = _log(rng, 40, 480)
        W = max(24, int(n * rng.uniform(0.9, 1.5)))
        return _cap({"kind": "backward", "W": W, "N": _log(rng, 45, 400), "H": max(24, int(W * rng.uniform(0.6, 1.0))),
                     "X": n, "Y": max(24, int(n * rng.uniform(0.8, 1.0))), "Z": max(8, int(n * rng.uniform(0.3, 1.0))),
                     "D": round(W * rng.uniform(3.0, 10.0), 2), "scale": round(rng.uniform(0.6, 1.0) * W / n, 3),
                     "shift": round(rng.uniform(-0.05, 0.05) * n, 2), "layout": layout, "window": window})
    if kind == "refine":
        n = _log(rng, 48, 300)
        W = max(32, int(n * rng.uniform(0.9, 1.5)) // 8 * 8)
        return _cap({"kind": "refine", "W": W, "N": _log(rng, 60, 300), "H": max(24, int(W * rng.uniform(0.6, 1.0))),
                     "X": n, "Y": n, "Z": max(8, int(n * rng.uniform(0.4, 1.0))),
                     "D": round(W * rng.uniform(3.0, 10.0), 2), "scale": round(rng.uniform(0.6, 1.0) * W / n, 3),
                     "shift": round(rng.uniform(-0.05, 0.05) * n, 2), "steps": rng.choice([1, 2, 3]),
                     "half": rng.random() < 0.5})
    if kind == "batch":
        small = _log(rng, 40, 160)
        return {"kind": "batch", "items": rng.randrange(3, 13), "small": small,
                "large": min(320, int(small * rng.uniform(1.2, 3.0))), "sizes": rng.randrange(1 << 20),
                "precision": rng.choice(["f16", "f16", "bf16", "f32c"])}
    if kind == "engine":
        n, zb = _log(rng, 64, 384), rng.choice([8, 16, 32])
        W = max(32, int(n * rng.uniform(0.9, 1.4)))
        return {"kind": "engine", "W": W, "N": _log(rng, 60, 300), "H": max(32, int(W * rng.uniform(0.7, 1.0))),
                "X": n, "Z": max(1, int(n * rng.uniform(0.4, 1.0)) // zb) * zb, "D": round(W * rng.uniform(3.0, 10.0), 2),
                "scale": round(rng.uniform(0.7, 1.0) * W / n, 3), "zb": zb, "precision": rng.choice(["f32", "f16"])}
    W = _log(rng, 60, 1000)
    return {"kind": "rebin", "op": rng.choice(["full", "parallel"]), "W": W, "N": 2 * _log(rng, 45, 700),
            "rows": _log(rng, 8, 400), "am": rng.randrange(0, max(1, W // 6)), "D": round(W * rng.uniform(2.0, 8.0), 2),
            "flip": rng.random() < 0.3}


# ------------------------------------------------------------------ geometry
def _geometry(c):
    W, N, H = c["W"], c["N"], c["H"]
    X, Y, Z = c.get("X", 8), c.get("Y", c.get("X", 8)), c.get("Z", c.get("nz", 8))
    shift, flips = c.get("shift", 0.0), c.get("flips", 0)
    # the detector of an off-centre scan is itself a little off centre
    return FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2.0 + 0.25 * shift, cZ=(H - 1) / 2.0 - 0.1 * shift,
                       dfi=float(np.float32(2.0 * math.pi / N)), D=c["D"], tau=TAU, X=X, Y=Y, Z=Z,
                       cx=(X - 1) / 2.0 + shift, cy=(Y - 1) / 2.0 - 0.5 * shift, cz=0.0,
                       rot=0.02 * shift, scale=c.get("scale", 1.0), dirx=flips & 1, diry=flips >> 1 & 1,
                       dirz=flips >> 2 & 1)


def _batch_cases(c):
    """The uneven items of a batch: cubes or near-cubes, full turns, half of them with whole quarter turns."""
    r = np.random.default_rng(c["sizes"])
    out = []
    for _ in range(c["items"]):
        n = int(round(math.exp(r.uniform(math.log(c["small"]), math.log(c["large"])))))
        W = int(n * r.uniform(0.9, 1.5)) // 8 * 8
        out.append({"W": W, "N": int(r.integers(90, 301)), "H": W, "X": n, "Y": n, "Z": n,
                    "D": round(W * float(r.uniform(4.0, 8.0)), 2), "scale": round(min(0.9 * W / n, 1.5), 3)})
    return out


def _zoffsets(g, zb):
    """(number of blocks, first-slice offset of each) of the engine's Z blocks."""
    nr = float(np.float32(g.Z - 1) / np.float32(zb))
    n = math.ceil(nr)
    dcor = float(np.float32((n - nr) * zb / 2))
    return [(k - n / 2.0) * zb + dcor - g.cz for k in range(n)]


# -------------------------------------------------------------------- inputs
def _angles(g):
    b = np.arange(g.N, dtype=np.float32) * np.float32(g.dfi) + np.float32(g.rot)
    return np.cos(b.astype(np.float64)), np.sin(b.astype(np.float64))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _line_integrals(g, seed):
    """[N][H][W] float32 line integrals (cm) of seeded ellipsoids around the axis, in virtual-pixel coordinates."""
    r = np.random.default_rng(int(seed))
    R = 0.46 * g.W
    half = 0.46 * g.H
    ell = [((0.0, 0.0, 0.0), (0.9 * R, 0.8 * R, 0.85 * half), 0.0, 0.9),
           ((0.0, 0.0, 0.0), (0.82 * R, 0.72 * R, 0.8 * half), 0.0, -0.5)]
    for _ in range(6):
        t, q = r.uniform(0, 2 * np.pi), 0.55 * R * math.sqrt(r.uniform())
        ell.append(((q * math.cos(t), q * math.sin(t), float(r.uniform(-0.4, 0.4)) * half),
                    tuple(r.uniform(0.05, 0.25, 3) * (R, R, half)), float(r.uniform(0, np.pi)), float(r.uniform(-0.3, 0.8))))
    per_px = 4.0 / (2 * R)  # at most a few optical depths through the body
    cs, sn = (torch.from_numpy(a).cuda().float() for a in _angles(g))
    T = (torch.arange(g.W, device="cuda", dtype=torch.float32) - g.cX)[None, None, :]
    Zd = (torch.arange(g.H, device="cuda", dtype=torch.float32) - g.cZ)[None, :, None]
    out = torch.empty((g.N, g.H, g.W), device="cuda")
    step = max(1, (1 << 26) // (g.H * g.W))
    for b in range(0, g.N, step):
        c, s = cs[b:b + step, None, None], sn[b:b + step, None, None]
        o = out[b:b + step]
        o.zero_()
        length = torch.sqrt(g.D ** 2 + T * T + Zd * Zd)
        for (x, y, z), (ax, ay, az), phi, rho in ell:
            cp, sp = math.cos(phi), math.sin(phi)
            # the ray from (D c, D s, 0) to (-T s, T c, Z), in the ellipsoid's unit-sphere coordinates
            ox, oy, oz = ((g.D * c - x) * cp + (g.D * s - y) * sp) / ax, ((g.D * s - y) * cp - (g.D * c - x) * sp) / ay, -z / az
            dx = ((-T * s - g.D * c) * cp + (T * c - g.D * s) * sp) / ax
            dy = ((T * c - g.D * s) * cp - (-T * s - g.D * c) * sp) / ay
            dz = Zd / az
            A = dx * dx + dy * dy + dz * dz
            B = ox * dx + oy * dy + oz * dz
            disc = B * B - A * (ox * ox + oy * oy + oz * oz - 1.0)
            o.add_(disc.clamp_(min=0.0).sqrt_().mul_(2.0 * rho * per_px).div_(A).mul_(length))
    return out


def _scan(c, g, seed):
    """The projections as the case's input type has them, their flat-field parameters, in the case's layout."""
    p = _line_integrals(g, seed)
    gen = _gen(seed)
    ff = None
    if c["input"] == "u16":
        if c.get("maps"):
            flat = I0 * (0.9 + 0.1 * torch.rand((g.H, g.W), device="cuda", generator=gen))
            dark = 90.0 + 20.0 * torch.rand((g.H, g.W), device="cuda", generator=gen)
        else:
            flat, dark = None, None
        fl, dk = (I0, 100.0) if flat is None else (flat, dark)
        counts = p.neg_().exp_().mul_(fl)
        for b in range(0, g.N, 64):
            counts[b:b + 64] = torch.poisson(counts[b:b + 64], generator=gen)
        x = counts.add_(dk).round_().clamp_(0, 65535).to(torch.int32).to(torch.int16)  # the bits of a uint16
        ff = (device.flatfield(flat_value=I0 + 100.0, dark_value=100.0) if flat is None
              else device.flatfield(flat=flat + dark, dark=dark))
    else:
        for b in range(0, g.N, 64):
            p[b:b + 64] += 0.01 * torch.randn(p[b:b + 64].shape, device="cuda", generator=gen)
        x = p
    if c["layout"] == "sinogram":
        x = x.transpose(0, 1).contiguous()
    return x, ff


def _spectrum(g, window):
    """tau |FFT(h)| of the reference's taps with the window's gain, 64 bits, and the pad length."""
    p = 2
    while p < g.W:
        p *= 2
    p *= 2
    i = np.arange(g.W) - g.W // 2
    tau = float(np.float32(g.tau))
    h = np.where(i == 0, 1.0 / (4 * tau * tau), 0.0)
    odd = i % 2 != 0
    h[odd] = -1.0 / (i[odd].astype(np.float64) ** 2 * np.pi ** 2 * tau * tau)
    h = h.astype(np.float32) / np.float32(2)
    H = tau * np.abs(np.fft.rfft(h.astype(np.float64), p))
    f = np.arange(p // 2 + 1) / p
    if window == "shepp_logan":
        H = H * np.sinc(f)
    elif window == "hann":
        H = H * 0.5 * (1.0 + np.cos(2.0 * np.pi * f))
    return H, p


def _filtered(g, p, window):
    """[n][H][W] float64 cosine-weighted, ramp-filtered rows of projections p [n][H][W]."""
    H, pad = _spectrum(g, window)
    H = torch.from_numpy(H).cuda()
    x = (torch.arange(g.W, device="cuda", dtype=torch.float64) - g.cX)[None, :]
    z = (torch.arange(g.H, device="cuda", dtype=torch.float64) - g.cZ)[:, None]
    w = g.D / torch.sqrt(g.D ** 2 + x * x + z * z)
    return torch.fft.irfft(torch.fft.rfft(p.double() * w, pad) * H, pad)[..., :g.W] * pad


def _coefficients(q):
    """(Q, dU, dV, dUV) of samples q [n][H][W], zero outside."""
    e = torch.nn.functional.pad(q, (0, 1, 0, 1))
    Q, r, d, rd = e[:, :-1, :-1], e[:, :-1, 1:], e[:, 1:, :-1], e[:, 1:, 1:]
    return Q, r - Q, d - Q, (rd - d) - (r - Q)


def _projections64(c, g, x, ff):
    """Line integrals [N][H][W] in 64 bits from the case's input."""
    x = x.transpose(0, 1) if c["layout"] == "sinogram" else x
    if c["input"] == "f32":
        return x.double()
    fl, dk = ff._keep[0], ff._keep[1]
    dk = 100.0 if dk is None else dk.double()
    fl = I0 + 100.0 if fl is None else fl.double()
    n = torch.bitwise_and(x.to(torch.int32), 0xFFFF).double()
    den = fl - dk
    den = den.clamp(min=0.5) if isinstance(den, torch.Tensor) else max(den, 0.5)
    return -torch.log((n - dk).clamp_(min=0.5) / den)


def _stored(g, q, precision):
    """Filtered projections q (float64) in a storage format, as the stage API hands them on, and their scale."""
    scale = torch.ones(1, device="cuda")
    if precision == "f32":
        out = torch.zeros((g.N, g.H, device.row_pitch(g.W)), device="cuda")
        out[..., :g.W] = q
        return out, scale
    if precision == "f32c":
        return torch.stack(_coefficients(q.float()), -1).contiguous(), scale
    scale.fill_(2.0 ** math.floor(math.log2(16384.0 / (4 * float(q.abs().max()) + 1e-30))))
    Q, dU, dV, dUV = _coefficients(q.float() * scale)
    e = torch.stack((Q, dV, dU, dUV), -1)
    if g.W % 2:
        e = torch.nn.functional.pad(e, (0, 0, 0, 1))
    return e.to(torch.float16 if precision == "f16" else torch.bfloat16).contiguous(), scale


def _slab_q(c, g, seed):
    return _filtered(g, _line_integrals(g, seed), "ramlak")


def _volume(g, seed, scale=1.0):
    """A smooth-plus-noise volume such as a gradient or a reconstruction is."""
    gen = _gen(seed + 17)
    lo = torch.randn((1, 1, 8, 8, 8), device="cuda", generator=gen)
    v = torch.nn.functional.interpolate(lo, size=(g.Z, g.Y, g.X), mode="trilinear", align_corners=True)[0, 0]
    for z in range(0, g.Z, 64):
        v[z:z + 64] += 0.3 * torch.randn(v[z:z + 64].shape, device="cuda", generator=gen)
    return v.mul_(scale).contiguous()


def _refine_alpha(c, g):
    """A step size below 1 / lambda_max(B B^T): one over (row sums) x (column sums) of B, bounded."""
    _, p = _spectrum(g, "ramlak")
    u2 = (g.D / (g.D - 0.5 * g.W)) ** 2
    rows = g.N * (g.dfi / p) * u2
    cols = (g.dfi / p) * u2 * 2.0 * g.W / g.scale ** 3
    return 1.0 / (rows * cols)


def _sinogram_host(g, seed):
    return np.ascontiguousarray(_line_integrals(g, seed).transpose(0, 1).cpu().numpy())


# ----------------------------------------------------------- the public calls
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "rebin":
        s["sino"] = torch.rand((case["rows"], case["N"], case["W"]), device="cuda", generator=_gen(seed))
        return s
    if kind == "batch":
        prec = _lib.PRECISIONS[case["precision"]]
        b, vols = Batch(prec), []
        for k, c in enumerate(_batch_cases(case)):
            g = _geometry(c)
            x = _line_integrals(g, seed * 100 + k).transpose(0, 1).contiguous()
            vols.append(torch.zeros((g.Z, g.Y, g.X), device="cuda"))
            b.submit(g, x, vols[-1])
        b.plan()
        s.update(batch=b, vols=vols)
        return s
    g = _geometry(case)
    s["g"] = g
    if kind == "engine":
        # a program keeps its volume file mapped: the blocks go to pages that are there
        s.update(sino=_sinogram_host(g, seed), out=np.ones((g.Z, g.Y, g.X), np.float32))
        return s
    if kind in ("fdk", "filter"):
        s["prec"] = _lib.PRECISIONS[case["precision"]]
        s["x"], s["ff"] = _scan(case, g, seed)
        s["args"] = (_lib.TK_INPUT_U16 if case["input"] == "u16" else _lib.TK_INPUT_F32, _lib.LAYOUTS[case["layout"]],
                     s["ff"], _lib.WINDOWS[case["window"]], s["prec"])
        if kind == "filter":
            q, scale = device.alloc_filtered(g, s["prec"])
            s["out"] = (q.zero_(), scale)
        else:
            s["ws"] = torch.empty(device.workspace_bytes(g, s["prec"]), dtype=torch.uint8, device="cuda")
            s["vol"] = torch.zeros((g.Z, g.Y, g.X), device="cuda")
    elif kind == "slab":
        s["prec"] = _lib.PRECISIONS[case["precision"]]
        s["q"], s["scale"] = _stored(g, _slab_q(case, g, seed), case["precision"])
        s["x0"] = _volume(g, seed, 0.01)
        s["vol"] = torch.empty_like(s["x0"])
    elif kind == "backward":
        s["grad"] = _volume(g, seed)
        s["ws"] = torch.empty(device.workspace_bytes(g), dtype=torch.uint8, device="cuda")
    else:  # refine: the checkpoint holds FP16 or FP32 samples [N][H][W], W a multiple of the row pitch
        q = _filtered(g, _line_integrals(g, seed), "ramlak")
        s["ckpt"] = (q.half() if case["half"] else q.float()).contiguous()
        s["x0"] = _volume(g, seed, float(q.std()) * 0.1)
        s["vol"] = torch.empty_like(s["x0"])
        s["alpha"] = _refine_alpha(case, g)
        s["loss"] = torch.zeros(case["steps"], dtype=torch.float64, device="cuda")
        s["ws"] = device.refine_workspace(g)
    return s


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "fdk":
        it, layout, ff, window, prec = s["args"]
        return device.fdk_device(s["g"], s["x"], it, layout, ff, window, prec, workspace=s["ws"], vol=s["vol"])
    if kind == "filter":
        it, layout, ff, window, prec = s["args"]
        q, scale = device.filter_projections(s["g"], s["x"], it, layout, ff, window, prec, out=s["out"])
        # the 16-bit images are handed on as the numbers they hold
        return {"q": {"f16": q.view(torch.float16), "bf16": q.view(torch.bfloat16), "f32c": q.view(torch.float32),
                      "f32": q}[c["precision"]] if c["precision"] != "f32" else q, "scale": scale}
    if kind == "slab":
        s["vol"].copy_(s["x0"])  # the partial sums of earlier angles
        return device.backproject(s["g"], s["q"], s["scale"], s["prec"], vol=s["vol"], nz=c["nz"], zoff=c["z0"],
                                  accumulate=True)
    if kind == "backward":
        return device.fdk_backward(s["g"], s["grad"], _lib.WINDOWS[c["window"]], _lib.LAYOUTS[c["layout"]],
                                   workspace=s["ws"])
    if kind == "refine":
        s["vol"].copy_(s["x0"])
        device.refine_volume(s["g"], s["ckpt"], s["vol"], s["alpha"], c["steps"], loss=s["loss"], workspace=s["ws"])
        return {"vol": s["vol"], "loss": s["loss"].float()}  # the loss is a sum of 32-bit terms
    if kind == "batch":
        s["batch"].run(graph=True)
        return s["vols"]
    if kind == "engine":
        g, f = s["g"], FilteredBackProjection(raise_on_error=True)
        f.SetBlockSize(c["zb"])
        f.SetSinogramProperties(s["sino"], g.W, g.cX, g.N, g.H, g.cZ, g.dfi, g.D, g.tau)
        f.SetReconstructionProperties(VolumeSink(g.X, g.Y, g.Z, c["zb"], out=s["out"]), g.X, g.cx, g.Y, g.cy, g.Z, g.cz,
                                      g.rot)
        f.SetScaleXYZ(g.scale)
        f.SetPrecision(c["precision"])
        f.Initialize()
        f.CalculateReconstruction()
        f.close()
        return s["out"]
    dfi = 2.0 * math.pi / c["N"]
    if c["op"] == "full":
        return device.half_to_full_fan(s["sino"], c["am"], c["D"], dfi, c["flip"])
    return device.half_to_parallel(s["sino"], c["am"], c["D"], dfi)


# ---------------------------------------------------------------------- work
def _updates(g, nz):
    """Voxel-projection updates inside the field of view."""
    x = g.scale * (np.arange(g.X) - g.cx)
    y = g.scale * (np.arange(g.Y) - g.cy)
    return int((np.hypot(x[None, :], y[:, None]) < g.W / 2.0).sum()) * nz * g.N


def _filter_flops(g):
    p = 2
    while p < g.W:
        p *= 2
    return g.N * g.H * 5.0 * 2 * p * (math.log2(p) + 1)


def work(case):
    kind = case["kind"]
    if kind == "rebin":
        wc = 2 * case["W"] - 1 - 2 * case["am"]
        n_out = case["N"] if case["op"] == "full" else case["N"] // 2
        return {"bytes": 4.0 * case["rows"] * (case["N"] * case["W"] + n_out * wc), "flops": 3.0 * case["rows"] * n_out * wc}
    if kind == "batch":
        gs = [_geometry(c) for c in _batch_cases(case)]
        return {"bytes": sum(4.0 * (g.N * g.H * g.W + g.X * g.Y * g.Z) for g in gs),
                "flops": sum(14.0 * _updates(g, g.Z) + _filter_flops(g) for g in gs)}
    g = _geometry(case)
    samples, voxels = float(g.N) * g.H * g.W, float(g.X) * g.Y * g.Z
    entry = {"f32": 4, "f16": 8, "bf16": 8, "f32c": 16}[case.get("precision", "f32")]
    raw = 2 if case.get("input") == "u16" else 4
    if kind == "filter":
        return {"bytes": samples * (raw + entry), "flops": _filter_flops(g)}
    up = _updates(g, g.Z)
    if kind == "slab":
        return {"bytes": samples * entry + 8 * voxels, "flops": 14.0 * up}
    if kind == "refine":
        return {"bytes": samples * (2 if case["half"] else 4) * case["steps"] + 8 * voxels,
                "flops": case["steps"] * (28.0 * up + 5 * samples)}
    return {"bytes": samples * raw + 4 * voxels, "flops": 14.0 * up + _filter_flops(g)}


# ------------------------------------------------------------------ 64 bits
def _columns(g):
    """Flat indices of the columns inside the field of view and their coordinates (virtual pixels)."""
    sc = float(np.float32(g.scale))
    fx, fy = (-1.0 if g.dirx else 1.0), (-1.0 if g.diry else 1.0)
    x = fx * sc * (torch.arange(g.X, device="cuda", dtype=torch.float64) - float(np.float32(g.cx)))
    y = fy * sc * (torch.arange(g.Y, device="cuda", dtype=torch.float64) - float(np.float32(g.cy)))
    aY, aX = torch.meshgrid(y, x, indexing="ij")
    idx = (torch.sqrt(aX * aX + aY * aY) < g.W / 2.0).reshape(-1).nonzero()[:, 0]
    return idx, aX.reshape(-1)[idx], aY.reshape(-1)[idx]


def _slices(g, nz, zoff):
    f = -1.0 if g.dirz else 1.0
    return f * float(np.float32(g.scale)) * (torch.arange(nz, device="cuda", dtype=torch.float64) + zoff)


def _walk(g, aX, aY, aZ, c, s):
    """Column and row taps of every voxel at one angle: (c0, fu, inside, U^2), (r0, fv, inside)."""
    D = float(np.float32(g.D))
    U = D / (D - (aX * c + aY * s))
    u = (aY * c - aX * s) * U + float(np.float32(g.cX))
    uin = (u >= 0) & (u <= g.W - 1)
    c0 = u.floor().clamp(0, g.W - 1)
    v = aZ[:, None] * U[None, :] + float(np.float32(g.cZ))
    vin = (v >= 0) & (v <= g.H - 1)
    r0 = v.floor().clamp(0, g.H - 1)
    return (c0.long(), u - c0, uin, U * U), (r0.long(), v.sub_(r0), vin)


def _fscale(g):
    _, p = _spectrum(g, "ramlak")
    return float(np.float32(g.dfi)) / p


def _back64(g, q, nz, zoff):
    """B q: [nz][Y][X] float64 from samples q [N][H][W] float64."""
    idx, aX, aY = _columns(g)
    aZ, (cs, sn) = _slices(g, nz, zoff), _angles(g)
    acc = torch.zeros((nz, idx.numel()), dtype=torch.float64, device="cuda")
    for b in range(g.N):
        (c0, fu, uin, U2), (r0, fv, vin) = _walk(g, aX, aY, aZ, cs[b], sn[b])
        e = torch.nn.functional.pad(q[b], (0, 1, 0, 1))
        L = e[:, c0] + fu * (e[:, c0 + 1] - e[:, c0])
        lo = L.gather(0, r0)
        hi = L.gather(0, r0 + 1)
        acc += torch.where(vin, lo + fv * (hi - lo), 0.0) * (U2 * uin)
    vol = torch.zeros((nz, g.Y * g.X), dtype=torch.float64, device="cuda")
    vol[:, idx] = acc * _fscale(g)
    return vol.reshape(nz, g.Y, g.X)


def _forward64(g, vol, nz, zoff):
    """B^T vol: [N][H][W] float64, the transpose of _back64."""
    idx, aX, aY = _columns(g)
    aZ, (cs, sn) = _slices(g, nz, zoff), _angles(g)
    x = vol.double().reshape(nz, -1)[:, idx] * _fscale(g)
    out = torch.zeros((g.N, g.H, g.W), dtype=torch.float64, device="cuda")
    for b in range(g.N):
        (c0, fu, uin, U2), (r0, fv, vin) = _walk(g, aX, aY, aZ, cs[b], sn[b])
        w = torch.where(vin, x, 0.0) * (U2 * uin)
        G = torch.zeros((g.H + 1, idx.numel()), dtype=torch.float64, device="cuda")
        hi = w * fv
        G.scatter_add_(0, r0, w.sub_(hi))
        G.scatter_add_(0, r0 + 1, hi)
        e = torch.zeros((g.W + 1, g.H + 1), dtype=torch.float64, device="cuda")
        G = G.t().contiguous()
        e.index_add_(0, c0, G * (1 - fu)[:, None])
        e.index_add_(0, c0 + 1, G * fu[:, None])
        out[b] = e[:g.W, :g.H].t()
    return out


def _zoff(g):
    return -(g.Z - 1.0) / 2.0 - g.cz


def _fdk64(c, g, x, ff):
    q = torch.empty((g.N, g.H, g.W), dtype=torch.float64, device="cuda")
    p = _projections64(c, g, x, ff)
    for b in range(0, g.N, 32):
        q[b:b + 32] = _filtered(g, p[b:b + 32], c["window"])
    return q


def _scale64(c, g, p):
    """The power-of-two storage scale of the 16-bit formats (1 for the others)."""
    if c["precision"] in ("f32", "f32c"):
        return 1.0
    H, pad = _spectrum(g, c["window"])
    K = np.fft.irfft(H, pad) * pad
    l1 = abs(K[0]) + 2 * np.abs(K[1:g.W]).sum()
    if c["input"] == "u16":  # bounded without looking at the data
        fl, den = 0.5, I0
        bound = max(abs(math.log(fl / den)), abs(math.log(65535.0 / fl))) * l1
    else:
        w = torch.sqrt(g.D ** 2 + (torch.arange(g.W, device="cuda", dtype=torch.float64) - g.cX)[None, :] ** 2
                       + (torch.arange(g.H, device="cuda", dtype=torch.float64) - g.cZ)[:, None] ** 2)
        bound = float((p.abs().amax(0) * g.D / w).max()) * l1 * (1 + 2.0 ** -20)
        return 2.0 ** (14 - math.frexp(bound)[1])
    return 2.0 ** math.floor(math.log2(16384.0 / bound))


def exact(case, seed):
    kind = case["kind"]
    if kind != "rebin" and kind != "filter" and work(case)["flops"] > 1.6e12:
        return None  # longer than some seconds in 64 bits
    if kind == "rebin":
        return _rebin64(case, seed)
    if kind == "batch":
        vols = []
        for k, c in enumerate(_batch_cases(case)):
            g = _geometry(c)
            vols.append(_back64(g, _filtered(g, _line_integrals(g, seed * 100 + k), "ramlak"), g.Z, _zoff(g)))
        return vols
    g = _geometry(case)
    if kind == "engine":
        q = _filtered(g, _line_integrals(g, seed), "ramlak")
        return torch.cat([_back64(g, q, case["zb"], z) for z in _zoffsets(g, case["zb"])])
    if kind == "fdk":
        x, ff = _scan(case, g, seed)
        return _back64(g, _fdk64(case, g, x, ff), g.Z, _zoff(g))
    if kind == "filter":
        x, ff = _scan(case, g, seed)
        p = _projections64(case, g, x, ff)
        scale = _scale64(case, g, p)
        rows = []
        for b in range(0, g.N, 16):
            q = _filtered(g, p[b:b + 16], case["window"]) * scale
            if case["precision"] == "f32":
                rows.append(torch.nn.functional.pad(q, (0, device.row_pitch(g.W) - g.W)))
                continue
            Q, dU, dV, dUV = _coefficients(q)
            if case["precision"] == "f32c":
                rows.append(torch.stack((Q, dU, dV, dUV), -1).reshape(-1))
            else:
                e = torch.nn.functional.pad(torch.stack((Q, dV, dU, dUV), -1), (0, 0, 0, g.W % 2))
                rows.append(e.reshape(-1))
        return {"q": torch.cat(rows), "scale": torch.full((1,), scale, dtype=torch.float64)}
    if kind == "slab":
        q = _slab_q(case, g, seed)
        return _volume(g, seed, 0.01).double() + _back64(g, q, case["nz"], case["z0"])
    if kind == "backward":
        r = _forward64(g, _volume(g, seed), g.Z, _zoff(g))
        x = (torch.arange(g.W, device="cuda", dtype=torch.float64) - g.cX)[None, :]
        z = (torch.arange(g.H, device="cuda", dtype=torch.float64) - g.cZ)[:, None]
        w = g.D / torch.sqrt(g.D ** 2 + x * x + z * z)
        H, pad = _spectrum(g, case["window"])
        H = torch.from_numpy(H).cuda()
        for b in range(0, g.N, 32):
            r[b:b + 32] = torch.fft.irfft(torch.fft.rfft(r[b:b + 32], pad) * H, pad)[..., :g.W] * pad * w
        return r.transpose(0, 1).contiguous() if case["layout"] == "sinogram" else r
    q = _filtered(g, _line_integrals(g, seed), "ramlak")
    v = _volume(g, seed, float(q.std()) * 0.1).double()
    q = (q.half() if case["half"] else q.float()).double()
    loss = []
    for _ in range(case["steps"]):
        r = _forward64(g, v, g.Z, _zoff(g)) - q
        loss.append((r * r).sum())
        v = v - float(np.float32(_refine_alpha(case, g))) * _back64(g, r, g.Z, _zoff(g))
    return {"vol": v, "loss": torch.stack(loss)}


def _rebin64(c, seed):
    sino = torch.rand((c["rows"], c["N"], c["W"]), device="cuda", generator=_gen(seed)).double()
    W, N, am, D = c["W"], c["N"], c["am"], c["D"]
    dfi, c0 = 2.0 * math.pi / N, W - 1 - am
    wc = 2 * W - 1 - 2 * am

    def mix(at, col):
        """Rows at fractional angles `at` [n][cols] of the columns col, linear in the angle, wrapped."""
        lo = np.floor(at)
        f = torch.from_numpy(at - lo).cuda()
        k = torch.from_numpy(lo.astype(np.int64)).cuda()
        j = torch.from_numpy(col).cuda()
        return torch.stack([s[k % N, j] * (1 - f) + s[(k + 1) % N, j] * f for s in sino])

    if c["op"] == "full":
        f = np.arange(N, dtype=np.float64)[:, None]
        t = np.arange(c0, dtype=np.float64) - c0
        a = f - (2 * np.arctan(t / D) + np.pi) / dfi
        b = f - (2 * np.arctan(t / D) - np.pi) / dfi
        at = np.where((a < 0) | (a > N - 1), b, a)
        col = np.broadcast_to((am - t).astype(np.int64), at.shape).copy()
        out = torch.cat((mix(at, col), sino[:, :, am:]), 2)
        return out.flip(1) if c["flip"] else out
    f = np.arange(N // 2, dtype=np.float64)[:, None]
    s = np.arange(wc, dtype=np.float64) - c0
    shift = np.where(s >= 0, np.arcsin(s / D), np.pi - np.arcsin(s / D)) / dfi
    at = f + shift
    col = np.broadcast_to(np.minimum(np.abs(s) + am, W - 1).astype(np.int64), at.shape).copy()
    return mix(np.where(at < 0, at + N, at), col)
