"""Inputs that the filter kernels read in different ways -- rows aligned to 16, 8, 4 and 2 bytes (by width and by the
buffer's start), FP32 and uint16, with a dark map, a flat map, both or none, map rows aligned or not -- give what the
same samples give as FP32 line integrals formed here.

Bound: the device forms log(t) with an absolute error below 4e-7 per sample and the Toeplitz product carries 2e-5
relative; log values here have an RMS above 0.3, random from sample to sample, so 4e-7 / 0.3 stays below 2e-6 and
FP16 entries add half an ulp, 2^-11: 1e-5 for FP32 samples by the FFT, 4e-5 + 2^-11 for FP16 entries."""
import math

import numpy as np
import pytest

from _util import rel_rmse
from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


def _padded(a, torch, skip):
    """Device copy of a that starts `skip` elements into a 256-byte aligned buffer."""
    flat = torch.zeros(a.size + skip, dtype=torch.int16 if a.dtype == np.uint16 else torch.float32, device="cuda")
    flat[skip:] = torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda().reshape(-1)
    return flat[skip:]


@pytest.mark.parametrize("maps", ["none", "dark", "flat", "both"])
@pytest.mark.parametrize("W,skip", [(64, 0), (64, 4), (60, 0), (62, 2), (61, 0), (64, 1), (130, 0), (200, 0), (201, 3),
                                    (385, 0), (500, 0), (512, 0)])
def test_rows_and_maps(cuda, W, skip, maps):
    import torch

    H, N = 9, 3
    g = FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2, cZ=(H - 1) / 2, dfi=float(np.float32(2 * math.pi / N)), D=5.0 * W,
                    tau=0.02, X=4, Y=4, Z=4, cx=1.5, cy=1.5)
    rng = np.random.default_rng(W + skip)
    raw = rng.integers(200, 40000, size=(N, H, W)).astype(np.uint16)
    dark = rng.uniform(50, 150, size=(H, W)).astype(np.float32)
    flat = rng.uniform(45000, 55000, size=(H, W)).astype(np.float32)
    d = torch.from_numpy(dark).cuda() if maps in ("dark", "both") else None
    f = torch.from_numpy(flat).cuda() if maps in ("flat", "both") else None
    ff = device.flatfield(flat=f, dark=d, flat_value=50000.0, dark_value=100.0)
    dk = dark.astype(np.float64) if d is not None else 100.0
    fl = flat.astype(np.float64) if f is not None else 50000.0
    line = -np.log(np.maximum(raw - dk, 0.5) / (fl - dk)) * np.ones((N, H, W))
    x16, x32 = _padded(raw, torch, skip), _padded(line.astype(np.float32), torch, skip)
    lay = _lib.TK_LAYOUT_PROJECTION
    want, _ = device.filter_projections(g, torch.from_numpy(line.astype(np.float32)).cuda(), layout=lay)
    want = want[..., :W].cpu().numpy().astype(np.float64)
    full = np.zeros((N, H + 1, W + 1))
    full[:, :H, :W] = want
    Q, r, b, rb = full[:, :-1, :-1], full[:, :-1, 1:], full[:, 1:, :-1], full[:, 1:, 1:]
    want16 = np.stack((Q, b - Q, r - Q, (rb - b) - (r - Q)), -1)
    for x, kind, fa in ((x16, _lib.TK_INPUT_U16, ff), (x32, _lib.TK_INPUT_F32, None)):
        q, _ = device.filter_projections(g, x, kind, lay, fa)
        assert rel_rmse(q[..., :W].cpu().numpy(), want) < 1e-5
        q, s = device.filter_projections(g, x, kind, lay, fa, precision=_lib.TK_F16)
        e = q.view(torch.float16).cpu().numpy().astype(np.float64).reshape(N, H, -1, 4)[:, :, :W] / float(s)
        assert rel_rmse(e, want16) < 4e-5 + 2.0 ** -11
    assert device.device_error_flags() == 0
