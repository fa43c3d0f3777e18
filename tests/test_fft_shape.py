"""Index rules of the FFT filter on the host (tests/cpp/fft_shape_check.cpp over csrc/tk_fft_shape.h), and on the GPU the
widths of few butterflies (pad lengths to 256), whose transforms share a warp and where a thread without a column once
read another group's buffer.

GPU bound: as for the other lengths, the FP32 transform's error is below 2e-6 of the filtered rows' RMS (about log2(p)
roundings of 2^-24 per value, random rows); dU, dV and dUV are differences of such values, formed in FP32: 4e-6 relative
RMSE over all four."""
import math
import os
import subprocess

import numpy as np
import pytest

from _util import rel_rmse
from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_edge_reads_stay_in_their_group(tmp_path):
    exe = str(tmp_path / "fft_shape_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "tomokvas_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fft_shape_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("W", [1, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65, 100, 112, 127, 128])
def test_coefficients_of_narrow_rows(orc, cuda, W):
    import torch

    H, N = 75, 40  # several groups per CTA, several units per projection
    g = FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2 + 0.2, cZ=(H - 1) / 2, dfi=float(np.float32(2 * math.pi / N)),
                    D=6.0 * W, tau=0.02, X=4, Y=4, Z=4, cx=1.5, cy=1.5)
    x = np.random.default_rng(W).normal(size=(N, H, W)).astype(np.float32)
    ref = orc.weight_filter_f64(np.ascontiguousarray(x.transpose(1, 0, 2)), orc.geom_from(g)).transpose(1, 0, 2)
    full = np.zeros((N, H + 1, W + 1))
    full[:, :H, :W] = ref * _lib.load().tk_pad_length(W)  # the oracle normalises by 1/p
    Q, r, d, rd = full[:, :-1, :-1], full[:, :-1, 1:], full[:, 1:, :-1], full[:, 1:, 1:]
    want = np.stack((Q, r - Q, d - Q, (rd - d) - (r - Q)), -1)
    q, _ = device.filter_projections(g, torch.from_numpy(x).cuda(), layout=_lib.TK_LAYOUT_PROJECTION,
                                     precision=_lib.TK_F32_COEF)
    got = q.view(torch.float32).cpu().numpy().reshape(N, H, W, 4)
    assert rel_rmse(got, want) < 4e-6
    assert device.device_error_flags() == 0
