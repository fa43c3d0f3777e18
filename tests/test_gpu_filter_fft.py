"""FFT filter at the edges of its transform lengths: one pad length below and above each power of two, the smallest
widths (one pass in registers), odd widths (the last column's neighbour is zero; the 16-bit images carry a pad
entry), one row, an odd number of rows, units of rows that do not divide the detector.

Oracle: the FP64 filter of the oracle library.  FP32 transform error: about log2(p) roundings of 2^-24 per value
relative to the row's largest, amplified by the ramp on smooth rows; random rows keep it below 2^-24 * 2 log2(p) <
2e-6; bound 4e-6 relative RMSE for FP32 samples, plus half an ulp of the entry for FP16 (2^-11)."""
import math

import numpy as np
import pytest

from _util import rel_rmse
from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


def _geo(W, H, N):
    return FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2 + 0.2, cZ=(H - 1) / 2, dfi=float(np.float32(2 * math.pi / N)),
                       D=6.0 * W + 40, tau=0.02, X=4, Y=4, Z=4, cx=1.5, cy=1.5)


@pytest.mark.parametrize("H,N", [(1, 3), (7, 2), (130, 3)])
@pytest.mark.parametrize("W", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 65, 129, 255, 257, 513, 1024, 1025, 2047, 2049])
def test_fft_filter_edges(orc, cuda, W, H, N):
    import torch

    L = _lib.load()
    g = _geo(W, H, N)
    G = orc.geom_from(g)
    x = np.random.default_rng(W * 7 + H).normal(size=(N, H, W)).astype(np.float32)
    sino = np.ascontiguousarray(x.transpose(1, 0, 2))
    ref = orc.weight_filter_f64(sino, G).transpose(1, 0, 2) * L.tk_pad_length(W)  # the oracle normalises by 1/p
    _lib.check(L.tk_filter_select_form(_lib.TK_FILTER_FFT))
    try:
        for layout, a in ((_lib.TK_LAYOUT_PROJECTION, x), (_lib.TK_LAYOUT_SINOGRAM, sino)):
            q, _ = device.filter_projections(g, torch.from_numpy(a).cuda(), layout=layout)
            assert rel_rmse(q[..., :W].cpu().numpy(), ref) < 4e-6
        if W <= 2048:
            q, s = device.filter_projections(g, torch.from_numpy(x).cuda(), layout=_lib.TK_LAYOUT_PROJECTION,
                                             precision=_lib.TK_F16)
            e = q.view(torch.float16).cpu().numpy().astype(np.float64).reshape(N, H, -1, 4)[:, :, :W] / float(s)
            full = np.zeros((N, H + 1, W + 1))
            full[:, :H, :W] = ref
            Q, r, d, rd = full[:, :-1, :-1], full[:, :-1, 1:], full[:, 1:, :-1], full[:, 1:, 1:]
            want = np.stack((Q, d - Q, r - Q, (rd - d) - (r - Q)), -1)
            assert rel_rmse(e, want) < 4e-6 + 2.0 ** -11
    finally:
        _lib.check(L.tk_filter_select_form(_lib.TK_FILTER_AUTO))
    assert device.device_error_flags() == 0
