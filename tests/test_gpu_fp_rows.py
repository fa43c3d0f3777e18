"""Row-lane forward projector (the default form of B^T) at the edges of its tiles: K = 2, 3 and 4 slices per
detector row (row steps from 1, 2/3 and 1/2), ragged 16 x 8 tiles, one slice, slices past a chunk, volumes that
leave the detector on every side, flips and a negative voxel pitch, fewer projections than warps, slabs.

Reference: the slice-lane form with FP32 atomics, which scatters the same weights (v and u with the same
roundings).  The two differ by FP32 rounding: three products per contribution and a few hundred additions per
sample in another order, about 2^-24 sqrt(100) = 6e-7 at the most of the root mean square; bound 1e-6."""
import math

import numpy as np
import pytest

from _util import rel_rmse
from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,N,H,X,Y,Z,D,scale,shift,flips,zoff", [
    (64, 40, 64, 64, 64, 48, 400.0, 1.0, 0.0, 0, None),
    (64, 3, 70, 17, 9, 65, 300.0, 1.3, 1.1, 1, None),      # K = 2, fewer projections than warps
    (60, 130, 20, 50, 33, 40, 280.0, 0.8, -3.0, 6, None),   # K = 3, rows masked above and below
    (48, 21, 48, 90, 70, 33, 260.0, 0.62, 2.0, 4, None),    # K = 4, columns past both detector edges
    (33, 7, 21, 33, 31, 1, 200.0, 1.2, 0.0, 0, None),
    (64, 30, 64, 40, 40, 30, 400.0, -1.1, 1.0, 3, None),
    (64, 24, 64, 48, 48, 20, 400.0, 1.5, 0.0, 5, -31.25),   # a slab that starts outside the detector
    (200, 9, 300, 60, 60, 90, 1000.0, 2.4, 0.0, 0, None),
])
def test_row_lanes_match_slice_lanes(cuda, W, N, H, X, Y, Z, D, scale, shift, flips, zoff):
    import torch

    L = _lib.load()
    g = FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2 + 0.3 * shift, cZ=(H - 1) / 2 - 0.2 * shift,
                    dfi=float(np.float32(2 * math.pi / N)), D=D, tau=0.02, X=X, Y=Y, Z=Z, cx=(X - 1) / 2 + shift,
                    cy=(Y - 1) / 2 - 0.4 * shift, rot=0.1 * shift, scale=scale, dirx=flips & 1, diry=flips >> 1 & 1,
                    dirz=flips >> 2 & 1)
    y = torch.from_numpy(np.random.default_rng(W + Z).normal(size=(Z, Y, X)).astype(np.float32)).cuda()
    out = []
    try:
        for v in (0, 2):
            _lib.check(L.tk_fp_select_variant(v))
            acc = torch.ones((g.N, g.H, device.row_pitch(g.W)), device="cuda")  # accumulated into
            q = device.forward_project(g, y, zoff=zoff, out=acc, accumulate=True)
            out.append(q[..., :W].cpu().numpy().astype(np.float64) - 1.0)
            out.append(device.forward_project(g, y, zoff=zoff)[..., :W].cpu().numpy().astype(np.float64))
    finally:
        _lib.check(L.tk_fp_select_variant(0))
    assert device.device_error_flags() == 0
    assert np.abs(out[3]).max() > 0
    assert rel_rmse(out[1], out[3]) < 1e-6
    # added to ones: one rounding of sums near 1 per partial sum, at most ten of them
    assert np.abs(out[0] - out[1]).max() <= 10 * 2.0 ** -24 * (1 + np.abs(out[1]).max())
