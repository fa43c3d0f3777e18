"""Forms of the forward projector at large footprints and fine voxels.  Slice lanes where the default takes them: row
steps below 1/2 (many contributions per cell: both words of the fixed-point box with their bias subtraction) and
footprints that leave the row lanes no shape (few contributions: the hi word windowed, or both words).  Row lanes whose
chunks are cut short by shared memory, in volumes small enough that they are still the faster form.

Reference: the slice lanes with FP32 atomics, the same weights in another order of addition; as for the row lanes,
three roundings per contribution and a few hundred additions per sample: below 1e-6 of the root mean square."""
import math

import numpy as np
import pytest

from _util import rel_rmse
from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu

# (W, N, H, X, Y, Z, D, scale, flips); in the names the most contributions per cell, as a power of two, or the slices of a
# row-lane chunk
GEOMS = {
    "cbits11_fine": (64, 30, 48, 60, 52, 45, 260.0, 0.35, 5),
    "cbits9_wide": (64, 21, 64, 42, 42, 37, 70.0, 1.0, 0),
    "cbits8_wide": (64, 24, 60, 30, 28, 40, 80.0, 1.3, 2),
    "cbits6_coarse": (160, 9, 200, 50, 44, 70, 420.0, 2.4, 4),
    "one_chunk": (160, 16, 90, 60, 56, 20, 420.0, 2.3, 1),
    "rows_11_slices": (112, 40, 112, 64, 60, 61, 448.0, 1.5, 2),
    "rows_9_slices": (88, 21, 90, 64, 50, 50, 176.0, 1.2, 5),
}


def _geometry(name):
    W, N, H, X, Y, Z, D, scale, flips = GEOMS[name]
    return FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2 + 0.3, cZ=(H - 1) / 2 - 0.2, dfi=float(np.float32(2 * math.pi / N)),
                       D=D, tau=0.02, X=X, Y=Y, Z=Z, cx=(X - 1) / 2, cy=(Y - 1) / 2, rot=0.1, scale=scale,
                       dirx=flips & 1, diry=flips >> 1 & 1, dirz=flips >> 2 & 1)


@pytest.mark.parametrize("name", list(GEOMS))
def test_default_matches_fp32_atomics(cuda, name):
    import torch

    L = _lib.load()
    g = _geometry(name)
    y = torch.from_numpy(np.random.default_rng(5).normal(size=(g.Z, g.Y, g.X)).astype(np.float32)).cuda()
    out = []
    try:
        for v in (0, 2):
            _lib.check(L.tk_fp_select_variant(v))
            out.append(device.forward_project(g, y)[..., :g.W].cpu().numpy().astype(np.float64))
    finally:
        _lib.check(L.tk_fp_select_variant(0))
    assert np.abs(out[1]).max() > 0
    assert rel_rmse(out[0], out[1]) < 1e-6
    assert device.device_error_flags() == 0
