"""The scan for the 16-bit storage scale sees every sample of a row with dark and flat maps, whatever the run of samples
that a lane loads at once (two for rows of up to 64, four up to 128, eight beyond): one attenuated sample anywhere sets
the same power-of-two scale, below the scale of the scan without it."""
import math

import numpy as np
import pytest

from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 31, 33, 63, 64, 65, 96, 97, 127, 128, 129, 255, 257, 400])
def test_one_sample_sets_the_scale(cuda, W):
    import torch

    H, N = 3, 2
    g = FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2, cZ=1.0, dfi=float(np.float32(math.pi)), D=1e6, tau=0.02, X=4, Y=4, Z=4,
                    cx=1.5, cy=1.5)  # D: cosine weights of one
    dark = torch.full((H, W), 100.0, device="cuda")
    flat = torch.full((H, W), 50100.0, device="cuda")
    ff = device.flatfield(flat=flat, dark=dark)

    def scale(at=None):
        raw = np.full((N, H, W), 49000, np.uint16)
        if at is not None:
            raw[at] = 110
        q, s = device.filter_projections(g, torch.from_numpy(raw.view(np.int16)).cuda(), _lib.TK_INPUT_U16,
                                         _lib.TK_LAYOUT_PROJECTION, ff, precision=_lib.TK_F16)
        return float(s)

    without, first = scale(), scale((0, 0, 0))
    assert first < without
    for x in range(W):
        assert scale(((x + 1) % N, x % H, x)) == first
    assert device.device_error_flags() == 0
