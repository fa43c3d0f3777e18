"""A frame's coefficient image does not depend on the frames that are filtered with it: the FFT form gives the same bits
for N frames in one call, in chunks and one by one (the rows per work unit follow the number of frames, the row pairs of
a transform must not).  Streamed and pipelined reconstructions filter in chunks."""
import math

import numpy as np
import pytest

from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,N,precision", [(600, 130, 45, "f16"), (520, 67, 33, "bf16"), (601, 300, 24, "f16"),
                                             (300, 257, 60, "f32c"), (60, 96, 90, "f32c"), (1030, 72, 20, "f32c")])
def test_frames_in_chunks_same_bits(cuda, W, H, N, precision):
    import torch

    prec = _lib.PRECISIONS[precision]
    rng = np.random.default_rng(W + H)
    x = torch.from_numpy(rng.integers(200, 50000, size=(N, H, W)).astype(np.uint16).view(np.int16)).cuda()
    ff = device.flatfield(flat_value=50000.0, dark_value=100.0)  # the 16-bit storage scale does not follow the data

    def images(n):
        out = []
        for b in range(0, N, n):
            k = min(n, N - b)
            g = FDKGeometry(W=W, N=k, H=H, cX=(W - 1) / 2, cZ=(H - 1) / 2, dfi=float(np.float32(2 * math.pi / N)),
                            D=5.0 * W, tau=0.02, X=4, Y=4, Z=4, cx=1.5, cy=1.5)
            q, _ = device.filter_projections(g, x[b:b + k].contiguous(), _lib.TK_INPUT_U16, _lib.TK_LAYOUT_PROJECTION,
                                             ff, precision=prec)
            out.append(q.reshape(k, -1).cpu().numpy())
        return np.concatenate(out)

    _lib.check(_lib.load().tk_filter_select_form(_lib.TK_FILTER_FFT))
    try:
        whole = images(N)
        for n in (1, 7, 16):
            np.testing.assert_array_equal(images(n), whole)
    finally:
        _lib.check(_lib.load().tk_filter_select_form(_lib.TK_FILTER_AUTO))
    assert device.device_error_flags() == 0
