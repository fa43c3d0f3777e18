"""Thin tiles of the FP32 backprojection for small volumes (8 and 4 slices instead of 32): the same operations per
voxel, so the same bits as the 32-slice tiles, for every remainder of the slices, accumulating or not."""
import math

import numpy as np
import pytest

from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y,nz,N,flips", [(20, 33, 1, 1, 0), (48, 40, 3, 7, 4), (64, 64, 4, 30, 0), (16, 16, 9, 5, 3),
                                            (40, 50, 31, 8, 0), (33, 17, 67, 13, 5)])
def test_thin_tiles_same_bits(cuda, X, Y, nz, N, flips):
    import torch

    L = _lib.load()
    names = [L.tk_bp_variant_name(i).decode() for i in range(L.tk_bp_variant_count())]
    idx = [i for i, n in enumerate(names) if n.startswith("direct_x2<f32,")]
    assert sorted(int(names[i].split(",")[3]) for i in idx) == [4, 8, 32]
    g = FDKGeometry(W=60, N=N, H=37, cX=29.7, cZ=18.2, dfi=float(np.float32(2 * math.pi / N)), D=380.0, tau=0.02, X=X,
                    Y=Y, Z=nz, cx=(X - 1) / 2 + 1.5, cy=(Y - 1) / 2, rot=0.3, scale=1.1, dirx=flips & 1,
                    diry=flips >> 1 & 1, dirz=flips >> 2 & 1)
    rng = np.random.default_rng(nz)
    q = torch.from_numpy(rng.normal(size=(N, g.H, device.row_pitch(g.W))).astype(np.float32)).cuda()
    v0 = torch.from_numpy(rng.normal(size=(nz, Y, X)).astype(np.float32)).cuda()
    for acc in (False, True):
        out = []
        try:
            for i in [-1] + idx:
                _lib.check(L.tk_bp_select_variant(i))
                out.append(device.backproject(g, q, None, vol=v0.clone(), zoff=-3.5, accumulate=acc).cpu().numpy())
        finally:
            _lib.check(L.tk_bp_select_variant(-1))
        assert np.abs(out[0] - (v0.cpu().numpy() if acc else 0)).max() > 0
        for o in out[1:]:
            np.testing.assert_array_equal(o, out[0])
    assert device.device_error_flags() == 0
