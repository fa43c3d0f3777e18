"""Tile shapes of the general backprojection walks by footprint: wide cones and slabs far from the mid-plane, whose thin
FP32 tiles (eight staged boxes nearly as tall as a 32-slice tile's four) do not fit shared memory, and large footprints,
which take 16 x 16 columns instead of 16 x 8.  Whatever is picked runs, and gives the bits of each form that can run."""
import math

import numpy as np
import pytest

from tomokvas_gb300 import _lib, device
from tomokvas_gb300.geometry import FDKGeometry

pytestmark = pytest.mark.gpu


def _walks(L, prefix):
    names = [L.tk_bp_variant_name(i).decode() for i in range(L.tk_bp_variant_count())]
    return [i for i, n in enumerate(names) if n.startswith(prefix)]


@pytest.mark.parametrize("W,N,H,X,nz,D,scale,zoff,cZ,precision", [
    (48, 448, 96, 84, 208, 35.2, 0.39, None, None, "f32"),     # 16 x 16 x 32 needs 229936 B, 8-slice tiles 233040 B
    (64, 96, 1000, 64, 16, 140.0, 1.0, 560.0, 0.0, "f32"),     # 8- and 4-slice tiles need more than 232448 B
    (190, 30, 150, 128, 100, 400.0, 1.45, None, None, "f32"),  # 16 x 16 columns
    (190, 30, 150, 128, 100, 400.0, 1.45, None, None, "f16"),
    (190, 30, 150, 128, 100, 400.0, 1.45, None, None, "bf16"),
    (190, 30, 60, 120, 20, 400.0, 1.45, None, None, "f16"),    # fewer slices than a tile has
])
def test_large_footprints(cuda, W, N, H, X, nz, D, scale, zoff, cZ, precision):
    import torch

    L = _lib.load()
    prec = _lib.PRECISIONS[precision]
    g = FDKGeometry(W=W, N=N, H=H, cX=(W - 1) / 2, cZ=(H - 1) / 2 if cZ is None else cZ,
                    dfi=float(np.float32(2 * math.pi / N)), D=D, tau=0.02, X=X, Y=X, Z=nz, cx=(X - 1) / 2,
                    cy=(X - 1) / 2, rot=0.05, scale=scale)
    rng = np.random.default_rng(X)
    if precision == "f32":
        q = torch.from_numpy(rng.normal(size=(N, H, device.row_pitch(W))).astype(np.float32)).cuda()
        scale_word = None
    else:
        x = torch.from_numpy(rng.normal(size=(N, H, W)).astype(np.float32)).cuda()
        q, scale_word = device.filter_projections(g, x, layout=_lib.TK_LAYOUT_PROJECTION, precision=prec)
    want = device.backproject(g, q, scale_word, prec, nz=nz, zoff=zoff).cpu().numpy()
    assert np.abs(want).max() > 0
    ran = 0
    try:
        for i in _walks(L, "direct_" if precision == "f32" else f"cimg_f32i<{precision},"):
            if L.tk_bp_variant_name(i).decode().startswith("direct<"):
                continue  # the unpacked walk
            _lib.check(L.tk_bp_select_variant(i))
            try:
                got = device.backproject(g, q, scale_word, prec, nz=nz, zoff=zoff).cpu().numpy()
            except Exception as e:  # a selected form that does not fit says so
                assert "shared memory" in str(e)
                continue
            ran += 1
            np.testing.assert_array_equal(got, want)
    finally:
        _lib.check(L.tk_bp_select_variant(-1))
    assert ran >= 2
    assert device.device_error_flags() == 0


@pytest.mark.parametrize("precision", ["f16", "bf16", "f32c"])
@pytest.mark.parametrize("W,X,nz,D,scale,zoff,flips", [(80, 64, 1, 300.0, 1.0, -3.0, 0), (90, 70, 2, 260.0, 1.2, 10.5, 4),
                                                       (60, 75, 5, 150.0, 0.7, -40.0, 3), (130, 88, 33, 420.0, 1.3, -16.0, 5),
                                                       (64, 50, 63, 300.0, 1.0, -31.0, 1)])
def test_thin_slabs_same_bits(cuda, precision, W, X, nz, D, scale, zoff, flips):
    """Fewer slices than a chunk, whose staged boxes hold the rows of those slices only, against the first slices of a
    whole chunk."""
    import torch

    prec = _lib.PRECISIONS[precision]
    g = FDKGeometry(W=W, N=17, H=100, cX=(W - 1) / 2, cZ=48.3, dfi=float(np.float32(2 * math.pi / 17)), D=D, tau=0.02,
                    X=X, Y=X - 5, Z=nz, cx=(X - 1) / 2 + 0.7, cy=(X - 6) / 2, rot=0.05, scale=scale, dirx=flips & 1,
                    diry=flips >> 1 & 1, dirz=flips >> 2 & 1)
    x = torch.from_numpy(np.random.default_rng(nz).normal(size=(g.N, g.H, W)).astype(np.float32)).cuda()
    q, s = device.filter_projections(g, x, layout=_lib.TK_LAYOUT_PROJECTION, precision=prec)
    thin = device.backproject(g, q, s, prec, nz=nz, zoff=zoff).cpu().numpy()
    whole = device.backproject(g, q, s, prec, nz=64, zoff=zoff).cpu().numpy()
    assert np.abs(thin).max() > 0
    np.testing.assert_array_equal(thin, whole[:nz])
    assert device.device_error_flags() == 0
