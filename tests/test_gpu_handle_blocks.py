"""The handle's regular (not pipelined) path with its volume in blocks: block
n + 1 is launched, on the other of two streams, before block n is delivered.
A sink that ends the call at any block leaves nothing behind: the same handle
then gives the volume of an undisturbed one, bit for bit."""
import numpy as np
import pytest

from _util import small_geometry
from tomokvas_gb300 import _lib
from tomokvas_gb300.fbp import FilteredBackProjection, VolumeSink
from tomokvas_gb300.phantom import head_phantom

pytestmark = pytest.mark.gpu


class EndingSink(VolumeSink):
    def __init__(self, g, last):
        super().__init__(g.X, g.Y, g.Z, g.zb)
        self.last = last

    def GetBlock(self, n, collecting=False):
        return None if n == self.last else super().GetBlock(n, collecting)


@pytest.mark.parametrize("last", [0, 1, 2, 4])
def test_a_sink_that_ends_the_call(orc, cuda, last):
    g = small_geometry(W=64, N=60, H=64, vol=(64, 64, 73), zb=16)  # five blocks, the last of nine slices
    sino = orc.project_ellipsoids(head_phantom(g.fov_radius_cm * 0.8, seed=8), orc.geom_from(g), "sino")
    fbp, ref = FilteredBackProjection(), FilteredBackProjection()
    try:
        for f in (fbp, ref):
            f.SetBlockSize(g.zb)
            f.SetSinogramProperties(sino, g.W, g.cX, g.N, g.H, g.cZ, g.dfi, g.D, g.tau)
            f.SetScaleXYZ(g.scale)
            f.SetPrecision("f32")
        full, got = VolumeSink(g.X, g.Y, g.Z, g.zb), VolumeSink(g.X, g.Y, g.Z, g.zb)
        ref.SetReconstructionProperties(full, g.X, g.cx, g.Y, g.cy, g.Z, g.cz, g.rot)
        assert ref.Initialize() == 0 and ref.CalculateReconstruction() == 0
        fbp.SetReconstructionProperties(EndingSink(g, last), g.X, g.cx, g.Y, g.cy, g.Z, g.cz, g.rot)
        assert fbp.Initialize() == 0
        assert fbp.CalculateReconstruction() == _lib.TK_ERR_IO
        fbp.SetReconstructionProperties(got, g.X, g.cx, g.Y, g.cy, g.Z, g.cz, g.rot)
        assert fbp.Initialize() == 0 and fbp.CalculateReconstruction() == 0
    finally:
        fbp.close()
        ref.close()
    assert [n for n, _ in got.blocks_requested] == [0, 1, 2, 3, 4]
    np.testing.assert_array_equal(got.volume, full.volume)
