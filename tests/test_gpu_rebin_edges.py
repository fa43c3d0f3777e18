"""Half-fan completion and rebinning where batches of eight angles start, end, wrap and change conjugate: fewer angles
than a batch, one more and one less than whole batches, chunks of angles, single rows and columns left of the axis.
Against the FP64 restatement; bound as in test_gpu_rebin.py: FP32 rounding of the samples, 1e-6 of their range."""
import math

import numpy as np
import pytest

from tomokvas_gb300 import device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,N,am,D,rows", [(3, 2, 0, 9.0, 1), (9, 6, 2, 40.0, 2), (17, 8, 1, 60.5, 1), (17, 10, 15, 60.0, 3),
                                           (40, 16, 3, 90.0, 1), (130, 18, 0, 400.0, 2), (70, 66, 5, 150.0, 1),
                                           (33, 254, 2, 34.5, 5), (129, 1026, 0, 700.0, 1)])
def test_batches_of_angles(orc, cuda, W, N, am, D, rows):
    import torch

    dfi = 2 * math.pi / N
    sino = np.random.default_rng(W * N).normal(size=(rows, N, W)).astype(np.float32)
    d = torch.from_numpy(sino).cuda()
    tol = 1e-6 * np.abs(sino).max()
    for flip in (False, True):
        got = device.half_to_full_fan(d, am, D, dfi, flip).cpu().numpy()
        assert np.abs(got - orc.half2fullfan(sino.astype(np.float64), am, D, dfi, flip)).max() <= tol
    got = device.half_to_parallel(d, am, D, dfi).cpu().numpy()
    assert np.abs(got - orc.half2para(sino.astype(np.float64), am, D, dfi)).max() <= tol
