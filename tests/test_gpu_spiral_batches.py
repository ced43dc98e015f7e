"""Reconstructions of more images than one pass takes (592 where the iterations are one launch, 256 where
they are a launch per step): each image equals its own reconstruction, in FP64, across the passes' ends."""
from __future__ import annotations

import numpy as np
import pytest

from mrsim_acq_b200 import spiral as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,il,dw,batch,at", [(32, 4, 0.008, 594, (0, 255, 256, 591, 592, 593)),
                                              (24, 4, 0.008, 258, (0, 255, 256, 257))])
def test_images_past_one_pass(gpu_ctx, n, il, dw, batch, at):
    tr = S.spiral_trajectory(n, n, il, 4.0, dw, 1.2)
    rec = S.SpiralRecon(tr.k.reshape(-1, 2), n, ctx=gpu_ctx)
    rng = np.random.default_rng(n)
    d = rng.normal(size=(batch, rec.npts)) + 1j * rng.normal(size=(batch, rec.npts))
    got = rec.image(d)
    assert got.shape == (batch, n, n) and np.all(np.isfinite(got))
    for b in at:
        one = rec.image(d[b])
        # the spread's order differs with the batch: 80 steps at condition 100 of 2e-16 each
        assert np.linalg.norm(got[b] - one) <= 1e-10 * np.linalg.norm(one)
    rec.close()
