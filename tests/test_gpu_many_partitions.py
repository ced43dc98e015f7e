"""3D trains of more partitions than a z-DFT tile's shared memory holds (3,632), and the last that fits:
against the FP64 oracle.  A partition's sum has 3,640 FP32 terms: sqrt(3640) half-ulps is 2e-6, inside the
bar of 1e-5."""
from __future__ import annotations

import numpy as np
import pytest

from cases3d import blobs, grase, train
from mrsim_acq_b200 import kspace3d as K3
from mrsim_acq_b200.api import Acquisition, T2
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("nz,segments,maps", [(3632, 227, False), (3640, 364, False), (3640, 364, True)])
def test_partitions_past_shared_memory(gpu_ctx, nz, segments, maps):
    n = 4
    t2 = T2.of_map(np.full(n * n * nz, 80.0, np.float32)) if maps else T2.uniform(80.0)
    args = ([n, n, nz], [n, n, nz], 1, blobs(n, n, nz, 1, 1), [t2], [T2.uniform(1330.0)],
            np.full(n * n * nz, 3.0, np.float32), None, Acquisition(n_coils=2, signal_scale=100.0),
            train(nz, segments, esp_ms=5.0), grase(1, 0.1))
    assert rel_l2(K3.kspace_3d_observed(*args, g=0, ctx=gpu_ctx), O.kspace_3d_observed(*args, g=0)) <= 1e-5
    mag, ph = K3.simulate_acquisition_3d(*args, seed=42, ctx=gpu_ctx)
    vols, _, _ = O.simulate_acquisition_3d(*args, seed=42)
    assert rel_l2(mag.astype(np.float64) * np.exp(1j * ph.astype(np.float64)), vols.T.ravel()) <= 1e-5
