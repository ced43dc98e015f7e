"""The whole slice pipeline against the FP64 oracle (relative L2 <= 1e-5, the bar of every FP32 result)
where the reconstruction kernels change form: the FFT combine (32 E points per axis, one and several
blocks to a slice, odd coil counts) and the direct sums beside it; GRAPPA systems in and out of shared
memory (16 and 17 coils), three-fold acceleration (two offsets), coil counts off the eight coils a thread
fills, band widths off the readout chunk; and the z-DFT's partition tiles (whole and partial, shared and
per-shot images are in the GRASE tests)."""

import numpy as np
import pytest

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, KspaceWindow, PartialFourierMode, SliceInput, T2
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,coils,accel,acs,window", [
    (32, 32, 1, 1, 0, "none"), (32, 64, 3, 1, 0, "hann"), (64, 32, 8, 1, 0, "none"), (64, 64, 8, 2, 24, "hann"),
    (96, 64, 5, 1, 0, "hann"), (64, 96, 2, 2, 20, "none"), (128, 96, 4, 1, 0, "hann"), (128, 128, 3, 1, 0, "none"),
    (96, 128, 9, 1, 0, "none"), (40, 32, 4, 3, 16, "hann"), (33, 48, 10, 2, 16, "none"), (32, 64, 16, 2, 20, "none"),
    (32, 48, 17, 2, 16, "none"), (64, 64, 7, 3, 24, "hann")])
def test_slice_matches_the_oracle(gpu_ctx, nx, ny, coils, accel, acs, window):
    y, x = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
    img = (np.exp(-((x - 0.45) ** 2 + (y - 0.55) ** 2) / 0.05) + 0.3 * (np.hypot(x - 0.6, y - 0.4) < 0.2)).astype(np.float32)
    inp = SliceInput(compartments=[img.ravel()], t2=[T2.uniform(80.0)], fmap=(30.0 * (x - y)).astype(np.float32).ravel(),
                     sim=(nx, ny), acq_matrix=(nx, ny), phase0=(0.5 * x - 0.3 * y).ravel(), slice_seed=7)
    acq = Acquisition(n_coils=coils, accel=accel, acs_lines=acs, t_line=0.4, t_echo=60.0, noise_variance=0.5,
                      partial_fourier=0.75 if accel == 2 else 1.0, pf_mode=PartialFourierMode.Scanner,
                      window=KspaceWindow.hann() if window == "hann" else KspaceWindow.none())
    got = api.simulate_slice_full(inp, acq, ctx=gpu_ctx)
    want = oracle.simulate_slice_full(inp, acq)
    for key in ("coil_images", "combined"):
        w = np.asarray(want[key])
        err = np.linalg.norm(np.ravel(got[key]) - np.ravel(w)) / np.linalg.norm(w)
        assert err <= 1e-5, (key, err)
