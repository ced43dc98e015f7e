"""The reconstruction's rounding beside the forward's: the error of a slice's combined image against FP64 is
at most what the error of its k-space and the error of combining that k-space give in quadrature (5 % for
the scatter of 4,096 voxels), so the two do not share their rounding; and the coils' images are within
1.5e-7, a dozen float32 roundings of a 64 x 64 transform."""
from __future__ import annotations

import math

import numpy as np
import pytest

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, SliceInput
from oracle import oracle
from tests import cases

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def test_errors_add_in_quadrature(gpu_ctx):
    n, coils = 64, 8
    s = cases.series_case(nx=n, ny=n, nz=1, o=2, nv=1, ncomp=2)
    y, x = np.meshgrid((np.arange(2 * n) + 0.5) / (2 * n), (np.arange(2 * n) + 0.5) / (2 * n), indexing="ij")
    inp = SliceInput(compartments=s["images"], t2=s["t2"], t_inhom=s["t_inhom"], fmap=s["fmap"], sim=(2 * n, 2 * n),
                     acq_matrix=(n, n), phase0=(0.4 * x - 0.7 * y * y).ravel())
    acq = Acquisition(n_coils=coils, t_line=0.5, t_echo=28.0, ghost_offset=0.02, noise_variance=0.0, n_spikes=0)
    out = api.simulate_slice_full(inp, acq, ctx=gpu_ctx)
    f = np.arange(n) - n // 2
    dft = np.exp(-2j * math.pi * np.outer(f, f) / n)
    sens = np.stack([[[oracle.lib().oracle_coil_sensitivity(q, coils, float(i), float(j), n, n) for i in range(n)]
                      for j in range(n)] for q in range(coils)])

    def combine(k):
        img = np.einsum("qkl,ky,lx->qyx", k, dft, dft)
        return img, (sens * img).sum(0) / (sens * sens).sum(0)

    want_k = np.stack([oracle.build_coil_kspace(inp, acq, q, coils).reshape(n, n) for q in range(coils)])
    images, own = combine(out["acquired"].astype(np.complex128))
    want = combine(want_k)[1]
    k_part, c_part, total = rel_l2(own, want), rel_l2(out["combined"], own), rel_l2(out["combined"], want)
    print(f"k-space {k_part:.3e}, combination {c_part:.3e}, both {total:.3e}")
    assert rel_l2(out["coil_images"], images) <= 1.5e-7
    assert total <= 1.05 * math.hypot(k_part, c_part)
