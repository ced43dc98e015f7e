"""Trajectory coordinates without a position (NaN, an infinity, or a value whose double overflows): the
kernels that order points, interpolate and spread form their grid cells from them, so every such cell
must be inside the grid, the point itself contributes and receives nothing, and the other points of the
call keep their values bit for bit.  Matrices on both sides of the tiled transform's rule (fine grids of
64 E points, and others), and segment counts on both sides of the wide point tiles' (33)."""
from __future__ import annotations

import math

import numpy as np
import pytest

from mrsim_acq_b200 import spiral as S
from mrsim_acq_b200.api import Acquisition, SliceInput, T2

pytestmark = pytest.mark.gpu
BAD = (math.nan, math.inf, -math.inf, 1.5e308)


def _spoil(k, at):
    """Coordinates `at` replaced, one axis or both in turn, by each of the values without a position."""
    out = k.copy()
    for i, j in enumerate(at):
        v = BAD[i % len(BAD)]
        if i % 3 != 1:
            out[j, 0] = v
        if i % 3 != 0:
            out[j, 1] = v
    return out


@pytest.mark.parametrize("n,o,hz,least", [(32, 2, 40.0, 1), (64, 2, 40.0, 1), (32, 2, 1000.0, 33), (18, 1, 40.0, 1),
                                          (20, 2, 40.0, 1)])
def test_segmented_forward(gpu_ctx, n, o, hz, least):
    sn = n * o
    rng = np.random.default_rng(n)
    tr = S.spiral_trajectory(n, n, 8, 4.096, 0.004, 1.2)
    k = tr.k.reshape(-1, 2).copy()
    idx = np.arange(len(k)) % len(tr.tau_ms)
    inp = SliceInput(compartments=[rng.uniform(0.0, 1.0, sn * sn).astype(np.float32)], t2=[T2.uniform(80.0)],
                     t_inhom=[T2.uniform(40.0)], fmap=rng.uniform(-hz, hz, sn * sn).astype(np.float32), sim=(sn, sn),
                     acq_matrix=(n, n), phase0=np.zeros(sn * sn))
    at = np.concatenate([[0, len(k) - 1], rng.choice(len(k), 40, replace=False)])
    at = np.unique(at)
    fine = np.setdiff1d(np.arange(len(k)), at)

    def run(kk):
        return S.spiral_segmented_forward(inp, Acquisition(n_coils=2, signal_scale=1.0), 0, 2, kk, idx, tr.tau_ms, 4.096,
                                          S.RateRect((0.0, 0.0), (-hz, hz)), None, False, ctx=gpu_ctx)

    want, info = run(k)
    assert info["l"] >= least
    bad = _spoil(k, at)
    got, _ = run(bad)
    assert np.array_equal(got[fine], want[fine])
    # the sum over the grid is 0 at such a point; the half-cell phase of a non-finite coordinate is NaN
    nan = ~np.isfinite(bad[at]).all(axis=1)
    assert np.all(np.isnan(got[at][nan])) and np.all(got[at][~nan] == 0)
    assert np.all(np.isfinite(want))


@pytest.mark.parametrize("n,lo,mo", [([16, 16], [-8, -8], [16, 16]), ([64, 64], [-32, -32], [64, 64])])
def test_pair(gpu_ctx, n, lo, mo):
    rng = np.random.default_rng(5)
    u = rng.uniform(-0.5, 0.5, (700, 2)) * np.array(n)
    w = rng.normal(size=700) + 1j * rng.normal(size=700)
    c = rng.normal(size=mo[0] * mo[1]) + 1j * rng.normal(size=mo[0] * mo[1])
    at = np.arange(3, 700, 17)
    fine = np.setdiff1d(np.arange(700), at)
    bad = _spoil(u, at)
    nu = S.Nufft2(n, lo, mo, 1e-12, ctx=gpu_ctx)
    got = nu.type2(c, bad, 1)
    assert np.array_equal(got[fine], nu.type2(c, u, 1)[fine])
    assert np.all(got[at] == 0)
    assert np.array_equal(nu.type1(bad, w, -1), nu.type1(u[fine], w[fine], -1))


def test_line(gpu_ctx):
    rng = np.random.default_rng(6)
    pos = rng.uniform(-32.0, 32.0, 300)
    wts = [rng.normal(size=300) + 1j * rng.normal(size=300)]
    at = np.arange(5, 300, 23)
    bad = pos.copy()
    bad[at] = [BAD[i % len(BAD)] for i in range(len(at))]
    fine = np.setdiff1d(np.arange(300), at)
    f = S.Nufft1(64, -20, 41, 1e-12, ctx=gpu_ctx)
    assert np.array_equal(f.run(bad, wts), f.run(pos[fine], [wts[0][fine]]))
