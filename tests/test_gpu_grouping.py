"""The same slices in different company: a slab computed alone, a whole series, and a unit of one slice
give the same bits, whichever form of the y kernels, clusters of the reconstruction and launches each
plan's size selects (`shard.slab_inputs` and `AcquisitionOptions.slice_z`: what ranks compute is what a
single rank would)."""
from __future__ import annotations

import numpy as np
import pytest

from mrsim_acq_b200 import api, shard
from mrsim_acq_b200.api import Acquisition, AcquisitionInput, AcquisitionOptions, KspaceWindow, PhaseModel
from tests import cases

pytestmark = pytest.mark.gpu


def _operator(ctx, d, acq, grads, tes):
    op = api.EpiOperator(d["sim_dims"], d["acq_dims"], d["n_volumes"], d["t2"], d["fmap"], acq, images=d["images"],
                         echo_times_ms=tes, grads=grads, t_inhom=d["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42,
                         slice_z=d.get("slice_z"), nz_full=d.get("nz_full", 0), ctx=ctx)
    out = {k: v.copy() for k, v in op.apply_host(None).items() if v is not None}
    op.close()
    return out


# one to four coils, class rows, basis rows (warp FFT and DFT GEMM), one to four compartments, partial
# tiles of lines, rows and columns; slabs of one slice (thin tiles), of some, and the series (full tiles,
# and at 90 slices the launches without the chain)
@pytest.mark.parametrize("coils,nx,ny,o,ncomp,grads,nz,accel", [
    (1, 64, 64, 2, 1, 3, 12, 1), (1, 64, 64, 2, 1, 0, 160, 1), (2, 32, 50, 2, 2, 1, 30, 1), (4, 48, 33, 2, 3, 2, 20, 1),
    (8, 64, 64, 2, 3, 3, 12, 2), (8, 64, 37, 2, 2, 0, 24, 1), (8, 96, 96, 2, 2, 3, 6, 2), (16, 64, 64, 2, 3, 3, 12, 1),
    (6, 32, 64, 1, 4, 0, 30, 1), (32, 36, 40, 2, 2, 3, 16, 1), (3, 100, 17, 2, 1, 3, 30, 1)])
def test_operator_slabs(gpu_ctx, coils, nx, ny, o, ncomp, grads, nz, accel):
    s = cases.series_case(nx=nx, ny=ny, nz=nz, o=o, nv=1, ncomp=min(ncomp, 3))
    for c in range(3, ncomp):
        for k in ("images", "t2", "t_inhom"):
            s[k] = list(s[k]) + [s[k][c % 3]]
    acq = Acquisition(n_coils=coils, accel=accel, t_line=0.5, t_echo=40.0, ghost_offset=0.02)
    whole = _operator(gpu_ctx, s, acq, grads, [40.0])
    for z0, z1 in ((0, 1), (nz // 2, nz // 2 + 1), (1, 1 + nz // 3), (0, nz)):
        d = shard.slab_inputs(s["sim_dims"], s["acq_dims"], 1, s["images"], s["fmap"], z0, z1, s["t2"], s["t_inhom"])
        part = _operator(gpu_ctx, d, acq, grads, [40.0])
        for k, v in part.items():
            assert np.array_equal(v, whole[k][:, z0:z1]), (k, z0, z1)


@pytest.mark.parametrize("coils,n,ny,accel", [(8, 32, 32, 2), (16, 64, 32, 1), (5, 32, 64, 1), (8, 24, 40, 2)])
def test_series_slabs_through_the_reconstruction(gpu_ctx, coils, n, ny, accel):
    nz, nv = 20, 8  # 160 slices: blocks per slice from 2 (the series) to 8 (one slice)
    s = cases.series_case(nx=n, ny=ny, nz=nz, o=2, nv=nv, ncomp=2)
    acq = Acquisition(n_coils=coils, accel=accel, acs_lines=12, t_line=0.5, t_echo=40.0, ghost_offset=0.02,
                      window=KspaceWindow.hann(), noise_variance=1.0)

    def run(d, opts):
        r = api.simulate_acquisition_complex(
            AcquisitionInput(d["sim_dims"], d["acq_dims"], d["n_volumes"], d["images"], d["t2"], d["fmap"],
                             t_inhom=d["t_inhom"], phase=PhaseModel.hbcd_like(), seed=9), acq, opts, ctx=gpu_ctx)
        return np.stack([r["re"], r["im"]]).reshape(2, -1, ny, n, d["n_volumes"])

    whole = run(s, None)
    for z0, z1 in ((0, 1), (7, 9), (0, nz)):
        d = shard.slab_inputs(s["sim_dims"], s["acq_dims"], nv, s["images"], s["fmap"], z0, z1, s["t2"], s["t_inhom"])
        part = run(d, AcquisitionOptions(slice_z=d["slice_z"], nz_full=nz))
        assert np.array_equal(part, whole[:, z0:z1]), (z0, z1)
    if accel == 1:  # fewer volumes: the last chunk of a longer series
        few = dict(s, n_volumes=1, images=[np.ascontiguousarray(i.reshape(-1, nv)[:, 0]) for i in s["images"]])
        assert np.array_equal(run(few, None)[..., 0], whole[..., 0])
