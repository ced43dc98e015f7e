"""The EPI operator on coil-basis rows against the FP64 oracle (relative L2 <= 1e-5, the bar of every
FP32 result): rings of 6 to 64 coils, where the basis has 4, 6 or 7 rows; rows in the warp FFT (one
width, and several in one plan), in the DFT GEMM (even and odd widths, copies of 4 and 8 bytes);
lines that leave a partial tile; more coils than an adjoint tile holds; voxel maps and eddy currents;
and the plans that keep one row per coil."""

import numpy as np
import pytest

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, PartialFourierMode, PhaseModel
from oracle import oracle
from tests import cases

pytestmark = pytest.mark.gpu
TOL = 1e-5


def rel_l2(a, b):
    n = np.linalg.norm(np.ravel(b))
    return np.linalg.norm(np.ravel(a) - np.ravel(b)) / (n if n > 0 else 1.0)


@pytest.mark.parametrize("coils,nx,ny,o,ncomp,maps,extra", [
    (6, 16, 16, 2, 3, False, {}),  # 4 rows, E = 1
    (7, 16, 24, 2, 2, False, {}),
    (9, 32, 18, 2, 1, False, {}),
    (10, 48, 16, 2, 3, False, dict(accel=2)),  # 6 rows, E = 3
    (12, 64, 20, 2, 3, True, {}),
    (16, 80, 16, 2, 4, False, {}),  # E = 5
    (8, 96, 20, 2, 2, False, dict(partial_fourier=0.75, pf_mode=PartialFourierMode.Scanner)),  # E = 6
    (32, 112, 8, 2, 2, False, {}),  # E = 7
    (32, 128, 12, 2, 3, False, dict(ghost_offset=0.03)),  # E = 8
    (33, 32, 16, 1, 2, False, {}),  # one coil past an adjoint tile
    (64, 64, 10, 2, 1, True, {}),
    (12, 75, 14, 2, 2, True, {}),  # DFT GEMM, 4-byte copies
    (11, 17, 21, 1, 3, False, {}),  # odd rows: 8-byte copies
    (32, 19, 17, 3, 2, False, {}),
    (40, 21, 16, 1, 2, False, {}),  # more coils than a GEMM tile: one row per coil
    (16, 16, 16, 2, 5, False, {}),  # eight-compartment kernels: one row per coil
    (12, 32, 16, 2, 2, False, dict(eddy_strength=2.0, eddy_quad=0.3, eddy_tau=70.0)),
    (12, 45, 16, 2, 2, False, dict(eddy_strength=2.0, eddy_quad=0.3, eddy_tau=70.0)),
])
def test_basis_operator_matches_the_oracle(gpu_ctx, coils, nx, ny, o, ncomp, maps, extra):
    s = cases.series_case(nx=nx, ny=ny, nz=2, o=o, nv=2, ncomp=min(ncomp, 3), maps=maps)
    for c in range(3, ncomp):
        for k in ("images", "t2", "t_inhom"):
            s[k] = list(s[k]) + [s[k][c % 3]]
    acq = Acquisition(n_coils=coils, t_line=0.5, t_echo=30.0, **extra)
    kw = dict(t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42)
    if "eddy_strength" in extra:
        kw["eddy_drive"] = [(0.3, -0.8, 0.5), (0.5, 0.5, 0.7)]
    op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 2, s["t2"], s["fmap"], acq, images=s["images"],
                         echo_times_ms=[30.0, 45.0], grads=3, ctx=gpu_ctx, **kw)
    out = op.apply_host(None)
    op.close()
    args = (s["sim_dims"], s["acq_dims"], 2, s["images"], s["t2"], s["fmap"], acq)
    errs = {"kspace": rel_l2(out["kspace"], oracle.series_forward(*args, echo_times_ms=[30.0, 45.0], **kw))}
    adj = oracle.series_adjoint(*args, out["kspace"].astype(np.complex128), echo_times_ms=[30.0, 45.0], **kw)
    for key in ("comp_grad", "fmap_grad", "r2_grad"):
        errs[key] = rel_l2(out[key], adj[key])
    assert max(errs.values()) <= TOL, errs


def test_mixed_widths_and_the_segmented_switch(gpu_ctx):
    """Widths 32, 64 and 96 in one plan (per-width launches); and an operator on basis rows that goes
    to the segmented path and back gives its first k-space again, bit for bit."""
    acq = Acquisition(n_coils=16, t_line=0.5, t_echo=30.0)
    series, want = [], []
    for n in (16, 32, 48):
        s = cases.series_case(nx=n, ny=16, nz=2, nv=1, ncomp=2)
        series.append(dict(sim_dims=s["sim_dims"], acq_dims=s["acq_dims"], n_volumes=1, images=s["images"], t2=s["t2"],
                           fmap=s["fmap"], t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42))
        want.append(oracle.series_forward(s["sim_dims"], s["acq_dims"], 1, s["images"], s["t2"], s["fmap"], acq,
                                          echo_times_ms=[30.0], t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(),
                                          seed=42))
    b = api.EpiBatch(series, acq, echo_times_ms=[30.0], grads=0, ctx=gpu_ctx)
    b.forward()
    b.adjoint()
    for i, s in enumerate(series):
        got = b.download(i)
        assert rel_l2(got["kspace"], want[i]) <= TOL
        adj = oracle.series_adjoint(s["sim_dims"], s["acq_dims"], 1, s["images"], s["t2"], s["fmap"], acq,
                                    got["kspace"].astype(np.complex128), echo_times_ms=[30.0], t_inhom=s["t_inhom"],
                                    phase=s["phase"], seed=42)
        assert rel_l2(got["comp_grad"], adj["comp_grad"]) <= TOL
    b.close()
    s = series[1]
    op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 1, s["t2"], s["fmap"], acq, images=s["images"],
                         echo_times_ms=[30.0], t_inhom=s["t_inhom"], phase=s["phase"], seed=42, grads=0, ctx=gpu_ctx)
    first = op.apply_host(None)
    op.set_segmented("f16")
    seg = op.apply_host(None)
    assert op.segmented_status() == 0 and rel_l2(seg["kspace"], want[1]) <= TOL
    assert rel_l2(seg["comp_grad"], first["comp_grad"]) <= 2 * TOL
    op.set_segmented("exact")
    again = op.apply_host(None)
    op.close()
    assert np.array_equal(again["kspace"], first["kspace"]) and np.array_equal(again["comp_grad"], first["comp_grad"])
