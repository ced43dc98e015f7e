"""Plans of few tiles, whose blocks share a tile in clusters (rows of the forward, lines of the
adjoint): against the FP64 oracle (relative L2 <= 1e-5, the bar of every FP32 result) for every coil
form (one to four coils, class rows, basis rows), one to four compartments, uneven shares of rows and
lines, partial tiles of columns and lines, and with and without the fieldmap and R2 gradients."""

import numpy as np
import pytest

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, PhaseModel
from oracle import oracle
from tests import cases

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    n = np.linalg.norm(np.ravel(b))
    return np.linalg.norm(np.ravel(a) - np.ravel(b)) / (n if n > 0 else 1.0)


@pytest.mark.parametrize("coils,nx,ny,o,ncomp,grads,accel", [
    (1, 64, 64, 2, 1, 0, 1), (1, 64, 64, 2, 3, 3, 1), (2, 32, 50, 2, 2, 1, 1), (4, 48, 33, 2, 3, 2, 1),
    (8, 64, 64, 2, 3, 3, 2), (8, 64, 37, 2, 1, 0, 1), (8, 96, 96, 2, 2, 3, 2), (16, 64, 64, 2, 3, 3, 1),
    (6, 32, 64, 1, 4, 0, 1), (32, 72, 40, 2, 2, 0, 3), (1, 100, 17, 2, 1, 3, 1), (4, 36, 128, 1, 1, 0, 1)])
def test_shared_tiles_match_the_oracle(gpu_ctx, coils, nx, ny, o, ncomp, grads, accel):
    s = cases.series_case(nx=nx, ny=ny, nz=1, o=o, nv=1, ncomp=min(ncomp, 3))
    for c in range(3, ncomp):
        for k in ("images", "t2", "t_inhom"):
            s[k] = list(s[k]) + [s[k][c % 3]]
    acq = Acquisition(n_coils=coils, accel=accel, t_line=0.5, t_echo=40.0, ghost_offset=0.02)
    kw = dict(t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42)
    op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 1, s["t2"], s["fmap"], acq, images=s["images"],
                         echo_times_ms=[40.0], grads=grads, ctx=gpu_ctx, **kw)
    out = op.apply_host(None)
    again = op.apply_host(None)
    op.close()
    args = (s["sim_dims"], s["acq_dims"], 1, s["images"], s["t2"], s["fmap"], acq)
    errs = {"kspace": rel_l2(out["kspace"], oracle.series_forward(*args, echo_times_ms=[40.0], **kw))}
    adj = oracle.series_adjoint(*args, out["kspace"].astype(np.complex128), echo_times_ms=[40.0], **kw)
    for key in ("comp_grad",) + (("fmap_grad",) if grads & 1 else ()) + (("r2_grad",) if grads & 2 else ()):
        errs[key] = rel_l2(out[key], adj[key])
        assert np.array_equal(out[key], again[key])
    assert max(errs.values()) <= 1e-5, errs
