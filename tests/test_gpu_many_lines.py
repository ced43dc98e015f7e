"""Trains of many echoes: the staged y kernels hold a table of every acquired line in shared memory, and
a plan whose lines do not fit takes the general kernels.  Few pixels, line counts on both sides of each
coil form's limit (about 1,900 lines with three compartments), against the FP64 oracle (relative L2 <=
1e-5, the bar of every FP32 result)."""

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


# rows of 32 points take the warp FFT, of 20 and 15 the DFT GEMM (15: odd rows)
@pytest.mark.parametrize("coils,nx,echoes,ncomp,grads", [
    (12, 32, 14, 3, 3), (12, 32, 16, 3, 3), (12, 20, 16, 3, 1), (12, 15, 16, 3, 0), (32, 32, 16, 3, 0), (6, 32, 19, 2, 2),
    (12, 32, 17, 1, 0), (8, 32, 16, 3, 3), (8, 20, 17, 3, 0), (4, 32, 16, 3, 1), (1, 32, 16, 3, 0)])
def test_line_tables_past_shared_memory(gpu_ctx, coils, nx, echoes, ncomp, grads):
    ny = 128
    s = cases.series_case(nx=nx, ny=ny, nz=1, o=1, nv=1, ncomp=ncomp)
    acq = Acquisition(n_coils=coils, t_line=0.02, t_echo=3.0, ghost_offset=0.02)
    tes = [3.0 + 2.7 * e for e in range(echoes)]
    kw = dict(t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42)
    op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 1, s["t2"], s["fmap"], acq, images=s["images"],
                         echo_times_ms=tes, grads=grads, ctx=gpu_ctx, **kw)
    out = op.apply_host(None)
    op.close()
    args = (s["sim_dims"], s["acq_dims"], 1, s["images"], s["t2"], s["fmap"], acq)
    errs = {"kspace": rel_l2(out["kspace"], oracle.series_forward(*args, echo_times_ms=tes, **kw))}
    adj = oracle.series_adjoint(*args, out["kspace"].astype(np.complex128), echo_times_ms=tes, **kw)
    for key in ("comp_grad",) + (("fmap_grad",) if grads & 1 else ()) + (("r2_grad",) if grads & 2 else ()):
        errs[key] = rel_l2(out[key], adj[key])
    assert max(errs.values()) <= 1e-5, errs
