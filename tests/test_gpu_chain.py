"""Small plans run as a chain of overlapping launches: the first step of a new operator (whose phase and
rows its own kernels write) and every later one give the same bits, forward and gradients, for each
coil form of the y kernels."""

import numpy as np
import pytest

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, PhaseModel
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coils,nx,ny,o,ncomp,nz", [(1, 64, 64, 2, 1, 1), (2, 32, 50, 2, 2, 1), (4, 48, 33, 2, 3, 1),
                                                    (8, 64, 64, 2, 3, 1), (16, 64, 64, 2, 3, 1), (8, 96, 96, 2, 2, 2),
                                                    (32, 72, 40, 2, 2, 1), (8, 64, 64, 2, 3, 12)])
def test_first_step_equals_later_ones(gpu_ctx, coils, nx, ny, o, ncomp, nz):
    s = cases.series_case(nx=nx, ny=ny, nz=nz, o=o, nv=1, ncomp=ncomp)
    acq = Acquisition(n_coils=coils, t_line=0.5, t_echo=40.0, ghost_offset=0.02)
    want = None
    for _ in range(4):  # new operators, whose buffers are other ones' old memory
        op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 1, s["t2"], s["fmap"], acq, images=s["images"],
                             echo_times_ms=[40.0], grads=3, t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42,
                             ctx=gpu_ctx)
        for _ in range(3):
            got = op.apply_host(None)
            want = want or {k: v.copy() for k, v in got.items()}
            for k, v in want.items():
                assert np.array_equal(got[k], v), k
        op.close()
