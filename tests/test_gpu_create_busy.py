"""Making an operator waits for no work but its own: with another stream busy for a second, operators of
every x-stage (warp FFT, and the DFT GEMM, whose tiles are made from the line table) are there before it
has ended, and so are a batch and a change of the plan."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, PhaseModel
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coils,nx", [(8, 32), (12, 25), (1, 25), (12, 32)])
def test_creation_beside_other_work(coils, nx):
    ctx = api.Context(0)
    s = cases.series_case(nx=nx, ny=20, nz=2, o=2, nv=1, ncomp=2)
    acq = Acquisition(n_coils=coils, t_line=0.5, t_echo=40.0)
    one = dict(sim_dims=s["sim_dims"], acq_dims=s["acq_dims"], n_volumes=1, images=s["images"], t2=s["t2"], fmap=s["fmap"],
               t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42)

    def make():
        op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 1, s["t2"], s["fmap"], acq, images=s["images"],
                             echo_times_ms=[40.0], t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42, grads=0,
                             ctx=ctx)
        return op, api.EpiBatch([one, one], acq, echo_times_ms=[40.0], grads=0, ctx=ctx)

    first = make()  # buffers and kernels are there
    want = first[0].apply_host(None)["kspace"].copy()
    torch.cuda.synchronize()
    busy, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(int(2e9))  # about a second of clock cycles
        done.record()
    second = make()
    free = not done.query()
    torch.cuda.synchronize()
    assert free
    assert np.array_equal(second[0].apply_host(None)["kspace"], want)
    for pair in (first, second):
        for o in pair:
            o.close()
    ctx.close()
