"""The pair on a coil basis is no less exact than with a row per coil: the relative L2 errors of its k-space
and of its compartment gradients against the FP64 oracle, beside those of the same operator with per-coil
rows (the autotuner's "classes=0", from its cache file).  The bar is 2 % for the scatter of one series: the
two sums round independently, and 300,000 samples determine each error to well under that."""
from __future__ import annotations

import numpy as np
import pytest

from mrsim_acq_b200 import api
from mrsim_acq_b200.api import Acquisition, PhaseModel
from oracle import oracle
from tests import cases

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


@pytest.mark.parametrize("coils,n,nz", [(12, 64, 36)])
def test_basis_rows_against_coil_rows(gpu_ctx, tmp_path, coils, n, nz):
    s = cases.series_case(nx=n, ny=n, nz=nz, o=2, nv=1, ncomp=2)
    acq = Acquisition(n_coils=coils, t_line=0.5, t_echo=40.0, ghost_offset=0.02)
    kw = dict(t_inhom=s["t_inhom"], phase=PhaseModel.hbcd_like(), seed=42)
    op = api.EpiOperator(s["sim_dims"], s["acq_dims"], 1, s["t2"], s["fmap"], acq, images=s["images"],
                         echo_times_ms=[40.0], grads=0, ctx=gpu_ctx, **kw)
    basis = {k: v.copy() for k, v in op.apply_host(None).items() if v is not None}
    cache = tmp_path / "rows.txt"
    cache.write_text(f"epi snx{2 * n} sny{2 * n} nx{n} ny{n} coils{coils} comp2 lines{n} echoes1 maps0 grads00\t"
                     "classes=0 x=fft adjoint_rows=0 path=exact\n")
    assert op.tune(cache)["choice"].endswith("(cached)")
    rows = op.apply_host(None)
    op.close()
    assert not np.array_equal(rows["kspace"], basis["kspace"])
    args = (s["sim_dims"], s["acq_dims"], 1, s["images"], s["t2"], s["fmap"], acq)
    k = oracle.series_forward(*args, echo_times_ms=[40.0], **kw)
    cg = oracle.series_adjoint(*args, k, echo_times_ms=[40.0], **kw)["comp_grad"]
    for name, want in (("kspace", k), ("comp_grad", cg)):
        got, bar = rel_l2(basis[name], want), rel_l2(rows[name], want)
        print(name, f"basis {got:.3e}, per coil {bar:.3e}")
        assert got <= 1.02 * bar, name
