"""The work that programs built on this framework have it do, as timed cases.

Every case goes through a public entry point with the inputs, plans and handles that such a program
holds.  The kinds:

- "operator": one step of the forward / adjoint operator of a 2D EPI series with its images resident
  (`EpiOperator`), the k-space and every gradient left on the device: the inner loop of a fit;
- "batch": series of different geometries as one plan (`EpiBatch`), forward + adjoint, and the
  results brought to the host (the only way its interface gives them out);
- "slice": one slice through the host call `simulate_slice` (forward, window, inverse DFT, coil
  combine): the smallest thing the command line of the reference does;
- "series": `simulate_acquisition_complex`, the whole pipeline of a series on host arrays (forward,
  receiver noise, GRAPPA fit and fill, window, reconstruction);
- "grase": `simulate_acquisition_3d` with the GRASE train, one volume on host arrays;
- "spiral_forward": the certified time-segmented spiral forward of one coil of a slice;
- "spiral_volume": `simulate_acquisition_3d` with the stack of spirals (forward, noise, kz GRAPPA,
  POCS, gridding + CG reconstruction), one volume on host arrays;
- "spin": one volume's excitations of the spin history, terms left on the device.

The 3D entry points give magnitude and phase; their cases hand on the complex image, because the
phase of a voxel that holds only noise says nothing.

Sizes are those of this repository's benchmark, tests and configurations; `draw` spreads them over
the same ranges, odd and ragged ones among them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mrsim_acq_b200 import api
from mrsim_acq_b200 import kspace3d as K3
from mrsim_acq_b200 import spiral as S
from mrsim_acq_b200.api import T2, Acquisition, EchoFormation, KspaceWindow, PartialFourierMode, PhaseModel
from mrsim_acq_b200.motion import Pose
from mrsim_acq_b200.spin_history import Recovery, Shot, Slabs, Source, SpinHistory

TAU = 2.0 * math.pi
T2_MS = (80.0, 250.0, 30.0)
TI_MS = (40.0, 60.0, 20.0)
T1_MS = (1330.0, 4000.0, 900.0)
BACKGROUND = (0.0, 0.13, 0.10, 0.02, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)  # PhaseModel.hbcd_like's


def listed():
    op = dict(kind="operator", nx=64, ny=64, o=2, nz=1, nv=1, ncomp=1, coils=1, accel=1, pf=1.0, echoes="30",
              t_line=0.5, grads=0, maps=False, gradient=False, ghost=0.0, eddy=False, step="pair")
    return [
        # the plain single-shot slice: five launches of a few microseconds, where latency counts
        dict(op, name="single-shot"),
        # one step of a fieldmap fit (the differentiation workload): a new fieldmap from the host,
        # the forward, and every VJP; 192-point rows, a short last wave
        dict(op, name="fieldmap-fit-step", nx=96, ny=96, nz=16, ncomp=2, coils=8, accel=2, pf=0.75, grads=3,
             step="fieldmap"),
        # the benchmark series: 30 slices x 40 volumes x 3 echoes, 8 coils, R = 2, partial Fourier 6/8
        dict(op, name="series-operator", nz=30, nv=40, ncomp=3, coils=8, accel=2, pf=0.75, echoes="15,35,55", grads=3,
             ghost=0.05),
        # precision at scale: 128 x 128 on 256 x 256, 32 coils, every line
        dict(op, name="scale-32-coils", nx=128, ny=128, nz=60, nv=2, ncomp=3, coils=32, echoes="40", ghost=0.05),
        # a ragged gradient-echo series with voxel T2 maps, eddy currents, 12 coils and rows that are
        # no multiple of a warp
        dict(op, name="ragged-maps-12-coils", nx=75, ny=90, nz=5, nv=3, ncomp=2, coils=12, echoes="42", grads=3,
             maps=True, gradient=True, eddy=True, ghost=0.02),
        # three geometries as one plan, 32 coils
        dict(kind="batch", name="mixed-batch", n="64,96,128", nz="17,23,31", o=2, ncomp=3, coils=32, te=40.0),
        # one slice, host arrays in and out
        dict(kind="slice", name="slice-host-call", nx=64, ny=64, o=2, coils=8, ncomp=3),
        # a short series through the whole pipeline
        dict(kind="series", name="series-pipeline", n=64, o=2, nz=30, nv=20, ncomp=3, coils=8, accel=2, pf=0.75, te=30.0),
        # one GRASE volume: 4 shots, 150-degree refocusing, 32 coils
        dict(kind="grase", name="grase-volume", n=64, o=2, nz=32, shots=4, coils=32, ncomp=3, refocusing=150.0),
        # the in-plane spiral forward of one coil: 32 interleaves x 2048 samples
        dict(kind="spiral_forward", name="spiral-slice", n=64, o=2, interleaves=32, readout=8.192, fieldmap=80.0),
        # one stack-of-spirals volume with its reconstruction: 16 coils in 2 rings, kz 6/8, R = 2
        dict(kind="spiral_volume", name="spiral-volume", n=64, o=2, nz=48, interleaves=32, readout=8.192, coils=16,
             rows=2, kz_pf=0.75, kz_accel=2, fieldmap=80.0),
        # one volume (20 single-slice shots) of the spin history at the reference's motivating size
        dict(kind="spin", name="spin-history-volume", nx=197, ny=233, nz=100, every=3, sx=128, sy=136, slices=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator"] * 6 + ["batch", "slice", "series", "grase", "spiral_forward", "spiral_volume", "spin"])
    if kind == "operator":
        coils = rng.choice([1, 2, 3, 4, 6, 8, 8, 12, 16, 24, 32])
        o = rng.choice([1, 2, 2, 2, 3])
        nx = rng.choice([32, 48, 64, 64, 80, 96, 128, rng.randint(24, 128)])
        ny = rng.choice([nx, nx, rng.randint(24, 128)])
        nx = min(nx, 256 // o)
        units = min(_log_int(rng, 1, 600), max(1, int(6e9 / (o * o * nx * ny * ny * max(coils, 8)))))
        nz = rng.randint(1, max(1, min(units, 60)))
        n_echoes = rng.choice([1, 1, 2, 3])
        base = rng.uniform(0.0, 10.0) + 0.25 * ny + 2.0
        tes = ",".join("%.1f" % (base + 15.0 * e) for e in range(n_echoes))
        return dict(kind="operator", nx=nx, ny=ny, o=o, nz=nz, nv=max(1, units // nz), ncomp=rng.randint(1, 3),
                    coils=coils, accel=rng.choice([1, 1, 2, 3]), pf=rng.choice([1.0, 1.0, 0.75]), echoes=tes, t_line=0.5,
                    grads=rng.choice([0, 0, 1, 3]), maps=rng.random() < 0.25, gradient=rng.random() < 0.25,
                    ghost=rng.choice([0.0, 0.05]), eddy=rng.random() < 0.25, step=rng.choice(["pair", "pair", "fieldmap"]))
    if kind == "batch":
        k = rng.randint(2, 3)
        ns = [rng.choice([32, 48, 64, 96, rng.randint(24, 96)]) for _ in range(k)]
        return dict(kind=kind, n=",".join(map(str, ns)), nz=",".join(str(rng.randint(1, 30)) for _ in ns), o=2,
                    ncomp=rng.randint(1, 3), coils=rng.choice([4, 8, 16, 32]), te=rng.uniform(30.0, 60.0))
    if kind == "slice":
        nx = rng.choice([32, 64, 96, rng.randint(16, 128)])
        return dict(kind=kind, nx=nx, ny=rng.choice([nx, rng.randint(16, 128)]), o=rng.choice([1, 2, 2]),
                    coils=rng.choice([1, 3, 4, 8, 16, 32]), ncomp=rng.randint(1, 3))
    if kind == "series":
        return dict(kind=kind, n=rng.choice([32, 48, 64, rng.randint(24, 64)]), o=2, nz=rng.randint(1, 30),
                    nv=rng.randint(1, 20), ncomp=rng.randint(1, 3), coils=rng.choice([4, 8, 16]), accel=rng.choice([1, 2]),
                    pf=rng.choice([1.0, 0.75]), te=rng.uniform(25.0, 50.0))
    if kind == "grase":
        return dict(kind=kind, n=rng.choice([32, 48, 64]), o=rng.choice([1, 2]), nz=rng.randint(8, 32),
                    shots=rng.choice([2, 4]), coils=rng.choice([4, 8, 16, 32]), ncomp=rng.randint(1, 3),
                    refocusing=rng.choice([150.0, 180.0]))
    if kind == "spiral_forward":
        return dict(kind=kind, n=rng.choice([32, 48, 64]), o=rng.choice([1, 2]), interleaves=rng.choice([16, 24, 32]),
                    readout=rng.choice([4.096, 8.192]), fieldmap=rng.uniform(20.0, 100.0))
    if kind == "spiral_volume":
        return dict(kind=kind, n=rng.choice([32, 48]), o=2, nz=rng.choice([8, 12, 16]), interleaves=rng.choice([16, 24]),
                    readout=8.192, coils=rng.choice([4, 8]), rows=rng.choice([1, 2]), kz_pf=1.0, kz_accel=1,
                    fieldmap=rng.uniform(20.0, 80.0))
    return dict(kind=kind, nx=rng.randint(60, 197), ny=rng.randint(60, 233), nz=rng.randint(20, 100),
                every=rng.randint(1, 6), sx=rng.randint(48, 128), sy=rng.randint(48, 136), slices=rng.randint(4, 20))


# ---- inputs -----------------------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _phantom(seed, snx, sny, nz, nv, ncomp):
    """Ten ellipses split over the compartments, each volume moved rigidly by up to 2 degrees and
    2 mm: float32 host arrays in the layout (x + snx (y + sny z)) nv + g, one per compartment."""
    rng = np.random.default_rng(seed)
    dev = _device()
    ell = [(rng.uniform(0.3, 0.7), rng.uniform(0.3, 0.7), rng.uniform(0.08, 0.3), rng.uniform(0.08, 0.3),
            rng.uniform(0.0, math.pi), rng.uniform(0.2, 1.0)) for _ in range(10)]
    g = torch.as_tensor(rng.uniform(-1.0, 1.0, (3, nv)), device=dev, dtype=torch.float32)
    rot, tx, ty = g[0] * math.radians(2.0), g[1] * 0.01, g[2] * 0.01
    x = ((torch.arange(snx, device=dev) + 0.5) / snx).view(1, snx, 1)
    y = ((torch.arange(sny, device=dev) + 0.5) / sny).view(sny, 1, 1)
    X = torch.cos(rot) * (x - 0.5) - torch.sin(rot) * (y - 0.5) + 0.5 - tx
    Y = torch.sin(rot) * (x - 0.5) + torch.cos(rot) * (y - 0.5) + 0.5 - ty
    imgs = [torch.zeros((nz, sny, snx, nv), device=dev) for _ in range(ncomp)]
    for k, (cx, cy, a, b, th, mag) in enumerate(ell):
        c, s = math.cos(th), math.sin(th)
        u, v = (c * (X - cx) + s * (Y - cy)) / a, (-s * (X - cx) + c * (Y - cy)) / b
        r2 = u * u + v * v
        for z in range(nz):
            scale = 1.0 - ((z + 0.5 - nz / 2) / nz / 0.6) ** 2
            imgs[k % ncomp][z] += mag * torch.clamp((scale - r2) * 8.0, 0.0, 1.0)
    return [im.reshape(-1).cpu().numpy() for im in imgs]


def _fieldmap(seed, snx, sny, nz, hz=60.0):
    rng = np.random.default_rng(seed + 7919)
    x, y = ((np.arange(n) + 0.5) / n for n in (snx, sny))
    z = (np.arange(nz) + 0.5) / nz
    f = np.zeros((nz, sny, snx))
    for _ in range(3):
        a, w = rng.uniform(-hz, hz), rng.uniform(0.06, 0.16)
        cx, cy, cz = rng.uniform(0.3, 0.7), rng.uniform(0.3, 0.7), rng.uniform(0.2, 0.8)
        f += a * (np.exp(-((z - cz) / 0.5) ** 2)[:, None, None] * np.exp(-((y - cy) / w) ** 2 / 2)[None, :, None]
                  * np.exp(-((x - cx) / w) ** 2 / 2)[None, None, :])
    return np.clip(f, -hz, hz).astype(np.float32).reshape(-1)


def _t2_map(snx, sny, nz):
    x = (np.arange(snx) + 0.5) / snx
    return np.broadcast_to((60.0 + 40.0 * x).astype(np.float32), (nz, sny, snx)).reshape(-1).copy()


def _tes(case):
    return [float(t) for t in str(case["echoes"]).split(",")]


def _eddy_drive(seed, nv):
    rng = np.random.default_rng(seed + 31)
    d = rng.normal(size=(nv, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return [tuple(float(v) for v in row) for row in d]


class _Buffer:
    """A device buffer of an operator as an array interface; keeps the operator alive."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": kind, "data": (ptr, False), "version": 2,
                                         "strides": None}


def _operator_inputs(case, seed):
    nx, ny, o, nz, nv, nc = (int(case[k]) for k in ("nx", "ny", "o", "nz", "nv", "ncomp"))
    snx, sny = nx * o, ny * o
    t2 = [T2.uniform(v) for v in T2_MS[:nc]]
    if case["maps"]:
        t2[0] = T2.of_map(_t2_map(snx, sny, nz))
    acq = Acquisition(n_coils=int(case["coils"]), accel=int(case["accel"]), partial_fourier=float(case["pf"]),
                      pf_mode=PartialFourierMode.Scanner, t_line=float(case["t_line"]), t_echo=_tes(case)[0],
                      ghost_offset=float(case["ghost"]), signal_scale=100.0,
                      echo=EchoFormation.Gradient if case["gradient"] else EchoFormation.Spin)
    drive = None
    if case["eddy"]:
        acq = acq.replace(eddy_strength=3.0, eddy_quad=0.02, eddy_tau=70.0)
        drive = _eddy_drive(seed, nv)
    return dict(sim=(snx, sny, nz), mat=(nx, ny, nz), nv=nv, t2=t2, ti=[T2.uniform(v) for v in TI_MS[:nc]],
                images=_phantom(seed, snx, sny, nz, nv, nc), fmap=_fieldmap(seed, snx, sny, nz), acq=acq, drive=drive)


def _batch_inputs(case, seed):
    series = []
    for i, (n, nz) in enumerate(zip(str(case["n"]).split(","), str(case["nz"]).split(","))):
        n, nz, sn = int(n), int(nz), int(n) * int(case["o"])
        nc = int(case["ncomp"])
        series.append(dict(sim_dims=(sn, sn, nz), acq_dims=(n, n, nz), n_volumes=1,
                           images=_phantom(seed + 100 * i, sn, sn, nz, 1, nc), fmap=_fieldmap(seed + 100 * i, sn, sn, nz),
                           t2=[T2.uniform(v) for v in T2_MS[:nc]], t_inhom=[T2.uniform(v) for v in TI_MS[:nc]],
                           phase=PhaseModel.hbcd_like(), seed=42))
    acq = Acquisition(n_coils=int(case["coils"]), t_line=0.5, t_echo=float(case["te"]), ghost_offset=0.05,
                      signal_scale=100.0)
    return series, acq


def _slice_inputs(case, seed):
    nx, ny, o, nc = (int(case[k]) for k in ("nx", "ny", "o", "ncomp"))
    snx, sny = nx * o, ny * o
    y, x = np.meshgrid((np.arange(sny) + 0.5) / sny, (np.arange(snx) + 0.5) / snx, indexing="ij")
    inp = api.SliceInput(compartments=_phantom(seed, snx, sny, 1, 1, nc), t2=[T2.uniform(v) for v in T2_MS[:nc]],
                         t_inhom=[T2.uniform(v) for v in TI_MS[:nc]], fmap=_fieldmap(seed, snx, sny, 1), sim=(snx, sny),
                         acq_matrix=(nx, ny), phase0=(0.4 * x - 0.7 * y * y).ravel())
    acq = Acquisition(n_coils=int(case["coils"]), t_line=0.5, t_echo=0.25 * ny + 12.0, ghost_offset=0.02,
                      signal_scale=100.0, window=KspaceWindow.hann())
    return inp, acq


def _spiral_slice_inputs(case, seed):
    n, o = int(case["n"]), int(case["o"])
    sn = n * o
    tr = S.spiral_trajectory(n, n, int(case["interleaves"]), float(case["readout"]), 0.004, 1.2)
    k = tr.k.reshape(-1, 2)
    y, x = np.meshgrid((np.arange(sn) + 0.5) / sn, (np.arange(sn) + 0.5) / sn, indexing="ij")
    inp = api.SliceInput(compartments=_phantom(seed, sn, sn, 1, 1, 1), t2=[T2.uniform(80.0)],
                         t_inhom=[T2.uniform(40.0)], fmap=_fieldmap(seed, sn, sn, 1, float(case["fieldmap"])), sim=(sn, sn),
                         acq_matrix=(n, n), phase0=(0.4 * x - 0.7 * y * y).ravel())
    acq = Acquisition(n_coils=8, signal_scale=1.0)
    hz = float(case["fieldmap"])
    return inp, acq, tr, k, np.arange(len(k)) % len(tr.tau_ms), S.RateRect((0.0, 0.0), (-hz, hz))


def _kz_read(nz, pf, accel):
    lo = nz - min(nz, int(round(nz * pf)))
    return sum(1 for p in range(nz) if p >= lo and (p - nz // 2) % accel == 0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "operator":
        i = _operator_inputs(case, seed)
        op = api.EpiOperator(i["sim"], i["mat"], i["nv"], i["t2"], i["fmap"], i["acq"], images=i["images"],
                             echo_times_ms=_tes(case), t_inhom=i["ti"], phase=PhaseModel.hbcd_like(), seed=42,
                             eddy_drive=i["drive"], grads=int(case["grads"]))
        ptr, shp, outs = op.buffers(), op.shapes(), {}
        for name in ("kspace", "comp_grad", "fmap_grad", "r2_grad"):
            if ptr[name]:
                b = _Buffer(op, ptr[name], shp[name], "<f4" if name in ("fmap_grad", "r2_grad") else "<c8")
                outs[name] = torch.as_tensor(b, device="cuda")
        return dict(kind=kind, op=op, outs=outs, fmap=i["fmap"] if case["step"] == "fieldmap" else None)
    if kind == "batch":
        series, acq = _batch_inputs(case, seed)
        return dict(kind=kind, batch=api.EpiBatch(series, acq, echo_times_ms=[float(case["te"])], grads=0), n=len(series))
    if kind == "slice":
        inp, acq = _slice_inputs(case, seed)
        return dict(kind=kind, inp=inp, acq=acq)
    if kind == "series":
        n, o, nz, nv, nc = (int(case[k]) for k in ("n", "o", "nz", "nv", "ncomp"))
        sn = n * o
        inp = api.AcquisitionInput((sn, sn, nz), (n, n, nz), nv, _phantom(seed, sn, sn, nz, nv, nc),
                                   [T2.uniform(v) for v in T2_MS[:nc]], _fieldmap(seed, sn, sn, nz), t_inhom=[T2.uniform(v) for v in TI_MS[:nc]],
                                   phase=PhaseModel.hbcd_like(), seed=9)
        acq = Acquisition(n_coils=int(case["coils"]), accel=int(case["accel"]), acs_lines=24,
                          partial_fourier=float(case["pf"]), pf_mode=PartialFourierMode.Scanner, t_line=0.5,
                          t_echo=float(case["te"]), ghost_offset=0.05, window=KspaceWindow.hann(), signal_scale=100.0,
                          noise_variance=1.56)
        return dict(kind=kind, inp=inp, acq=acq)
    if kind == "grase":
        n, o, nz, nc = (int(case[k]) for k in ("n", "o", "nz", "ncomp"))
        sn = n * o
        acq = Acquisition(n_coils=int(case["coils"]), signal_scale=100.0, noise_variance=1e-4)
        train = K3.EchoTrain(etl=nz, esp_ms=20.0, refocusing_deg=float(case["refocusing"]), kz_order=K3.KzOrder.Centric,
                             kz_segments=1, refocusing_time_ms=2.0)
        args = ((sn, sn, nz), (n, n, nz), 1, _phantom(seed, sn, sn, nz, 1, nc), [T2.uniform(v) for v in T2_MS[:nc]],
                [T2.uniform(v) for v in T1_MS[:nc]], _fieldmap(seed, sn, sn, nz, 40.0), None, acq, train,
                K3.GraseReadout(ky_segments=int(case["shots"]), t_line_ms=0.5, reverse_phase=False))
        return dict(kind=kind, args=args, kw=dict(phase=PhaseModel.none(), seed=5))
    if kind == "spiral_forward":
        inp, acq, tr, k, idx, rect = _spiral_slice_inputs(case, seed)
        return dict(kind=kind, args=(inp, acq, 0, 8, k, idx, tr.tau_ms, float(case["readout"]), rect, None, False))
    if kind == "spiral_volume":
        n, o, nz = (int(case[k]) for k in ("n", "o", "nz"))
        sn = n * o
        kz = K3.KzSampling(float(case["kz_pf"]), int(case["kz_accel"]))
        train = K3.EchoTrain(etl=_kz_read(nz, kz.partial_fourier, kz.accel), esp_ms=12.0, refocusing_deg=180.0,
                             kz_order=K3.KzOrder.Centric, kz_segments=1)
        images = _phantom(seed, sn, sn, nz, 1, 1)
        acq = Acquisition(n_coils=int(case["coils"]), signal_scale=100.0, noise_variance=1e-4)
        opts = K3.KzOptions(coil_rows=int(case["rows"]))
        if kz.accel > 1:
            opts = K3.KzOptions(coil_rows=int(case["rows"]), calibration_images=images, calibration_seed=3, pocs=True)
        # one in-plane field for every slice, as the benchmark's volume has it
        field = np.tile(_fieldmap(seed, sn, sn, 1, float(case["fieldmap"])), nz)
        args = ((sn, sn, nz), (n, n, nz), 1, images, [T2.uniform(80.0)], [T2.uniform(1300.0)], field, None, acq, train,
                K3.SpiralReadout(int(case["interleaves"]), float(case["readout"]), 0.004, 1.2, kz))
        return dict(kind=kind, args=args, kw=dict(seed=5, kz_opts=opts))
    nx, ny, nz = (int(case[k]) for k in ("nx", "ny", "nz"))
    rng = np.random.default_rng(seed)
    nvox = nx * ny * nz
    cls = np.full(nvox, 255, np.uint8)
    cls[rng.integers(0, int(case["every"]))::int(case["every"])] = 0
    src = Source((nx, ny, nz), np.eye(4), rng.uniform(0.8, 1.6, nvox).astype(np.float32),
                 rng.uniform(0.2, 1.0, nvox).astype(np.float32), cls, 1)
    aff = np.eye(4)
    ns = int(case["slices"])
    aff[0, 0], aff[1, 1], aff[2, 2] = nx / int(case["sx"]), ny / int(case["sy"]), nz / ns
    aff[2, 3] = (nz / ns - 1.0) / 2.0
    hist = SpinHistory(src, Slabs((int(case["sx"]), int(case["sy"]), ns), aff))
    centre, ph = (nx / 2.0, ny / 2.0, nz / 2.0), rng.uniform(0.0, TAU)
    # the head's slow drift over the session, as a motion trace of 64 volumes gives it
    trace = [Pose((0.5, 0.0, 0.3), (0.0, 0.0, 0.5 * math.sin(TAU * v / 64.0 + ph))).to_matrix(centre) for v in range(64)]
    out = torch.zeros(ns * 2 * int(case["sx"]) * int(case["sy"]), device="cuda")
    return dict(kind=kind, hist=hist, trace=trace, out=out, volume=0, slices=ns)


def run(state):
    kind = state["kind"]
    if kind == "operator":
        if state["fmap"] is not None:
            state["op"].set_fieldmap(state["fmap"])
        state["op"].forward()
        state["op"].adjoint()
        return state["outs"]
    if kind == "batch":
        state["batch"].forward()
        state["batch"].adjoint()
        return [state["batch"].download(i) for i in range(state["n"])]
    if kind == "slice":
        return api.simulate_slice(state["inp"], state["acq"])
    if kind == "series":
        return api.simulate_acquisition_complex(state["inp"], state["acq"])
    if kind in ("grase", "spiral_volume"):
        mag, ph = K3.simulate_acquisition_3d(*state["args"], **state["kw"])
        img = np.empty(mag.size, np.complex64)
        np.multiply(mag, np.cos(ph), out=img.real)
        np.multiply(mag, np.sin(ph), out=img.imag)
        return img
    if kind == "spiral_forward":
        return S.spiral_segmented_forward(*state["args"])[0]
    v, n = state["volume"], state["slices"]
    state["volume"] = v + 1
    m = state["trace"][v % len(state["trace"])]
    shots = [Shot(v * 4.6 + 3.6 + 0.04 * k, m, [k], Recovery(4.6)) for k in range(n)]
    state["hist"].excite_device(shots, state["out"].data_ptr())
    return state["out"]


# ---- the least a pass can do -------------------------------------------------------------------------
def _acquired(ny, accel, pf):
    """The lines read: Scanner partial Fourier keeps the first round(ny pf), every accel-th of them."""
    keep = ny if pf >= 1.0 else int(math.floor(ny * pf + 0.5))
    return [k for k in range(ny) if k < keep and (accel <= 1 or k % accel == (ny // 2) % accel)]


def _pair_work(units, snx, sny, nx, lines, ncomp, coils, grads):
    """Forward + adjoint of `lines` lines: each plane read once, each output written once; the sums
    over the rows per coil (a real weight times a complex value, added), the weights, phases and
    gradient sums per voxel and line, and an FFT per row and direction."""
    vox = snx * sny
    g = (1 if grads & 1 else 0) + (ncomp if grads & 2 else 0)
    nbytes = units * (vox * 4 * (2 * ncomp + 2) + 2 * 8 * coils * lines * nx + vox * (8 * ncomp + 4 * g))
    per = 2 * (4 * coils + 8) + 6 * ncomp + 4 * g
    return nbytes, units * (vox * lines * per + 2 * coils * lines * 5 * snx * math.log2(max(snx, 2)))


def work(case):
    kind = case["kind"]
    if kind == "operator":
        nx, ny, o = (int(case[k]) for k in ("nx", "ny", "o"))
        lines = len(_acquired(ny, int(case["accel"]), float(case["pf"]))) * len(_tes(case))
        b, f = _pair_work(int(case["nz"]) * int(case["nv"]), nx * o, ny * o, nx, lines, int(case["ncomp"]),
                          int(case["coils"]), int(case["grads"]))
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0
        for n, nz in zip(str(case["n"]).split(","), str(case["nz"]).split(",")):
            n, o = int(n), int(case["o"])
            w = _pair_work(int(nz), n * o, n * o, n, n, int(case["ncomp"]), int(case["coils"]), 0)
            b, f = b + w[0], f + w[1]
        return {"bytes": b, "flops": f}
    if kind == "slice":
        nx, ny, o, nc, q = (int(case[k]) for k in ("nx", "ny", "o", "ncomp", "coils"))
        vox = nx * ny * o * o
        fft = q * (ny * 5 * nx * o * math.log2(nx * o) + 10 * nx * ny * math.log2(nx * ny) / 2)
        return {"bytes": 4 * vox * (nc + 3) + 8 * nx * ny, "flops": vox * ny * (4 * q + 8 + 2 * nc) + fft}
    if kind in ("series", "grase"):
        n, o, nz, nc, q = (int(case[k]) for k in ("n", "o", "nz", "ncomp", "coils"))
        lines = n if kind == "grase" else len(_acquired(n, int(case["accel"]), float(case["pf"])))
        images = int(case["nv"]) if kind == "series" else 1
        echoes = 1 if kind == "series" else nc  # GRASE: one forward per compartment
        vox = n * n * o * o * nz * images
        fft = q * nz * images * echoes * 10 * n * n * math.log2(n * o)
        return {"bytes": 4 * vox * nc + 8 * n * n * nz * images,
                "flops": vox * lines * echoes * (4 * q + 8 + 2 * nc) + fft}
    if kind in ("spiral_forward", "spiral_volume"):
        n, o, il = (int(case[k]) for k in ("n", "o", "interleaves"))
        nz, q = (int(case["nz"]), int(case["coils"])) if kind == "spiral_volume" else (1, 1)
        samples = il * int(math.floor(float(case["readout"]) / 0.004 * (1 + 1e-12)))
        grid = (2 * n * o) ** 2
        # at least one gridding of every coil's slice images onto the samples
        flops = q * nz * (5 * grid * math.log2(grid) + samples * 64 * 4)
        return {"bytes": 4 * n * n * o * o * nz * 2 + 8 * (samples if kind == "spiral_forward" else n * n * nz),
                "flops": flops}
    tracked = int(case["nx"]) * int(case["ny"]) * int(case["nz"]) // int(case["every"])
    cells = int(case["sx"]) * int(case["sy"]) * int(case["slices"])
    # every tracked voxel's state (two pieces of it at the least) read and written, the terms written
    return {"bytes": tracked * (2 * 2 * 16 + 12) + cells * 8, "flops": tracked * 60}


# ---- the same values in 64 bits ------------------------------------------------------------------------
def _line_times(nx, ny, t_line, te):
    """Per PE line the echo-relative time of its centre sample and its time from excitation (ms): a
    snake from the last line down, odd lines read backwards."""
    ky = np.arange(ny)
    pos = np.where(ky % 2 == 1, nx - nx // 2 - 1, nx // 2)
    t = t_line / nx * ((ny - 1 - ky) * nx + pos + 0.5) - ny * t_line / 2.0
    return t, te + t


def _coil_amp(q, nc, xa, ya, nx, ny):
    if nc <= 1:
        return np.ones((len(ya), len(xa)))
    big = float(max(nx, ny))
    ang = TAU * q / nc
    px, py = nx / 2.0 + 0.6 * big * math.cos(ang), ny / 2.0 + 0.6 * big * math.sin(ang)
    return np.exp(-((xa[None, :] - px) ** 2 + (ya[:, None] - py) ** 2) / (2.0 * (0.9 * big) ** 2)) + 0.15


def _exact_epi(images, fmap, t2, ti, phases, tes, nx, ny, o, coils, accel, pf, t_line, gradient, ghost, scale, grads=0,
               eddy=None, t2_map=None, adjoint=True):
    """The EPI sums and their Hermitian transpose / gradients, unit by unit.  images [units][comp][sny]
    [snx], fmap and phases (radians) [units][sny][snx], eddy [units] (cx, qx, cy, qy, z) or None."""
    dev = images.device
    D, Z = torch.float64, torch.complex128
    units, nc, sny, snx = images.shape
    kys = _acquired(ny, accel, pf)
    skipped = (ny - min(ny, int(math.floor(ny * pf + 0.5)))) if pf < 1.0 else 0
    off = (o - 1.0) / 2.0
    xc, yc = np.arange(snx) - o * (nx // 2) - off, np.arange(sny) - o * (ny // 2) - off
    amp = torch.as_tensor(np.stack([_coil_amp(q, coils, (np.arange(snx) - off) / o, (np.arange(sny) - off) / o, nx, ny)
                                    for q in range(coils)]), device=dev).to(Z)  # [q][y][x]
    ampx = amp.permute(2, 0, 1).contiguous()
    tt, trf, rows, inh, dec, twx = [], [], [], [], [], []
    dft = np.exp(1j * TAU * np.outer(xc, np.arange(nx) - nx // 2) / snx)
    tw = [torch.as_tensor(dft * np.exp(1j * TAU * sg * ghost * xc / snx)[:, None], device=dev) for sg in (1.0, -1.0)]
    for e, te in enumerate(tes):
        t_ms, r_ms = _line_times(nx, ny, t_line, te)
        for k in kys:
            tt.append((t_ms[k] + te) / 1e3 if gradient else t_ms[k] / 1e3)
            trf.append(r_ms[k])
            inh.append(r_ms[k] if gradient else abs(t_ms[k]))
            read = t_ms[k] + ny * t_line / 2.0 - skipped * t_line
            dec.append(math.exp(-read / 70.0) * t_ms[k] / 1e3)
            rows.append(e * ny + k)
            twx.append(k % 2)
    J = len(rows)
    tt, trf, inh, dec = (torch.as_tensor(np.array(v, np.float64), device=dev) for v in (tt, trf, inh, dec))
    ky = torch.as_tensor([r % ny for r in rows], device=dev, dtype=D)
    ytab = (ky[:, None] - ny // 2) * torch.as_tensor(yc, device=dev)[None, :] / sny  # [j][y]
    even = torch.as_tensor([i for i in range(J) if twx[i] == 0], device=dev)
    odd = torch.as_tensor([i for i in range(J) if twx[i] == 1], device=dev)
    rows_t = torch.as_tensor(rows, device=dev)
    n_rows = len(tes) * ny
    ks = torch.zeros((units, coils, n_rows, nx), dtype=Z, device=dev)
    cg = torch.zeros((units, nc, sny, snx), dtype=Z, device=dev) if adjoint else None
    fg = torch.zeros((units, sny, snx), dtype=D, device=dev) if grads & 1 else None
    rg = torch.zeros((units, nc, sny, snx), dtype=D, device=dev) if grads & 2 else None
    t2s = [torch.as_tensor(v, dtype=D, device=dev) for v in t2]
    xo, yo = (torch.as_tensor(v / o, device=dev) for v in (xc, yc))
    for u in range(units):
        turns = (phases[u] / TAU)[None] + fmap[u].to(D)[None] * tt[:, None, None] + ytab[:, :, None]
        ex = None
        if eddy is not None:
            cx, qx, cy, qy, cz = eddy[u]
            turns = turns + ((cy * yo + qy * yo * yo)[None, :] * dec[:, None])[:, :, None]
            ex = torch.exp(1j * TAU * (cx * xo + qx * xo * xo + cz)[None, :] * dec[:, None])  # [j][x]
        P = torch.polar(torch.ones_like(turns), TAU * (turns - torch.round(turns)))
        rel = []
        for c in range(nc):
            tc = t2_map[u].to(D) if (t2_map is not None and c == 0) else t2s[c]
            rel.append(torch.exp(-trf[:, None, None] / tc - inh[:, None, None] / float(ti[c])))
        W = sum(rel[c] * images[u, c].to(D)[None] for c in range(nc))
        g = scale * torch.matmul(ampx, (W * P).permute(2, 1, 0))  # [x][q][j]
        if ex is not None:
            g = g * ex.t()[:, None, :]
        k = torch.zeros((coils, J, nx), dtype=Z, device=dev)
        for sel, t in ((even, tw[0]), (odd, tw[1])):
            if len(sel):
                k[:, sel] = torch.einsum("xqj,xk->qjk", g[:, :, sel], t) / (snx * sny)
        ks[u][:, rows_t] = k
        if not adjoint:
            continue
        h = torch.zeros((snx, coils, J), dtype=Z, device=dev)
        for sel, t in ((even, tw[0]), (odd, tw[1])):
            if len(sel):
                h[:, :, sel] = torch.einsum("qjk,xk->xqj", k[:, sel], t.conj()) / (snx * sny)
        if ex is not None:
            h = h * ex.t().conj()[:, None, :]
        H = scale * torch.matmul(ampx.transpose(1, 2), h).permute(2, 1, 0)  # [j][y][x]
        H = P.conj() * H
        for c in range(nc):
            V = rel[c] * H
            cg[u, c] = V.sum(0)
            m = images[u, c].to(D)
            if fg is not None:
                fg[u] += 2.0 * TAU * m * (tt[:, None, None] * V.imag).sum(0)
            if rg is not None:
                rg[u, c] = -2.0 * m * (trf[:, None, None] * V.real).sum(0)
    return ks, cg, fg, rg


def _units(images, snx, sny, nz, nv, dev):
    """Host arrays [comp] of (vox, g) as [g z][comp][y][x] on the device."""
    im = torch.stack([torch.as_tensor(a).to(dev).reshape(nz, sny, snx, nv) for a in images])
    return im.permute(4, 1, 0, 2, 3).reshape(nv * nz, len(images), sny, snx)


def _background(snx, sny, nz, nv, o, dev):
    off = (o - 1.0) / 2.0
    r0 = torch.as_tensor((np.arange(snx) - snx / 2.0 - off) / o, device=dev)
    r1 = torch.as_tensor((np.arange(sny) - sny / 2.0 - off) / o, device=dev)
    r2 = torch.as_tensor(np.arange(nz) - nz / 2.0, device=dev)
    p = BACKGROUND[1] * r0[None, None, :] + BACKGROUND[2] * r1[None, :, None] + BACKGROUND[3] * r2[:, None, None]
    return p[None].expand(nv, nz, sny, snx).reshape(nv * nz, sny, snx)


def exact(case, seed):
    kind, dev = case["kind"], _device()
    if kind == "operator":
        i = _operator_inputs(case, seed)
        snx, sny, nz = i["sim"]
        nx, ny, _ = i["mat"]
        nv, o = i["nv"], int(case["o"])
        fm = torch.as_tensor(i["fmap"]).to(dev).reshape(1, nz, sny, snx).expand(nv, nz, sny, snx).reshape(-1, sny, snx)
        eddy = None
        if i["drive"] is not None:
            eddy = []
            for d in i["drive"]:
                for z in range(nz):
                    zc = float(z - nz // 2)
                    eddy.append((3.0 * d[0], 0.02 * d[0], 3.0 * d[1], 0.02 * d[1], 3.0 * d[2] * zc + 0.02 * d[2] * zc * zc))
        maps = None
        if case["maps"]:
            maps = torch.as_tensor(_t2_map(snx, sny, nz)).to(dev).reshape(1, nz, sny, snx)
            maps = maps.expand(nv, nz, sny, snx).reshape(-1, sny, snx)
        ks, cg, fg, rg = _exact_epi(_units(i["images"], snx, sny, nz, nv, dev), fm, T2_MS, TI_MS,
                                    _background(snx, sny, nz, nv, o, dev), _tes(case), nx, ny, o, int(case["coils"]),
                                    int(case["accel"]), float(case["pf"]), float(case["t_line"]), bool(case["gradient"]),
                                    float(case["ghost"]), 100.0, int(case["grads"]), eddy, maps)
        ne, nc = len(_tes(case)), int(case["ncomp"])
        out = {"kspace": ks.reshape(nv, nz, int(case["coils"]), ne, ny, nx), "comp_grad": cg.reshape(nv, nz, nc, sny, snx)}
        if fg is not None:
            out["fmap_grad"] = fg.reshape(nv, nz, sny, snx)
        if rg is not None:
            out["r2_grad"] = rg.reshape(nv, nz, nc, sny, snx)
        return out
    if kind == "batch":
        series, acq = _batch_inputs(case, seed)
        out = []
        for s in series:
            (snx, sny, nz), (nx, ny, _), o = s["sim_dims"], s["acq_dims"], int(case["o"])
            ks, cg, _, _ = _exact_epi(_units(s["images"], snx, sny, nz, 1, dev),
                                      torch.as_tensor(s["fmap"]).to(dev).reshape(nz, sny, snx), T2_MS, TI_MS,
                                      _background(snx, sny, nz, 1, o, dev), [float(case["te"])], nx, ny, o, acq.n_coils, 1,
                                      1.0, 0.5, False, 0.05, 100.0)
            out.append({"kspace": ks.reshape(1, nz, acq.n_coils, 1, ny, nx),
                        "comp_grad": cg.reshape(1, nz, int(case["ncomp"]), sny, snx)})
        return out
    if kind == "slice":
        inp, acq = _slice_inputs(case, seed)
        (snx, sny), (nx, ny), o = inp.sim, inp.acq_matrix, int(case["o"])
        ks, _, _, _ = _exact_epi(_units(inp.compartments, snx, sny, 1, 1, dev),
                                 torch.as_tensor(inp.fmap).to(dev).reshape(1, sny, snx), T2_MS, TI_MS,
                                 torch.as_tensor(inp.phase0, device=dev).reshape(1, sny, snx), [acq.t_echo], nx, ny, o,
                                 acq.n_coils, 1, 1.0, 0.5, False, 0.02, 100.0, adjoint=False)
        fx, fy = (np.arange(nx) - nx // 2) / nx, (np.arange(ny) - ny // 2) / ny
        r = 2.0 * np.sqrt(fx[None, :] ** 2 + fy[:, None] ** 2)
        k = ks[0] * torch.as_tensor(np.where(r >= 1.0, 0.0, 0.5 * (1.0 + np.cos(math.pi * r))), device=dev)
        ix = torch.as_tensor(np.exp(-1j * TAU * np.outer(fx, np.arange(nx) - nx // 2)), device=dev)
        iy = torch.as_tensor(np.exp(-1j * TAU * np.outer(fy, np.arange(ny) - ny // 2)), device=dev)
        img = torch.einsum("qkl,ky,lx->qyx", k, iy, ix)
        s = torch.as_tensor(np.stack([_coil_amp(q, acq.n_coils, np.arange(nx), np.arange(ny), nx, ny)
                                      for q in range(acq.n_coils)]), device=dev)
        return (s * img).sum(0) / (s * s).sum(0)
    if kind == "spiral_forward":
        inp, acq, tr, k, idx, _ = _spiral_slice_inputs(case, seed)
        (sn, _), (n, _), o = inp.sim, inp.acq_matrix, int(case["o"])
        off = (o - 1.0) / 2.0
        xa = (np.arange(sn) - off) / o
        xc = torch.as_tensor((np.arange(sn) - o * (n // 2) - off) / o / n, device=dev)
        a = torch.as_tensor(_coil_amp(0, 8, xa, xa, n, n), device=dev) * torch.as_tensor(
            np.asarray(inp.compartments[0], np.float64), device=dev).reshape(sn, sn)
        a = torch.polar(a, torch.as_tensor(inp.phase0, device=dev).reshape(sn, sn))
        f = torch.as_tensor(np.asarray(inp.fmap, np.float64), device=dev).reshape(sn, sn)
        ns, il = len(tr.tau_ms), int(case["interleaves"])
        kk = torch.as_tensor(k, device=dev).reshape(il, ns, 2)
        out = torch.zeros((il, ns), dtype=torch.complex128, device=dev)
        for j0 in range(0, ns, 64):
            t = torch.as_tensor(tr.tau_ms[j0:j0 + 64], device=dev) / 1e3
            im = a[None] * torch.polar(torch.ones((len(t), sn, sn), dtype=torch.float64, device=dev),
                                       TAU * f[None] * t[:, None, None])
            phx = TAU * kk[:, j0:j0 + 64, 0, None] * xc
            phy = TAU * kk[:, j0:j0 + 64, 1, None] * xc
            ux, uy = torch.polar(torch.ones_like(phx), phx), torch.polar(torch.ones_like(phy), phy)
            rowsum = torch.matmul(uy.permute(1, 0, 2), im)  # [sample][interleaf][x]
            out[:, j0:j0 + 64] = (rowsum * ux.permute(1, 0, 2)).sum(-1).t()
        return out.reshape(-1) / (sn * sn)
    # receiver noise from the framework's own generator, GRAPPA and CG solves, or a stepped state
    # machine: no plain sum gives these
    return None
