"""Cases for timing the time-stepping path through its public entry points.

Each case is one piece of the work that a user of the framework has it do:
whole runs of the fused mixed-precision form (``device.Run``, alone and many at
once in a ``device.Batch``), loops over the FP64 drop-in calls in the order of
``Gencore::run`` (track, push, track, field solver, slippage, diagnostics), and
the single blocks that a program calls by themselves: a field solver on a
frozen beam, short-range space charge, the slice diagnostics.  Inputs are
seeded synthetic beams (quiet start of four-particle beamlets with shot noise)
at the parameters of ``workloads``: gamma 11357, 15 mm undulator, 0.4 um
emittance, 3 kA, FODO lattice.

The families of cases and their keys:

  run     nslice, npart, ngrid, steps, nwig; seeded (steady state) or started
          from shot noise; third (a 3rd-harmonic field beside the fundamental);
          ragged (slices of different, odd particle counts, as imported beams
          have); host state in, steps from a graph, records and state out
  batch   nrun single-slice runs of mixed sizes up to npart and ngrid, steps
  steps   the FP64 calls with diagnostics after every step; solver adi, fft or
          fft_filter; charge (short-range space charge before each push)
  field   one field solver alone on a frozen beam, steps field steps
  charge  short-range space charge: nz, nphi modes on a radial grid of nrad
  records beam (nharm bunching harmonics) and field diagnostics of one state

The mixed form holds its state in single precision, so its results are
returned in single precision; the FP64 form returns double.
"""
import math

import numpy as np
import torch

from genesis4_cuda_port_b200 import _lib
from genesis4_cuda_port_b200 import device as dev

GAMMA0, AW, LAMBDAU = 11357.0, 1.0, 0.015
EMIT, BETA, SPREAD, CURRENT = 0.4e-6, 15.0, 1e-4, 3000.0
GRIDMAX, SEED_POWER, WAIST = 2e-4, 1e3, 30e-6
QUAD_L, QUAD_K1, QUAD_STEPS = 0.1, 1.5, 7
VACIMP, EEV = 376.73031346177, 510998.95
KU = 2 * math.pi / LAMBDAU
# resonant wavelength of the mean particle of the matched beam
LAMBDA0 = LAMBDAU * (1 + AW ** 2 + 2 * GAMMA0 * EMIT / BETA
                     + AW ** 2 * KU * KU * EMIT * BETA / GAMMA0) / (2 * GAMMA0 ** 2)
# space-charge wall over the largest particle radius (which lies on no cell edge)
RMAX = 2.31
FILTER = (0.6, 0.6, 0.1)  # xcut, ycut, sigmoid of the source filter
NAMES = dev.BeamState.NAMES


# ----------------------------------------------------------------- the cases --

def listed():
    return [
        # one slice through the whole 344-step lattice: the smallest run, bound by latency
        dict(name="run_steady", kind="run", nslice=1, npart=8192, ngrid=151, steps=344, nwig=110,
             seeded=True, third=False, ragged=False),
        # a request of the served stream: some tens of slices, sizes off every tile
        dict(name="run_request", kind="run", nslice=37, npart=6148, ngrid=177, steps=110, nwig=40,
             seeded=False, third=False, ragged=False),
        # time-dependent SASE at the size the throughput is quoted on
        dict(name="run_sase", kind="run", nslice=1024, npart=8192, ngrid=201, steps=240, nwig=110,
             seeded=False, third=False, ragged=False),
        # fundamental and 3rd harmonic on the widest usual grid, many particles per slice
        dict(name="run_harmonics", kind="run", nslice=256, npart=16384, ngrid=255, steps=160,
             nwig=60, seeded=False, third=True, ragged=False),
        # a parameter scan: many small steady-state runs of mixed sizes at once
        dict(name="batch_scan", kind="batch", nrun=32, npart=32768, ngrid=301, steps=172, nwig=110),
        # the drop-in FP64 loop, steady state: the reference's default use at its smallest
        dict(name="steps_steady", kind="steps", nslice=1, npart=8192, ngrid=151, steps=60,
             solver="adi", seeded=True, charge=False, ragged=False),
        # the drop-in FP64 loop, time dependent
        dict(name="steps_sase", kind="steps", nslice=256, npart=8192, ngrid=201, steps=60,
             solver="adi", seeded=False, charge=False, ragged=False),
        # the same loop with the spectral field solver
        dict(name="steps_fft", kind="steps", nslice=96, npart=8192, ngrid=201, steps=48,
             solver="fft", seeded=False, charge=False, ragged=False),
        # the spectral solver with its source filter on a wide grid
        dict(name="field_filter", kind="field", nslice=64, npart=4096, ngrid=255, steps=24,
             solver="fft_filter"),
        # the ADI solver on a grid wider than the configurations', few slices
        dict(name="field_wide", kind="field", nslice=40, npart=4096, ngrid=401, steps=32,
             solver="adi"),
        # space charge of a short bunch train, two longitudinal modes, |m| <= 1
        dict(name="space_charge", kind="charge", nslice=48, npart=8192, nrad=100, nz=2, nphi=1,
             ragged=False),
        # one output step's diagnostics of imported slices with four bunching harmonics
        dict(name="records", kind="records", nslice=300, npart=5000, ngrid=129, nharm=4,
             ragged=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    kind = rng.choice(["run", "run", "batch", "steps", "steps", "field", "charge", "records"])
    npart = 4 * _log(rng, 512, 4096)
    if kind == "run":
        c = dict(kind=kind, nslice=_log(rng, 1, 512), npart=npart, ngrid=rng.randint(101, 255),
                 steps=rng.randint(60, 344), nwig=rng.randint(20, 110),
                 third=rng.random() < 0.25, ragged=rng.random() < 0.3)
        c["seeded"] = c["nslice"] == 1
        return c
    if kind == "batch":
        return dict(kind=kind, nrun=_log(rng, 8, 60), npart=4 * _log(rng, 1024, 8192),
                    ngrid=rng.randint(151, 301), steps=rng.randint(100, 344), nwig=110)
    if kind == "steps":
        c = dict(kind=kind, nslice=_log(rng, 1, 256), npart=npart, ngrid=rng.randint(101, 255),
                 steps=rng.randint(24, 80), solver=rng.choice(["adi", "adi", "fft", "fft_filter"]),
                 charge=rng.random() < 0.25, ragged=rng.random() < 0.3)
        c["seeded"] = c["nslice"] == 1
        return c
    if kind == "field":
        solver = rng.choice(["adi", "fft", "fft_filter"])
        return dict(kind=kind, nslice=_log(rng, 1, 128), npart=npart, steps=rng.randint(8, 48),
                    ngrid=rng.randint(65, 450 if solver == "adi" else 256), solver=solver)
    if kind == "charge":
        return dict(kind=kind, nslice=_log(rng, 1, 256), npart=npart, nrad=_log(rng, 40, 150),
                    nz=rng.randint(1, 3), nphi=rng.randint(0, 2), ragged=rng.random() < 0.3)
    return dict(kind=kind, nslice=_log(rng, 1, 512), npart=npart, ngrid=rng.randint(101, 255),
                nharm=rng.randint(1, 5), ragged=rng.random() < 0.3)


def draw(rng):
    most = max(work(c)["bytes"] for c in listed())
    while True:
        c = _draw(rng)
        if work(c)["bytes"] <= most and c.get("nslice", 1) * c["npart"] <= 5_000_000 and \
                c.get("nslice", 1) * c.get("ngrid", 1) ** 2 <= 45_000_000:
            return c


def work(case):
    """Every step has to read and write the particles (28 bytes in the mixed
    form, 48 in FP64) and the field cells (8 and 16 bytes) once; the states of
    all but the smallest cases are larger than the chip's caches."""
    kind, n = case["kind"], case.get("ngrid", 0)
    if kind == "batch":
        parts = cells = 0
        for j in _jobs(case):
            parts += j["npart"]
            cells += j["ngrid"] ** 2
        steps = case["steps"]
        return {"bytes": steps * (56 * parts + 16 * cells), "flops": steps * (300 * parts + 80 * cells)}
    parts = int(_counts(case).sum())
    cells = case["nslice"] * n * n
    if kind == "run":
        nf = 2 if case["third"] else 1
        return {"bytes": case["steps"] * (56 * parts + 16 * cells * nf),
                "flops": case["steps"] * (300 * parts + 80 * cells * nf)}
    if kind == "steps":
        return {"bytes": case["steps"] * (96 * parts + 32 * cells),
                "flops": case["steps"] * (500 * parts + 80 * cells)}
    if kind == "field":
        return {"bytes": case["steps"] * (32 * parts + 32 * cells),
                "flops": case["steps"] * (60 * parts + 80 * cells)}
    if kind == "charge":
        modes = case["nz"] * (2 * case["nphi"] + 1)
        return {"bytes": 32 * parts, "flops": (40 + 20 * modes) * parts}
    return {"bytes": 48 * parts + 16 * cells, "flops": (60 + 40 * case["nharm"]) * parts + 12 * cells}


# ---------------------------------------------------------------- the inputs --

def _counts(case):
    """Particles per slice: the same for every seed."""
    ns, npart = case["nslice"], case["npart"]
    if not case.get("ragged"):
        return np.full(ns, npart, np.int64)
    r = np.random.default_rng([ns, npart])
    return np.maximum(1, npart - r.integers(0, max(2, npart // 3), ns)).astype(np.int64)


def _beam(counts, seed, detune=0.0):
    """Quiet-start beamlets of four with shot noise, FP64, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)
    nb = int(math.ceil(counts.max() / 4))
    ns = len(counts)

    def normal():
        return torch.randn(ns, nb, 1, generator=g, device="cuda", dtype=torch.float64)

    geo = EMIT / GAMMA0
    sx, sp = math.sqrt(geo * BETA), math.sqrt(geo / BETA)
    gam = GAMMA0 * (1 + detune) * (1 + SPREAD * normal())
    p = {"x": sx * normal(), "y": sx * normal(), "px": gam * sp * normal(),
         "py": gam * sp * normal(), "gamma": gam}
    th = 0.5 * math.pi * (torch.rand(ns, nb, 1, generator=g, device="cuda", dtype=torch.float64)
                          + torch.arange(4, device="cuda", dtype=torch.float64))
    ne = CURRENT * LAMBDA0 / (1.602176634e-19 * 299792458.0) / nb  # electrons per beamlet
    dth = torch.zeros_like(th)
    for h in (1, 2):
        s = math.sqrt(2 / ne) / h
        dth = dth + s * normal() * torch.cos(h * th) + s * normal() * torch.sin(h * th)
    p["theta"] = th + dth
    keep = (torch.arange(4 * nb, device="cuda")[None, :]
            < torch.as_tensor(counts, device="cuda")[:, None])
    return {k: p[k].expand(ns, nb, 4).reshape(ns, 4 * nb)[keep].contiguous() for k in NAMES}


def _gaussian(n, dtype=torch.complex128):
    x = torch.linspace(-GRIDMAX, GRIDMAX, n, dtype=torch.float64, device="cuda")
    g = torch.exp(-(x[None, :] ** 2 + x[:, None] ** 2) / WAIST ** 2)
    unit = 2 * GRIDMAX / (n - 1) * EEV / (2 * math.pi / LAMBDA0)
    return (g * torch.sqrt(SEED_POWER * VACIMP / (unit ** 2 * (g * g).sum()))).to(dtype)


def _noise_field(ns, n, seed):
    """Seeded modes of different amplitude and tilt, one per slice."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 5)
    a = torch.rand(ns, 4, generator=g, device="cuda", dtype=torch.float64)
    x = torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda")
    amp = (0.2 + a[:, 0]) * torch.exp(2j * math.pi * a[:, 1])
    tilt_x = torch.exp(20j * (a[:, 2] - 0.5)[:, None] * x)
    tilt_y = torch.exp(20j * (a[:, 3] - 0.5)[:, None] * x)
    return (amp[:, None, None] * _gaussian(n)[None] * tilt_y[:, :, None] * tilt_x[:, None, :])


def _coupling(h):
    """Planar coupling factor aw (J_m(xi) - J_m+1(xi)) (-1)^m."""
    xi, m = h * AW ** 2 / (2 * (1 + AW ** 2)), (h - 1) // 2

    def bessel(k):
        return sum((-1) ** j / (math.factorial(j) * math.factorial(j + k)) * (xi / 2) ** (2 * j + k)
                   for j in range(20))

    return AW * (-1) ** m * (bessel(m) - bessel(m + 1))


def _lattice(steps, nwig):
    """Undulator sections of nwig steps between FODO quadrupoles."""
    out, sign = [], 1.0
    while len(out) < steps:
        out += [dict(delz=LAMBDAU, aw=AW, ky=KU * KU, ku=KU, qf=0.0, und=1,
                     slip=LAMBDAU * (1 + AW ** 2) / (2 * GAMMA0 ** 2) / LAMBDA0)] * nwig
        dz = QUAD_L / QUAD_STEPS
        out += [dict(delz=dz, aw=0.0, ky=0.0, ku=0.0, qf=sign * QUAD_K1, und=0,
                     slip=dz / (2 * GAMMA0 ** 2) / LAMBDA0)] * QUAD_STEPS
        sign = -sign
    return out[:steps]


def _step(s):
    return dev.Step(delz=s["delz"], aw=s["aw"], ky=s["ky"], ku=s["ku"], qf=s["qf"],
                    in_undulator=s["und"], gamma_ref=GAMMA0)


def _nwig(case):
    return case.get("nwig") or max(8, case["steps"] // 3)


def _jobs(case):
    """Sizes of the scan's runs: the same for every seed."""
    r = np.random.default_rng(case["nrun"] * 1000 + case["ngrid"])
    return [dict(npart=4 * int(r.integers(512, case["npart"] // 4 + 1)),
                 ngrid=int(r.integers(101, case["ngrid"] + 1)),
                 detune=float(r.uniform(-5e-4, 5e-4))) for _ in range(case["nrun"])]


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _host(t):
    return _pinned(t.shape, t.dtype).copy_(t).numpy()


def _offsets(counts):
    return np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)


# ------------------------------------------------------------------ prepare --

class _RunState:
    """A fused run and the host buffers its program keeps."""

    def __init__(self, ctx, counts, beam, ngrids, steps, seeded):
        lat = _lattice(*steps)
        ns = len(counts)
        harms = [1, 3][: len(ngrids)]
        self.nsteps = len(lat)
        self.seed = _host(_gaussian(ngrids[0])[None]) if seeded else None
        self.parts = {k: _host(v) for k, v in beam.items()}
        self.run = dev.Run(ctx, _offsets(counts), fields=[(h, n, GRIDMAX) for h, n in zip(harms, ngrids)],
                           lambda0=LAMBDA0, gamma_ref=GAMMA0, time_run=ns > 1)
        self.run.set_current(CURRENT)
        fc = [[_coupling(h) if s["und"] else 0.0 for h in harms] for s in lat]
        self.run.set_lattice([_step(s) for s in lat], fc, [s["slip"] for s in lat])
        self.beam_out = {k: _pinned(v.shape) for k, v in self.parts.items()}
        self.field_out = [_pinned((ns, n, n), torch.complex128) for n in ngrids]
        self.beam32 = {k: _pinned(v.shape, torch.float32) for k, v in self.parts.items()}
        self.field32 = [_pinned((ns, n, n), torch.complex64) for n in ngrids]

    def upload(self):
        self.run.upload_beam(self.parts)
        for i in range(len(self.field_out)):
            self.run.upload_field(i, self.seed if i == 0 else None)

    def results(self):
        beam, field = self.run.history_range(0, self.nsteps)
        self.run.download_beam({k: v.numpy() for k, v in self.beam_out.items()})
        for i, f in enumerate(self.field_out):
            self.run.download_field(i, f.numpy())
        return dict(beam_records=beam.astype(np.float32), field_records=field.astype(np.float32),
                    beam={k: self.beam32[k].copy_(v) for k, v in self.beam_out.items()},
                    field=[a.copy_(b) for a, b in zip(self.field32, self.field_out)])


def _solver(ctx, name):
    if name == "adi":
        return dev.FieldSolverADICUDA(ctx)
    s = dev.FieldSolverFFTCUDA(ctx)
    if name == "fft_filter":
        s.init_source_filter(*FILTER, True)
    return s


def prepare(case, seed):
    ctx = dev.Context(0)
    kind = case["kind"]
    st = dict(case=dict(case), ctx=ctx)
    if kind == "batch":
        st["runs"] = []
        for i, j in enumerate(_jobs(case)):
            counts = np.array([j["npart"]], np.int64)
            st["runs"].append(_RunState(ctx, counts, _beam(counts, seed * 64 + i, j["detune"]),
                                        [j["ngrid"]], (case["steps"], case["nwig"]), True))
        st["batch"] = dev.Batch(ctx, case["nrun"])
        torch.cuda.synchronize()
        return st
    counts = _counts(case)
    beam = _beam(counts, seed)
    ns, n = case["nslice"], case.get("ngrid", 0)
    if kind == "run":
        st["run"] = _RunState(ctx, counts, beam, [n, n] if case["third"] else [n],
                              (case["steps"], case["nwig"]), case["seeded"])
        torch.cuda.synchronize()
        return st
    st["parts"] = {k: _host(v) for k, v in beam.items()}
    st["beam"] = dev.BeamState(ctx, _offsets(counts), GAMMA0)
    st["beam"].set_current(np.full(ns, CURRENT))
    if kind == "charge":
        st["beam"].upload(st["parts"])
        st["efield"] = dev.EFieldSolver(ctx, RMAX, case["nrad"], case["nz"], case["nphi"], LAMBDA0)
        st["ez"] = _pinned(int(counts.sum()))
        return st
    st["field"] = dev.FieldState(ctx, ns, n, GRIDMAX, LAMBDA0)
    if kind == "steps":
        cells = _gaussian(n)[None] if case["seeded"] else \
            torch.zeros(ns, n, n, dtype=torch.complex128, device="cuda")
        st["solver"] = _solver(ctx, case["solver"])
        st["lattice"] = [(s, _step(s), _coupling(1) if s["und"] else 0.0)
                         for s in _lattice(case["steps"], _nwig(case))]
        st["efield"] = dev.EFieldSolver(ctx, RMAX, 60, 1, 0, LAMBDA0) if case["charge"] else None
        st["beam_out"] = {k: _pinned(v.shape) for k, v in st["parts"].items()}
    else:
        cells = _noise_field(ns, n, seed)
        st["beam"].upload(st["parts"])
    st["cells"] = _host(cells)
    st["field"].upload(st["cells"])
    if kind == "field":
        st["solver"] = _solver(ctx, case["solver"])
        st["solver"].init(LAMBDAU, st["field"].dgrid, st["field"].xks, n)
        st["step"] = _step(_lattice(1, 1)[0])
    st["field_out"] = _pinned((ns, n, n), torch.complex128)
    return st


# ---------------------------------------------------------------------- run --

def _download(field, out):
    _lib.check(field.lib.g4b_field_download(field.h, _lib.dptr(out.numpy().reshape(-1).view(np.float64))))
    return out


def run(st):
    return _RUN[st["case"]["kind"]](st)


def _run_run(st):
    r = st["run"]
    r.upload()
    r.run.advance(0, r.nsteps, graph=True)
    return r.results()


def _run_batch(st):
    batch, steps = st["batch"], st["case"]["steps"]
    slots = []
    for r in st["runs"]:
        r.upload()
        slots.append(batch.attach(r.run, 0, steps))
    batch.step(steps)
    got = [r.results() for r in st["runs"]]
    for s in slots:
        batch.detach(s)
    return dict(beam_records=np.concatenate([g["beam_records"] for g in got], 1),
                field_records=np.concatenate([g["field_records"] for g in got], 2),
                beam={k: torch.cat([g["beam"][k] for g in got]) for k in NAMES},
                field=torch.cat([g["field"][0].reshape(-1) for g in got]))


def _run_steps(st):
    beam, field, solver, efield = st["beam"], st["field"], st["solver"], st["efield"]
    time_run = field.nslice > 1
    beam.upload(st["parts"])
    field.upload(st["cells"])
    field.first, field.accuslip = 0, 0.0
    records = []
    for s, step, fc in st["lattice"]:
        solver.init(s["delz"], field.dgrid, field.xks, field.ngrid)
        beam.track(step, 0.5 * s["delz"], False)
        if efield:
            efield.short_range(beam, GAMMA0 ** 2 / (1 + s["aw"] ** 2))
        beam.advance([field], [fc], step)
        beam.track(step, 0.5 * s["delz"], True)
        solver.advance(field, beam, step, fc)
        field.apply_slippage(s["slip"], 1.0, time_run)
        records.append(beam.diagnostics() + field.diagnostics())
    _lib.check(beam.lib.g4b_beam_download(beam.h, *[_lib.dptr(st["beam_out"][k].numpy()) for k in NAMES]))
    return dict(records=[np.stack([r[i] for r in records]) for i in range(5)],
                beam=st["beam_out"], field=_download(field, st["field_out"]))


def _run_field(st):
    fc = _coupling(1)
    for _ in range(st["case"]["steps"]):
        st["solver"].advance(st["field"], st["beam"], st["step"], fc)
    return _download(st["field"], st["field_out"])


def _run_charge(st):
    st["efield"].short_range(st["beam"], GAMMA0 ** 2 / (1 + AW ** 2))
    _lib.check(st["beam"].lib.g4b_beam_get_particle_ez(st["beam"].h, _lib.dptr(st["ez"].numpy())))
    return st["ez"]


def _run_records(st):
    return list(st["beam"].diagnostics(st["case"]["nharm"], True)) + list(st["field"].diagnostics())


_RUN = dict(run=_run_run, batch=_run_batch, steps=_run_steps, field=_run_field,
            charge=_run_charge, records=_run_records)


# -------------------------------------------------------------------- exact --
# The same path in plain torch, 64 bits, from its equations.

class _Exact:
    def __init__(self, counts, parts):
        self.p = {k: v.clone() for k, v in parts.items()}
        self.ns = len(counts)
        self.counts = torch.as_tensor(counts, device="cuda")
        self.slice = torch.repeat_interleave(torch.arange(self.ns, device="cuda"), self.counts)
        self.ez = 0.0
        self.inv = {}

    # transverse map over dz of one plane: focusing, defocusing or drift
    @staticmethod
    def _plane(c, p, k, dz, gz):
        if k == 0.0:
            return c + p * dz / gz, p
        foc = torch.sqrt(abs(k) / gz)
        w = foc * dz
        cs, sn, sg = (torch.cos(w), torch.sin(w), -1.0) if k > 0 else (torch.cosh(w), torch.sinh(w), 1.0)
        return cs * c + sn / foc * p / gz, sg * sn * foc * c * gz + cs * p

    def track(self, s, dz):
        p = self.p
        gz = torch.sqrt(p["gamma"] ** 2 - 1 - s["aw"] ** 2 - p["px"] ** 2 - p["py"] ** 2)
        beta = math.sqrt(1 - (1 + s["aw"] ** 2) / GAMMA0 ** 2)
        quad, nat = s["qf"] * GAMMA0, s["ky"] * s["aw"] ** 2 / GAMMA0 / beta
        p["x"], p["px"] = self._plane(p["x"], p["px"], quad, dz, gz)
        p["y"], p["py"] = self._plane(p["y"], p["py"], -quad + nat, dz, gz)

    def _cells(self, n):
        x, y, d = self.p["x"], self.p["y"], 2 * GRIDMAX / (n - 1)
        fx, fy = (x + GRIDMAX) / d, (y + GRIDMAX) / d
        ix, iy = torch.floor(fx), torch.floor(fy)
        ok = (x.abs() < GRIDMAX) & (y.abs() < GRIDMAX) & (ix >= 0) & (ix < n - 1) & (iy >= 0) & (iy < n - 1)
        wx, wy = 1 + ix - fx, 1 + iy - fy
        at = torch.where(ok, iy * n + ix, torch.zeros_like(ix)).long()
        w = [torch.where(ok, a, torch.zeros_like(a))
             for a in (wx * wy, (1 - wx) * wy, wx * (1 - wy), (1 - wx) * (1 - wy))]
        return at, w, (0, 1, n, n + 1)

    def push(self, s, fields):
        p, dz = self.p, s["delz"]
        ks = 2 * math.pi / LAMBDA0
        ku = s["ku"] or ks * 0.5 / GAMMA0 ** 2
        awl = 1 + 0.5 * s["ky"] * p["y"] ** 2
        bt = 1 + p["px"] ** 2 + p["py"] ** 2 + s["aw"] ** 2 * awl ** 2
        rs = []
        for f in fields:
            n = f["n"]
            at, w, step = self._cells(n)
            plane = (self.slice + f["first"]) % self.ns
            flat = f["u"].reshape(-1)
            c = sum(flat[plane * (n * n) + at + o] * wi for o, wi in zip(step, w))
            rs.append((f["h"], f["fc"] * (LAMBDA0 / f["h"]) / (2 * math.pi) * awl * c.conj()))

        def ode(g, t):
            z = sum(r * torch.exp(-1j * h * t) for h, r in rs)
            e = (bt - 2 / ks * z.real) / g ** 2
            b = torch.sqrt(1 - e)
            return z.imag / b / g - self.ez, ku - ks * e / (b * (1 + b))

        g0, t0 = p["gamma"], p["theta"]
        a = ode(g0, t0)
        b = ode(g0 + 0.5 * dz * a[0], t0 + 0.5 * dz * a[1])
        c = ode(g0 + 0.5 * dz * b[0], t0 + 0.5 * dz * b[1])
        d = ode(g0 + dz * c[0], t0 + dz * c[1])
        p["gamma"], p["theta"] = (y + dz / 6 * (a[i] + 2 * b[i] + 2 * c[i] + d[i])
                                  for i, y in ((0, g0), (1, t0)))

    def source(self, s, f):
        n, p, d = f["n"], self.p, 2 * GRIDMAX / (f["n"] - 1)
        at, w, step = self._cells(n)
        scl = f["fc"] * VACIMP * CURRENT * (2 * math.pi * f["h"] / LAMBDA0) * s["delz"] / \
            (4 * EEV * self.counts.double() * d * d)
        q = scl[self.slice] * torch.sqrt(1 + s["ky"] * p["y"] ** 2) / p["gamma"]
        v = 1j * q * torch.exp(-1j * f["h"] * p["theta"])
        at = (self.slice + f["first"]) % self.ns * (n * n) + at
        src = torch.zeros(self.ns * n * n, dtype=torch.complex128, device="cuda")
        for o, wi in zip(step, w):
            src.index_add_(0, at + o, v * wi)
        return src.reshape(self.ns, n, n)

    def field(self, s, f, solver="adi"):
        n, d, ks = f["n"], 2 * GRIDMAX / (f["n"] - 1), 2 * math.pi * f["h"] / LAMBDA0
        src = self.source(s, f) if s["und"] else 0.0
        if solver == "adi":
            r = 0.25 * s["delz"] / (ks * d * d)
            key = (n, r)
            if key not in self.inv:
                e = torch.ones(n - 1, dtype=torch.complex128, device="cuda")
                lap = torch.diag(e, 1) + torch.diag(e, -1) - 2 * torch.eye(n, dtype=torch.complex128, device="cuda")
                eye = torch.eye(n, dtype=torch.complex128, device="cuda")
                self.inv[key] = torch.linalg.inv(eye - 1j * r * lap), eye + 1j * r * lap
            inv, fwd = self.inv[key]
            u = (fwd @ f["u"] + src) @ inv.T
            f["u"] = inv @ (u @ fwd.T + src)
            return
        k = torch.arange(n, dtype=torch.float64, device="cuda") - 0.5 * (n - 1)
        k = torch.roll(k, (n + 1) // 2)
        k2 = k[None, :] ** 2 + k[:, None] ** 2
        prop = torch.exp(-0.5j * k2 * (2 * math.pi / (n * d)) ** 2 / ks * s["delz"])
        spec = torch.fft.fft2(f["u"]) * prop
        if s["und"]:
            filt = 1.0
            if solver == "fft_filter":
                rad = torch.sqrt((k / n / FILTER[0])[None, :] ** 2 + (k / n / FILTER[1])[:, None] ** 2)
                filt = 1 / (1 + torch.exp((rad - 1) / FILTER[2]))
            spec = spec + 2 * filt * torch.fft.fft2(src)
        f["u"] = torch.fft.ifft2(spec)

    def slip(self, s, f):
        f["acc"] += s["slip"]
        while abs(f["acc"]) > 0.8:
            f["acc"] -= 1.0
            f["first"] = (f["first"] + self.ns - 1) % self.ns
            f["u"][f["first"]] = 0

    def _sum(self, v):
        return torch.zeros(self.ns, dtype=torch.float64, device="cuda").index_add_(0, self.slice, v)

    def beam_stats(self, nharm):
        p = self.p
        x, y, px, py, g, t = (p[k] for k in NAMES)
        cols = [self._sum(v) for v in (g, g * g, x, x * x, y, y * y, px, px * px, py, py * py, x * px,
                                       y * py, torch.ones_like(x))]
        for v in (x, px, y, py, g):
            for op in ("amin", "amax"):
                z = torch.zeros(self.ns, dtype=torch.float64, device="cuda")
                cols.append(z.scatter_reduce_(0, self.slice, v, op, include_self=False))
        b = [[self._sum(fn(h * t)) for h in range(1, nharm + 1)] for fn in (torch.cos, torch.sin)]
        return torch.stack(cols, 1), torch.stack(b[0], 1), torch.stack(b[1], 1)

    def field_stats(self, f):
        n = f["n"]
        u = torch.roll(f["u"], -f["first"], 0)
        d = torch.arange(n, dtype=torch.float64, device="cuda") - 0.5 * (n - 1)
        w = u.real ** 2 + u.imag ** 2
        wx, wy = w.sum(1), w.sum(2)
        s = u.sum((1, 2))
        c = u.reshape(self.ns, -1)[:, (n * n - 1) // 2]
        return (torch.stack([wx.sum(1), (wx * d).sum(1), (wx * d * d).sum(1), (wy * d).sum(1),
                             (wy * d * d).sum(1), s.real, s.imag], 1),
                torch.stack([c.real, c.imag], 1))

    def charge(self, gz2, n, nz, nphi):
        p, ks = self.p, 2 * math.pi / LAMBDA0
        cnt = self.counts.double()
        dx = p["x"] - (self._sum(p["x"]) / cnt)[self.slice]
        dy = p["y"] - (self._sum(p["y"]) / cnt)[self.slice]
        r = torch.sqrt(dx * dx + dy * dy)
        big = torch.zeros(self.ns, dtype=torch.float64, device="cuda")
        big.scatter_reduce_(0, self.slice, r, "amax", include_self=False)
        dr = RMAX * big / n
        cell = torch.clamp((r / dr[self.slice]).long(), max=n - 1)
        phi = torch.atan2(dy, dx)
        rc = torch.arange(n, dtype=torch.float64, device="cuda") + 0.5
        total = torch.zeros_like(r)
        for h in range(1, nz + 1):
            for m in range(-nphi, nphi + 1):
                e = torch.exp(-1j * (h * p["theta"] + m * phi))
                acc = torch.zeros(self.ns * n, dtype=torch.complex128, device="cuda")
                acc.index_add_(0, self.slice * n + cell, e)
                rhs = -acc.reshape(self.ns, n) / (2 * math.pi * cnt)[:, None]
                up, lo = rc + 0.5, rc - 0.5
                diag = -lo - torch.where(rc > n - 1, 2 * up, up)
                k2 = (h * ks * dr) ** 2 / gz2
                mat = torch.diag_embed(diag - m * m / rc - k2[:, None] * rc)
                mat = mat + torch.diag(up[:-1], 1) + torch.diag(lo[1:], -1)
                u = torch.linalg.solve(mat.to(torch.complex128), rhs)
                total = total + h * (u.reshape(-1)[self.slice * n + cell] * e.conj()).imag
        self.ez = -2 * VACIMP * ks / (EEV * gz2) * CURRENT * total
        return self.ez


def _exact_run(counts, beam, ngrids, lattice, seeded):
    e = _Exact(counts, beam)
    fields = [dict(n=n, h=h, first=0, acc=0.0,
                   u=torch.zeros(e.ns, n, n, dtype=torch.complex128, device="cuda"))
              for n, h in zip(ngrids, (1, 3))]
    if seeded:
        fields[0]["u"] += _gaussian(ngrids[0])
    rb, rf = [], []
    for s in lattice:
        for f in fields:
            f["fc"] = _coupling(f["h"]) if s["und"] else 0.0
        e.track(s, 0.5 * s["delz"])
        e.push(s, fields)
        e.track(s, 0.5 * s["delz"])
        for f in fields:
            e.field(s, f)
            if e.ns > 1:
                e.slip(s, f)
        st, re, im = e.beam_stats(1)
        rb.append(torch.cat([st, re, im], 1))
        rf.append(torch.stack([torch.cat(e.field_stats(f), 1) for f in fields]))
    return dict(beam_records=torch.stack(rb), field_records=torch.stack(rf), beam=e.p,
                field=[f["u"] for f in fields])


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        if case["nrun"] * case["steps"] > 6000:  # some 3 ms per run and step
            return None
        got = []
        for i, j in enumerate(_jobs(case)):
            counts = np.array([j["npart"]], np.int64)
            got.append(_exact_run(counts, _beam(counts, seed * 64 + i, j["detune"]), [j["ngrid"]],
                                  _lattice(case["steps"], case["nwig"]), True))
        return dict(beam_records=torch.cat([g["beam_records"] for g in got], 1),
                    field_records=torch.cat([g["field_records"] for g in got], 2),
                    beam={k: torch.cat([g["beam"][k] for g in got]) for k in NAMES},
                    field=torch.cat([g["field"][0].reshape(-1) for g in got]))
    counts = _counts(case)
    beam = _beam(counts, seed)
    ns, n = case["nslice"], case.get("ngrid", 0)
    if kind == "run":
        return _exact_run(counts, beam, [n, n] if case["third"] else [n],
                          _lattice(case["steps"], case["nwig"]), case["seeded"])
    e = _Exact(counts, beam)
    if kind == "charge":
        return e.charge(GAMMA0 ** 2 / (1 + AW ** 2), case["nrad"], case["nz"], case["nphi"])
    f = dict(n=n, h=1, first=0, acc=0.0, fc=_coupling(1))
    if kind == "records":
        f["u"] = _noise_field(ns, n, seed)
        return list(e.beam_stats(case["nharm"])) + list(e.field_stats(f))
    if kind == "field":
        f["u"] = _noise_field(ns, n, seed)
        for _ in range(case["steps"]):
            e.field(_lattice(1, 1)[0], f, case["solver"])
        return f["u"]
    f["u"] = _gaussian(n)[None].clone() if case["seeded"] else \
        torch.zeros(ns, n, n, dtype=torch.complex128, device="cuda")
    records = []
    for s in _lattice(case["steps"], _nwig(case)):
        f["fc"] = _coupling(1) if s["und"] else 0.0
        e.track(s, 0.5 * s["delz"])
        if case["charge"]:
            e.charge(GAMMA0 ** 2 / (1 + s["aw"] ** 2), 60, 1, 0)
        e.push(s, [f])
        e.track(s, 0.5 * s["delz"])
        e.field(s, f, case["solver"])
        if ns > 1:
            e.slip(s, f)
        records.append(e.beam_stats(1) + e.field_stats(f))
    return dict(records=[torch.stack([r[i] for r in records]) for i in range(5)], beam=e.p,
                field=f["u"])
