"""The work that users have this framework do, as cases that can be timed and
checked: whole stretches of the particle-in-cell loop in both number formats,
field-only build-up, Poisson solves, a served request and a batched scan, each
through the public Python entry points.

A case of kind ``run`` is a stretch of a simulation as a program does it that
holds its state in host memory (a restart from a saved state, or a driver that
looks at the fields between stretches): upload the fields and the beam from
page-locked arrays, advance ``steps`` steps of perform_integration's loop,
read the fields and the beam back and put the particles in the order of their
IDs.  The instance (mesh, geometry, solver set-up, screens) is made once.

Sizes: the 1.6-cell gun (3001 x 821 nodes, 1M macroparticles, Poisson every 20
steps) and the DC gun (1501 x 1001 nodes, 4M macroparticles, Poisson every
step) are the repository's benchmark configurations, the meshes between
120 x 80 and 1500 x 400 with 10k to 500k macroparticles are its scan's range.
"""
import math

import numpy as np
import torch

from spiffe_b200 import abi, geometry, gpu, serve, workloads

C = workloads.C_MKS
EPS0 = 8.85418781762039e-12
MU0 = 1.2566370614359173e-06
QOMC = -workloads.E_MKS / (9.1093837015e-31 * C)
RF_HZ = 2.856e9
BEAM_OUT = ("z", "r", "pz", "pr", "r_pphi", "rmax", "zmax")
TE_NAMES = ("Ephi", "Br", "Bz")


# ------------------------------------------------------------------ the cases

def listed():
    run = dict(kind="run", form="split32", workload="gun", te=False, smear=False, ordered=False)
    return [
        # the headline benchmark: the gun with space charge, split-precision form
        dict(run, name="gun", nz=3001, nr=821, n_macro=1_000_000, steps=200, interval=20),
        # the same state in the bit-faithful FP64 form, the default of every entry point
        dict(run, name="gun_f64", form="f64", nz=3001, nr=821, n_macro=1_000_000, steps=20, interval=20),
        # the DC gun: imposed field of the electrodes, a correction every step
        dict(run, name="dcgun", workload="dcgun", nz=1501, nr=1001, n_macro=4_000_000, steps=12, interval=1),
        # cavity fields built up by an antenna before any beam exists
        dict(run, name="buildup", workload="cavity", nz=3001, nr=821, n_macro=0, steps=400, interval=0),
        dict(run, name="buildup_f64", form="f64", workload="cavity", nz=1201, nr=329, n_macro=0, steps=400,
             interval=0),
        # every field component and smeared deposition (load-bearing for beams
        # with angular momentum in a solenoid), odd sizes
        dict(run, name="te_smear", nz=601, nr=165, n_macro=200_000, steps=100, interval=20, te=True, smear=True),
        # an input deck's run in the FP64 form: deposition in particle order, a small mesh
        dict(run, name="deck_f64", form="f64", nz=301, nr=83, n_macro=20_000, steps=60, interval=20, ordered=True),
        # one request of the server from its parameters to its beam: emission
        # from a cathode and 100 ps of flight (short of the exit), the smallest problem
        dict(kind="request", name="request", nz=105, nr=161, n_macro=20_000, steps=340),
        # a design scan: independent guns of the scan's range advanced together
        dict(kind="scan", name="scan", n=8, draw_seed=7, steps=200),
        # the Poisson solver alone: multigrid on the scan's largest, anisotropic mesh
        dict(kind="solve", name="solve", form="split32", nz=1500, nr=400, accuracy=1e-6, limit=1000),
        # and the reference's SOR in FP64 up to its usual iteration limit
        dict(kind="solve", name="solve_f64", form="f64", nz=1201, nr=329, accuracy=1e-6, limit=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "request", "scan", "solve", "solve"])
    if kind == "request":
        nz, nr = _log_int(rng, 80, 250), _log_int(rng, 80, 300)
        dt = 0.5 * min(0.026 / (nz - 1), 0.040 / (nr - 1)) / C / math.sqrt(2.0)
        return dict(kind=kind, nz=nz, nr=nr, n_macro=_log_int(rng, 5_000, 100_000), steps=int(100e-12 / dt))
    if kind == "scan":
        return dict(kind=kind, n=rng.randint(4, 8), draw_seed=rng.randrange(1, 10_000), steps=_log_int(rng, 50, 200))
    form = rng.choice(["split32", "f64"])
    if kind == "solve":
        return dict(kind=kind, form=form, nz=_log_int(rng, 120, 1600), nr=_log_int(rng, 80, 420),
                    accuracy=rng.choice([1e-4, 1e-5, 1e-6]), limit=rng.randint(400, 1000))
    f64 = form == "f64"
    w = rng.choice(["gun", "gun", "dcgun", "cavity"])
    c = dict(kind=kind, form=form, workload=w, nz=_log_int(rng, 120, 1500), nr=_log_int(rng, 80, 400),
             n_macro=0 if w == "cavity" else _log_int(rng, 10_000, 500_000),
             steps=_log_int(rng, 20, 60) if f64 else _log_int(rng, 50, 200), interval=0, te=False, smear=False,
             ordered=False)
    if w == "gun":
        c["interval"] = rng.choice([10, 20, 40])
        c["te"] = c["smear"] = rng.random() < 0.25
        c["ordered"] = f64 and rng.random() < 0.5
    elif w == "dcgun":
        c["interval"] = rng.choice([1, 4])
        c["steps"] = max(6, c["steps"] // 4)
    return c


# ------------------------------------------------------------- preparing them

def _pinned(a):
    t = torch.empty(a.shape, dtype=getattr(torch, str(a.dtype).replace("uint64", "int64")), pin_memory=True)
    out = t.numpy().view(a.dtype)
    out[...] = a
    return out


def _holding(f, arrays):
    """The problem of f with only these arrays, page-locked."""
    out = abi.Fields.__new__(abi.Fields)
    out.mesh, out.shape, out.flags = f.mesh, f.shape, _pinned(f.flags)
    out.a = {k: _pinned(v) for k, v in arrays.items()}
    return out


def _beam_out(n):
    b = abi.Beam(1)
    b.capacity = n
    b.a = {k: (_pinned(np.zeros(n)) if k in BEAM_OUT else None) for k in abi.BEAM_DOUBLES}
    b.particleID, b.generation = _pinned(np.zeros(n, np.int32)), _pinned(np.zeros(n, np.int16))
    b.status = _pinned(np.zeros(n, np.uint64))
    return b


def _modes(case):
    m = abi.FL_TM_FIELDS | abi.FL_RADIAL_INTERP | abi.FL_LONGIT_INTERP | abi.FL_SPACE_CHARGE
    if case["te"]:
        m |= abi.FL_TE_FIELDS
    if case["smear"]:
        m |= abi.FL_RADIAL_SMEAR | abi.FL_LONGIT_SMEAR
    return m


def _config(case, seed):
    """The workload's configuration with the seed's field, charge and beam."""
    rng = np.random.default_rng(seed)
    u = rng.uniform(0.9, 1.1, 3)
    if case["workload"] == "dcgun":
        return workloads.DcGunConfig(nz=case["nz"], nr=case["nr"], n_macro=case["n_macro"], charge=0.5e-9 * u[0],
                                     voltage=300e3 * u[1], seed=seed)
    return workloads.Gun16Config(nz=case["nz"], nr=case["nr"], n_macro=max(1, case["n_macro"]), charge=1e-9 * u[0],
                                 E_cathode=100e6 * u[1], B_peak=0.25 * u[2], B_z=0.01 if case["te"] else 0.1,
                                 step_interval=case["interval"], seed=seed)


def _state(case, seed):
    """Fields and beam of a run, as host containers."""
    cfg = _config(case, seed)
    f = geometry.fields_for(cfg.nz, cfg.nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=_modes(case))
    f.mesh.dt = cfg.dt
    if case["workload"] != "dcgun":
        f["Ez"] = cfg.initial_ez(f.flags)
        if case["workload"] == "gun":
            bz, br = cfg.solenoid()
            f["BzImposed"], f["BrImposed"] = bz, br
    n = case["n_macro"]
    b = abi.Beam(max(1, n))
    if n:
        b.set(n, **cfg.beam_arrays())
    b.npActive, b.nextParticleID, b.QoMC, b.stiffness = n, n + 1, QOMC, 1.0
    return cfg, f, b


def _antenna(case):
    """Direction, nodes, current and phase of the cavity's drive: a line of
    axial current in the full cell, half way to the wall."""
    nz, nr = case["nz"], case["nr"]
    return 0, int(nz * 0.25), int(nz * 0.40), nr // 2, 1e6, RF_HZ, 0.3


def _poisson(case):
    return abi.poisson_options(step_interval=case["interval"], accuracy=1e-6, maximum_iterations=1000)


class _Run:
    """One instance with the host arrays of a stretch's start and end."""

    def __init__(self, case, cfg, f, b):
        n, f64 = case["n_macro"], case["form"] == "f64"
        self.steps, self.n = case["steps"], n
        g = gpu.GpuInstance(f, capacity=max(16, int(1.25 * n)),
                            precision=gpu.PRECISION_F64 if f64 else gpu.PRECISION_SPLIT32)
        if case["ordered"]:
            g.set_deposit_order(1)
        g.add_screen(cfg.screen_z(), 1, capacity=max(16, n))
        if case["workload"] == "cavity":
            t = [-1.0, 0.0, 1.0]
            g.add_antenna(*_antenna(case), t=t, W=np.ones(3))
        g.configure_run(space_charge=1 if n else 0, push=abi.push_options(abi.COMPACT_SWAP, abi.SCREEN_PARTICLE),
                        poisson=_poisson(case) if case["interval"] else None)
        g.upload_beam(b)
        g.run_begin()
        g.synchronize()
        self.g, self.mesh = g, g.get_mesh()
        te = TE_NAMES if case["te"] else ()
        self.up = _holding(f, {k: f.a[k] for k in ("Ez", "Er", "Bphi", "Psi") + te})
        self.down = _holding(f, {k: np.zeros(f.shape) for k in ("Ez", "Er", "Bphi") + te})
        self.beam, self.beam_out = b, _beam_out(max(1, n))
        for k in abi.BEAM_DOUBLES:
            b.a[k] = _pinned(b.a[k])
        b.particleID, b.generation, b.status = _pinned(b.particleID), _pinned(b.generation), _pinned(b.status)

    def begin(self):
        g = self.g
        g.set_mesh(self.mesh)
        g.upload_fields(self.up)
        if self.n:
            g.upload_beam(self.beam)
            g.clear_screens()

    def end(self):
        g = self.g
        g.download_fields(self.down)
        out = dict(self.down.a)
        if self.n:
            g.download_beam(self.beam_out)
            out["beam"] = _by_id(self.beam_out, self.n)
        return out


def _by_id(b, n):
    """The beam's arrays in the order of particle IDs (absent ones zero)."""
    cuda = torch.device("cuda")
    at = torch.from_numpy(b.particleID[: b.np]).to(cuda, non_blocking=True).long() - 1
    out = torch.zeros((len(BEAM_OUT), n), dtype=torch.float64, device=cuda)
    for k, name in enumerate(BEAM_OUT):
        out[k, at] = torch.from_numpy(b.a[name][: b.np]).to(cuda, non_blocking=True)
    return out


def _scan_runs(case, seed):
    """(case, configuration, fields, beam) of each gun of a scan."""
    reqs = [r for r in serve.draw_requests(64, steps=case["steps"], seed=case["draw_seed"]) if r.kind == "gun"]
    for r in reqs[: case["n"]]:
        c = dict(kind="run", form="split32", workload="gun", nz=r.nz, nr=r.nr, n_macro=min(r.n_macro, 200_000),
                 steps=case["steps"], interval=20, te=False, smear=False, ordered=False)
        yield (c,) + _state(c, seed + r.index)


def _request(case, seed):
    u = np.random.default_rng(seed).uniform(0.9, 1.1, 2)
    return serve.ScanRequest(index=0, kind="pillbox", nz=case["nz"], nr=case["nr"], n_macro=case["n_macro"],
                             phase_deg=30.0, peak_field=80e6 * u[0], charge=1e-9 * u[1], solenoid=0.0,
                             steps=case["steps"], seed=1 + seed)


def _charge(case, cfg, seed):
    """A right-hand side as a correction forms it: minus the density of a few
    Gaussian bunches of error charge over epsilon_0, on the update nodes."""
    rng = np.random.default_rng(seed)
    nz, nr = case["nz"], case["nr"]
    z, r = np.arange(nz + 1) * cfg.dz, np.arange(nr + 1) * cfg.dr
    q = np.zeros((nz + 1, nr + 1))
    for _ in range(3):
        z0, sz, sr = rng.uniform(0.05, 0.9) * cfg.zmax, rng.uniform(0.01, 0.05) * cfg.zmax, \
            rng.uniform(0.02, 0.1) * cfg.rmax
        q += rng.normal() * np.exp(-0.5 * ((z - z0) / sz) ** 2)[:, None] * np.exp(-0.5 * (r / sr) ** 2)[None, :]
    return q * (1 + 0.1 * rng.normal(size=q.shape)) * 1e9


def _solve_state(case, seed):
    cfg = workloads.Gun16Config(nz=case["nz"], nr=case["nr"], n_macro=1, seed=seed)
    f = geometry.fields_for(cfg.nz, cfg.nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text())
    f.mesh.dt = cfg.dt
    f["Q"] = _charge(case, cfg, seed)
    return cfg, f


def prepare(case, seed):
    if case["kind"] == "run":
        return case, _Run(case, *_state(case, seed))
    if case["kind"] == "scan":
        return case, [_Run(*args) for args in _scan_runs(case, seed)]
    if case["kind"] == "request":
        return case, _request(case, seed)
    _, f = _solve_state(case, seed)
    f64 = case["form"] == "f64"
    g = gpu.GpuInstance(f, capacity=16, precision=gpu.PRECISION_F64 if f64 else gpu.PRECISION_SPLIT32)
    g.configure_run(space_charge=0, poisson=abi.poisson_options(step_interval=1))
    g.synchronize()
    return case, (g, _holding(f, {k: f.a[k] for k in ("Q", "Psi")}), _holding(f, {"Psi": f.a["Psi"]}))


def run(state):
    case, s = state
    if case["kind"] == "run":
        s.begin()
        s.g.run_steps(s.steps)
        return s.end()
    if case["kind"] == "scan":
        for r in s:
            r.begin()
        gpu.batch_run([r.g for r in s], [r.steps for r in s], workers=4)
        return [r.end() for r in s]
    if case["kind"] == "request":
        g, cfg = serve.build(s, "split32")
        g.run_steps(s.steps)
        f = abi.Fields(cfg.nz, cfg.nr, cfg.zmin, cfg.zmax, cfg.rmax)
        f.a = {k: f.a[k] for k in ("Ez", "Er", "Bphi")}
        g.download_fields(f)
        b = abi.Beam(s.capacity)
        g.download_beam(b)
        g.close()
        return {"fields": dict(f.a), "beam": _by_id(b, s.capacity)}
    g, up, down = s
    g.upload_fields(up)
    n = g.solve_poisson(0, case["accuracy"], case["limit"])
    g.download_fields(down)
    out = {"Psi": down.a["Psi"]}
    if case["form"] == "f64":
        out["iterations"] = n
    return out


# ---------------------------------------------- what a pass cannot do without

def _run_work(c):
    s = 4 if c["form"] == "split32" else 8
    nodes = (c["nz"] + 1) * (c["nr"] + 1)
    fdtd = nodes * (7 * s + 1 + (8 * s if c["te"] else 0))  # E, B read and E, B, half-step B written; a mask
    push = c["n_macro"] * (86 if c["form"] == "split32" else 144)  # position, momentum, charge, extrema, status
    ncorr = 0 if not c["interval"] else (c["steps"] + c["interval"] - 1) // c["interval"]
    corr = nodes * (4 * s + 25)  # Ez, Er read and written, Psi read and written, charge, mask
    io = nodes * 8 * (7 + (6 if c["te"] else 0)) + c["n_macro"] * (16 * 8 + 14 + 7 * 8 + 4)
    return (c["steps"] * (fdtd + push) + ncorr * corr + io,
            c["steps"] * (nodes * (20 + (20 if c["te"] else 0)) + c["n_macro"] * 250) + ncorr * nodes * 150)


def work(case):
    if case["kind"] == "run":
        b, f = _run_work(case)
    elif case["kind"] == "scan":
        b = f = 0
        reqs = [r for r in serve.draw_requests(64, steps=case["steps"], seed=case["draw_seed"]) if r.kind == "gun"]
        for r in reqs[: case["n"]]:
            x = _run_work(dict(form="split32", nz=r.nz, nr=r.nr, n_macro=min(r.n_macro, 200_000),
                               steps=case["steps"], interval=20, te=False))
            b, f = b + x[0], f + x[1]
    elif case["kind"] == "request":
        # the bunch is complete after about a third of the steps
        b, f = _run_work(dict(form="split32", nz=case["nz"], nr=case["nr"], n_macro=case["n_macro"] * 2 // 3,
                              steps=case["steps"], interval=0, te=False))
    else:
        nodes = (case["nz"] + 1) * (case["nr"] + 1)
        b, f = nodes * (25 + 24), nodes * 150  # rhs and Psi in, Psi out, and their copies
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """About four times the largest difference seen from ``exact`` over the
    listed cases and a score of drawn ones (2-norm, and largest over rms)."""
    if case["kind"] == "solve":
        # a multigrid solve ends anywhere below the stop rule: 0.6 x the
        # accuracy at most; the FP64 relaxation is the same sums bit for bit
        a = case["accuracy"]
        return {"rel": 1e-13} if case["form"] == "f64" else {"rel": 2 * a, "max": 8 * a}
    if case.get("form") == "f64":
        # 1.6e-14 and 4.4e-13: the order of sums in FP64
        return {"rel": 1e-13, "max": 2e-12}
    if case.get("workload") == "cavity":
        # 7.8e-6 (Er, small beside Ez) and 2.4e-4 after 400 FP32 steps
        return {"rel": 3e-5, "max": 1e-3}
    if case.get("workload") == "dcgun":
        # Bphi, near zero in an electrostatic gun, carries the rounding of E
        # that every step's correction moves: 4e-4 and 0.23 (E itself 5e-6)
        return {"rel": 2e-3, "max": 0.9}
    # 3.4e-5 and 3.2e-4 on the scan's small meshes (2e-6 on the benchmark's)
    return {"rel": 1.4e-4, "max": 2e-3}


# ------------------------------------------------- the same results in 64 bits

class _Plain:
    """The loop in plain FP64 torch: Yee update, area-weighted gather, leapfrog
    push, deposition and Poisson correction on conducting end walls."""

    def __init__(self, case, f, b):
        self.dev = torch.device("cuda")
        m = self.m = f.mesh
        self.case, self.nz, self.nr, self.dz, self.dr, self.dt = case, m.nz, m.nr, m.dz, m.dr, m.dt
        T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        self.fl = T(f.flags.astype(np.int32))
        self.F = {k: T(v) for k, v in f.a.items()}
        nz, nr, dz, dr = self.nz, self.nr, self.dz, self.dr
        ir = np.arange(nr + 1)
        iz = torch.arange(nz + 1, device=self.dev)[:, None]
        # rows stop after the first node flagged as the last active one
        last = (f.flags & abi.FL_LAST_ACTIVE_PT) != 0
        self.cut = [T(np.array([next((i for i in range(k, nz) if last[i, j]), nz - 1) for j in range(nr + 1)])
                      if last.any() else np.full(nr + 1, nz - 1))[None, :] for k in (0, 1)]
        jr = torch.arange(nr + 1, device=self.dev)[None, :]
        no = lambda bit: (self.fl & bit) == 0  # noqa: E731
        inner = (iz >= 1) & (iz <= nz - 1)
        self.mEz = inner & (jr < nr - 1) & (iz <= self.cut[1]) & no(abi.FL_EZ_ZERO)
        self.mEr = (iz <= nz - 1) & (jr >= 1) & (jr <= nr - 1) & (iz <= self.cut[0]) & no(abi.FL_ER_ZERO)
        self.mB = inner & (jr >= 1) & (jr <= nr - 2) & (iz <= self.cut[1]) & no(abi.FL_BPHI_ZERO)
        self.mEphi = (iz <= nz - 1) & (jr >= 1) & (jr <= nr - 1) & (iz <= self.cut[0]) & no(abi.FL_EPHI_ZERO)
        self.mBr = inner & (jr <= nr - 1) & (iz <= self.cut[1]) & no(abi.FL_BR_ZERO)
        self.mBz = (iz <= nz - 1) & (jr >= 1) & (jr <= nr - 1) & (iz <= self.cut[0]) & no(abi.FL_BZ_ZERO)
        k = 1 / (EPS0 * MU0)
        rp, rm = (ir + 0.5) * dr, (ir - 0.5) * dr
        cp = np.where(ir > 0, rp * 2 * k / np.where(ir > 0, rp ** 2 - rm ** 2, 1), 4 * k / dr)
        cm = np.where(ir > 0, rm * 2 * k / np.where(ir > 0, rp ** 2 - rm ** 2, 1), 0)
        self.cp, self.cm = T(cp)[None, :], T(cm)[None, :]
        self.bzf = T(-2 * m.dt / (dr * ((ir + 1.0) ** 2 - ir ** 2)))[None, :]
        self.topf = (m.rmax - dr / 2) / (m.rmax + dr / 2)
        self.metal = (self.fl & abi.FL_IS_METAL) != 0
        self.unk = (iz >= 1) & (iz <= nz - 2) & (jr < nr - 1) & ~self.metal
        # cell areas and volumes of the charge balance
        self.Ari = T(np.where(ir > 0, math.pi * (2 * ir - 1) * dr * dz, math.pi * dr * dz))[None, :]
        self.Aro = T(np.where(ir > 0, math.pi * (2 * ir + 1) * dr * dz, math.pi * dr * dz))[None, :]
        self.Az = T(np.where(ir > 0, math.pi * dr * dr * 2 * ir, math.pi * dr * dr / 4))[None, :]
        with np.errstate(divide="ignore"):
            self.crow = T(np.where(ir > 0, 1 / dr ** 2 * (1 + 1. / (2 * ir)), 4 / dr ** 2))[None, :]
            self.drow = T(np.where(ir > 0, 1 / dr ** 2 * (1 - 1. / (2 * ir)), 0))[None, :]
        e = -2 * (1 / dz ** 2 + 1 / dr ** 2)
        self.e = T(np.where(ir > 0, e, e - 2 / dr ** 2))[None, :]
        self.vol = T(np.where(ir > 0, ir, 0.125))[None, :]
        self.imposed = None
        n = self.n = b.np
        self.B = {x: T(b.a[x][:n]) for x in abi.BEAM_DOUBLES}
        self.lost = False

    def z(self):
        return torch.zeros((self.nz + 1, self.nr + 1), dtype=torch.float64, device=self.dev)

    # -- Poisson
    def apply(self, p):
        """The five-point cylindrical operator (zero on the border)."""
        out = self.z()
        c = slice(1, self.nz)
        out[c, 1:-1] = (p[2:, 1:-1] + p[:-2, 1:-1]) / self.dz ** 2 + self.crow[:, 1:-1] * p[c, 2:] + \
            self.drow[:, 1:-1] * p[c, :-2] + self.e[:, 1:-1] * p[c, 1:-1]
        out[c, 0] = (p[2:, 0] + p[:-2, 0]) / self.dz ** 2 + self.crow[0, 0] * p[c, 1] + self.e[0, 0] * p[c, 0]
        return out

    def solve(self, p, rhs, tol=1e-12, most=20000):
        """A p = rhs on the update nodes, by conjugate gradients."""
        u = self.unk
        r = torch.where(u, -self.vol * (rhs - self.apply(p)), 0.0)
        d = -(self.vol * self.e)
        zz = r / d
        q, rz = zz.clone(), (r * zz).sum()
        stop = tol * torch.where(u, self.vol * rhs, 0.0).norm()
        for k in range(most):
            Aq = torch.where(u, -self.vol * self.apply(q), 0.0)
            al = rz / (q * Aq).sum()
            p = p + al * q
            r = r - al * Aq
            if k % 50 == 0 and bool(r.norm() <= stop):
                break
            zz = r / d
            new = (r * zz).sum()
            q, rz = zz + (new / rz) * q, new
        return p

    def sor(self, p, rhs, accuracy, limit):
        """Red-black over-relaxation with Chebyshev factors, to the stop rule
        sum|r| < accuracy sum|rhs| over a colour, or the limit."""
        nz, nr = self.nz, self.nr
        k = self.dz / self.dr
        rj = (math.cos(math.pi / nz) + k * k * math.cos(math.pi / nr)) / (1 + k * k)
        par = (torch.arange(nz + 1, device=self.dev)[:, None] + torch.arange(nr + 1, device=self.dev)[None, :]) % 2
        mask = [self.unk & (par == c) for c in (0, 1)]
        thr = accuracy * float(rhs[:nz, : nr - 1].abs().sum()) if rhs is not None else 0.0
        om = 1.0
        for n in range(limit):
            res = torch.where(mask[n & 1], self.apply(p) - (rhs if rhs is not None else 0.0), 0.0)
            p = p - om * res / self.e
            total = float(res.abs().sum()) if n else math.inf
            if n and (total < thr or total == 0):
                return p, n
            om = 1 / (1 - rj * rj / 2) if n == 0 else 1 / (1 - rj * rj * om / 4)
        return p, -1

    def gradient(self, ez, er, psi, sign):
        """ez, er + sign grad psi, with the boundary copies."""
        nz, nr = self.nz, self.nr
        g = self.z()
        g[1:nz, :nr] = (psi[1:nz, :nr] - psi[: nz - 1, :nr]) / self.dz
        ez = torch.where((self.fl & abi.FL_EZ_ZERO) == 0, ez + sign * g, ez)
        g = self.z()
        g[:nz, 1:] = (psi[:nz, 1:] - psi[:nz, :-1]) / self.dr
        er = torch.where((self.fl & abi.FL_ER_ZERO) == 0, er + sign * g, er)
        return self.ends_e(ez, er, nr + 1)

    def ends_e(self, ez, er, top):
        nz, nr = self.nz, self.nr
        ez[1:nz, nr - 1] = 0
        ez[0, :nr], ez[nz, :nr] = ez[1, :nr], ez[nz - 1, :nr]
        er[0, 1:top], er[nz - 1, 1:top] = 0, 0
        er[0, nr], er[nz - 1, nr] = 0, 0
        er[:nz, 0] = -er[:nz, 1]
        return ez, er

    def correct(self):
        F, nz, nr, B = self.F, self.nz, self.nr, self.B
        q = self.z()
        ez, er = F["Ez"], F["Er"]
        flux = er[:nz, 1:] * self.Aro[:, :-1] + (ez[1:, :nr] - ez[:nz, :nr]) * self.Az[:, :nr]
        flux[:, 1:] -= er[:nz, 1:nr] * self.Ari[:, 1:nr]
        q[:nz, :nr] = EPS0 * flux
        q[self.metal] = 0
        q[0], q[nz - 1], q[:, nr - 1] = 0, 0, 0
        if self.n:
            sm = self.case["smear"]
            xz, xr = B["z"] / self.dz + (0 if sm else 0.5), B["r"] / self.dr + (0 if sm else 0.5)
            iz, jr = xz.long(), xr.long()
            fz, fr = (xz - iz, xr - jr) if sm else (torch.zeros_like(xz), torch.zeros_like(xr))
            for a in (0, 1):
                for c in (0, 1):
                    w = (fz if a else 1 - fz) * (fr if c else 1 - fr)
                    # a particle of the first row leaves its charge on the wall
                    ok = ~self.metal[iz + a, jr + c] & (iz > 0)
                    q.view(-1).index_add_(0, (iz + a) * (nr + 1) + jr + c, torch.where(ok, -B["Q"] * w, 0.0))
        rhs = -q / (self.Az * self.dz * EPS0)
        if self.case["form"] == "f64":
            F["Psi"], _ = self.sor(F["Psi"], rhs, 1e-6, 1000)
        else:
            F["Psi"] = self.solve(F["Psi"], rhs)
        F["Ez"], F["Er"] = self.gradient(ez.clone(), er.clone(), F["Psi"], 1.0)

    # -- fields
    def fdtd(self, J):
        F, nz, nr, dt, dz, dr = self.F, self.nz, self.nr, self.dt, self.dz, self.dr
        b = F["Bphi"]
        d = self.z()
        d[:, :-1] = self.cp[:, :-1] * b[:, 1:] - self.cm[:, :-1] * b[:, :-1]
        ez = torch.where(self.mEz, F["Ez"] + dt * (d - J[0] / EPS0), F["Ez"])
        d = self.z()
        d[:-1] = (b[1:] - b[:-1]) / (MU0 * EPS0 * dz)
        er = torch.where(self.mEr, F["Er"] - dt * (d + J[1] / EPS0), F["Er"])
        F["Ez"], F["Er"] = ez, er = self.ends_e(ez, er, nr)
        d = self.z()
        d[1:, 1:] = dt * ((ez[1:, 1:] - ez[1:, :-1]) / dr - (er[1:, 1:] - er[:-1, 1:]) / dz)
        self.Bphi2 = torch.where(self.mB, b + d / 2, 0.0)
        F["Bphi"] = torch.where(self.mB, b + d, b)
        for a in (F["Bphi"], self.Bphi2):
            a[1:nz, 0] = -a[1:nz, 1]
            a[1:nz, nr - 1] = a[1:nz, nr - 2] * self.topf
            a[0], a[nz] = a[1], a[nz - 1]
        if not self.case["te"]:
            return
        br, bz = F["Br"], F["Bz"]
        d = self.z()
        d[:-1, :-1] = (br[1:, :-1] - br[:-1, :-1]) / dz - (bz[:-1, 1:] - bz[:-1, :-1]) / dr
        e = torch.where(self.mEphi, F["Ephi"] + dt * (d / (EPS0 * MU0) - J[2] / EPS0), F["Ephi"])
        e[:, 0] = 0
        e[0] = e[nz - 1] = 0
        e[:, nr - 1] = 0
        F["Ephi"] = e
        d = self.z()
        d[1:] = dt * (e[1:] - e[:-1]) / dz
        self.Br2 = torch.where(self.mBr, br + d / 2, 0.0)
        F["Br"] = torch.where(self.mBr, br + d, br)
        for a in (F["Br"], self.Br2):
            a[0], a[nz] = a[1], a[nz - 1]
        jr = torch.arange(nr + 1, device=self.dev, dtype=torch.float64)[None, :]
        d = self.z()
        d[:, 1:] = (self.bzf * (jr + 1))[:, 1:] * e[:, 1:] - (self.bzf * jr)[:, 1:] * e[:, :-1]
        self.Bz2 = torch.where(self.mBz, bz + d / 2, 0.0)
        F["Bz"] = torch.where(self.mBz, bz + d, bz)
        for a in (F["Bz"], self.Bz2):
            a[0], a[nz - 1] = 0, 0
            a[:, 0] = a[:, 1]

    # -- particles
    def deposit(self):
        B, nz, nr, sm = self.B, self.nz, self.nr, self.case["smear"]
        out = []
        for comp, v in enumerate(("vz", "vr", "vphi")):
            J = self.z()
            out.append(J)
            if not self.n or (comp == 2 and not self.case["te"]):
                continue
            xz = B["z"] / self.dz + ((0.5 if comp == 0 else 0.0) if sm else (1.0 if comp == 0 else 0.5))
            xr = B["r"] / self.dr + ((0.5 if comp == 1 else 0.0) if sm else (1.0 if comp == 1 else 0.5))
            iz, jr = xz.long(), xr.long()
            q = B[v] * B["Q"] / (math.pi * self.dz * self.dr ** 2)
            fz, fr = xz - iz, xr - jr
            if comp == 0:
                fz = torch.where(iz == 0, torch.ones_like(fz), fz)
            k = jr.double()
            if comp == 1:
                wm, wp = torch.where(jr > 0, 1 / (2 * k - 1), 0.0), 1 / (2 * k + 1)
                wp0 = torch.ones_like(k)
            else:
                wm, wp = torch.where(jr > 0, 1 / (2 * k), 4.0), 1 / (2 * k + 2)
                wp0 = fr
            if sm:
                wm, wp = wm * (1 - fr), wp * torch.where(jr > 0, fr, wp0)
            for a in (0, 1) if sm else (0,):
                w = (fz if a else 1 - fz) if sm else 1.0
                for c in (0, 1) if sm else (0,):
                    J.view(-1).index_add_(0, (iz + a) * (nr + 1) + jr + c, q * w * (wp if c else wm))
        return out

    def _at(self, a, iz, jr):
        return a.reshape(-1)[iz * (self.nr + 1) + jr]

    def _bil(self, a, iz, iz1, fz, jr, jr1, fr):
        return (1 - fr) * ((1 - fz) * self._at(a, iz, jr) + fz * self._at(a, iz1, jr)) + \
            fr * ((1 - fz) * self._at(a, iz, jr1) + fz * self._at(a, iz1, jr1))

    def gather(self, z, r):
        F, nz, nr = self.F, self.nz, self.nr
        xz, xr = z / self.dz, r / self.dr
        iz0, ir0 = xz.long(), xr.long()
        izh, irh = (xz + 0.5).long(), (xr + 0.5).long()
        fz0, fr0, fzh, frh = xz - iz0, xr - ir0, xz + 0.5 - izh, xr + 0.5 - irh
        on = r != 0
        bit = lambda i, j, b: (self._at(self.fl, i, j) & b) != 0  # noqa: E731
        # Ez and Br: half nodes in z; a row of metal on either side is left out
        a, a1 = izh, (izh + 1).clamp(max=nz - 1)
        c1 = (ir0 + 1).clamp(max=nr - 1)
        lo = bit(a, ir0 + 1, abi.FL_ER_ZERO) & bit(a, ir0, abi.FL_ER_ZERO)
        up = bit(a1, ir0 + 1, abi.FL_ER_ZERO) & bit(a1, ir0, abi.FL_ER_ZERO)
        am = (a - 1).clamp(min=0)
        back = (a > 0) & ((self._at(self.fl, am, ir0) != 0) | (self._at(self.fl, am, ir0 + 1) != 0))
        na = torch.where(lo & back, a1, a)
        na1 = torch.where(lo & ~back, a, torch.where(~lo & up, a, a1))
        Ez = self._bil(F["Ez"] + F["EzImposed"], na, na1, fzh, ir0, c1, fr0)
        te = self.case["te"]
        Br = torch.where(on, self._bil(self.Br2, na, na1, fzh, ir0, c1, fr0), 0.0) if te else torch.zeros_like(Ez)
        # Er and Bz: half nodes in r
        c = irh.clamp(max=nr - 1)
        lo = bit(iz0 + 1, c, abi.FL_EZ_ZERO) & bit(iz0, c, abi.FL_EZ_ZERO)
        up = bit(iz0 + 1, c + 1, abi.FL_EZ_ZERO) & bit(iz0, c + 1, abi.FL_EZ_ZERO)
        nc, nc1 = torch.where(lo, c + 1, c), torch.where(~lo & up, c, c + 1)
        Er = torch.where(on, self._bil(F["Er"] + F["ErImposed"], iz0, iz0 + 1, fz0, nc, nc1, frh), 0.0)
        Bz = self._bil(self.Bz2, iz0, iz0 + 1, fz0, nc, nc1, frh) if te else torch.zeros_like(Ez)
        Ephi = torch.where(on, self._bil(F["Ephi"], iz0, iz0 + 1, fz0, ir0, c1, fr0), 0.0) if te \
            else torch.zeros_like(Ez)
        Bphi = torch.where(on, self._bil(self.Bphi2, izh, (izh + 1).clamp(max=nz - 1), fzh, c,
                                         (c + 1).clamp(max=nr - 1), frh), 0.0)
        if "BzImposed" in F:
            Bz = Bz + self._bil(F["BzImposed"], iz0, iz0 + 1, fz0, ir0, ir0 + 1, fr0)
            Br = Br + self._bil(F["BrImposed"], iz0, iz0 + 1, fz0, ir0, ir0 + 1, fr0)
        return Ez, Er, Ephi, Bz, Br, Bphi

    def push(self):
        B, dt = self.B, self.dt
        B["zmax"], B["rmax"] = torch.maximum(B["zmax"], B["z"]), torch.maximum(B["rmax"], B["r"])
        z, r = B["z"] + B["vz"] * dt, B["r"] + B["vr"] * dt
        pz, pr, pp = B["pz"], torch.where(r < 0, -B["pr"], B["pr"]), B["r_pphi"]
        r = r.abs()
        iz, jr = (z / self.dz).long(), (r / self.dr).long()
        out = (z < 0) | (z > self.m.zmax) | (r > self.m.rmax)
        iz, jr = iz.clamp(0, self.nz - 1), jr.clamp(0, self.nr - 1)
        inside = (self._at(self.fl, iz, jr) & abi.FL_IS_INSIDE) != 0
        solid = self._at(self.metal, iz, jr) & self._at(self.metal, iz + 1, jr) & \
            self._at(self.metal, iz, jr + 1) & self._at(self.metal, iz + 1, jr + 1)
        if bool((out | inside | solid).any()):
            self.lost = True
            return
        B["zmax"], B["rmax"] = torch.maximum(B["zmax"], z), torch.maximum(B["rmax"], r)
        Ez, Er, Ephi, Bz, Br, Bphi = self.gather(z, r)
        ir = torch.where(r != 0, 1 / torch.where(r != 0, r, 1.0), 0.0)
        pphi = pp * ir
        g = torch.sqrt(pr * pr + pz * pz + pphi * pphi + 1)
        vz, vr, vphi = B["vz"], B["vr"], B["vphi"]
        pr = pr + dt * (pphi * pphi * C / g * ir + QOMC * (Er + vphi * Bz - vz * Bphi))
        pz = pz + dt * QOMC * (Ez + vr * Bphi - vphi * Br)
        pp = pp + dt * QOMC * r * (Ephi + vz * Br - vr * Bz)
        g = torch.sqrt(pz * pz + pr * pr + (pp * ir) ** 2 + 1)
        B.update(z=z, r=r, pz=pz, pr=pr, r_pphi=pp, vz=C * pz / g, vr=C * pr / g, vphi=C * pp * ir / g)

    def steps(self):
        c = self.case
        if c["interval"]:
            # the electrodes' field, as the run's start leaves it
            psi, _ = self.sor(self.F["PsiImposed"], None, 1e-6, 1000) if bool(self.F["PsiImposed"].any()) \
                else (self.F["PsiImposed"], 0)
            self.F["EzImposed"], self.F["ErImposed"] = self.gradient(self.z(), self.z(), psi, -1.0)
        for k in range(c["steps"]):
            J = self.deposit()
            if c["workload"] == "cavity":
                _, i0, i1, at, current, hz, phase = _antenna(c)
                J[0][i0: i1 + 1, at] += current * math.sin(2 * math.pi * hz * (k * self.dt + self.dt / 2) + phase)
            if c["interval"] and k % c["interval"] == 0:
                self.correct()
            self.fdtd(J)
            if self.n:
                self.push()
            if self.lost:
                return None
        out = {k: self.F[k] for k in ("Ez", "Er", "Bphi") + (TE_NAMES if c["te"] else ())}
        if self.n:
            out["beam"] = torch.stack([self.B[k] for k in BEAM_OUT])
        return out


def exact(case, seed):
    if case["kind"] == "run":
        _, f, b = _state(case, seed)
        return _Plain(case, f, b).steps()
    if case["kind"] == "scan":
        return [_Plain(c, f, b).steps() for c, _, f, b in _scan_runs(case, seed)]
    if case["kind"] == "request":
        return None  # its particles come from the library's own random generator
    _, f = _solve_state(case, seed)
    c = dict(case, te=False, smear=False, n_macro=0)
    p = _Plain(c, f, abi.Beam(1))
    if case["form"] == "f64":
        psi, n = p.sor(p.F["Psi"], p.F["Q"], case["accuracy"], case["limit"])
        return {"Psi": psi, "iterations": n}
    return {"Psi": p.solve(p.F["Psi"], p.F["Q"])}
