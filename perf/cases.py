"""Performance cases of the particle loop: what a program does with the
library once it holds a run, through the public entry points.

A case is one of these kinds (``kind``):

* ``steps``   n time steps of one run, then its particles copied back into
              a buffer the program keeps: a run between two of its
              snapshots.  Both forms, the sphere and the spheroid, with and
              without a magnetic field, the other integrators and walls;
* ``dropin``  the drop-in call of one step on the program's own page-locked
              particle records (upload, step, download);
* ``record``  a step that records: potential energies, then the sums behind
              the macroscopic summary and the particles for the state file;
* ``sweep``   many uneven runs advanced together by the batch runtime, then
              its summary and every run's particles;
* ``phi``     the tree of the present particles and the potential along a
              set of directions (the profile file a run writes).

Plasmas are given in Debye lengths (``D`` the domain radius, ``a_rel`` the
grain, ``soft`` the softening, ``dt_w`` the time step times the electron
plasma frequency), with Te = 11,600 K, as in the benchmark configurations;
``si`` marks the program's own defaults, which are given in SI units.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from pot_b200 import configs
from pot_b200.gpu import PARTICLE_DTYPE, Batch, Run, RunConfig

KB, EPS0, QE, ME, MIME = 1.38065e-23, 8.85419e-12, 1.6021766e-19, 9.109383e-31, 1836.15
MI = MIME * ME
PI = 3.14159265358979
TE = 11600.0

# a run's settings; a case overrides what it needs
BASE = dict(form="fast", leaf=16, group=32, D=8.0, a_rel=0.1, te_ti=10.0, mach=0.5, soft=0.01, dt_w=0.005,
            theta=0.5, bz=0.0, A=0.0, integrator=0, dipoles=False, bounce=0.0, grain=True)


def listed():
    return [
        # the smallest runs, in the reference's arithmetic: a step is launches and latency
        dict(name="small_plain", kind="steps", config="small", N=8193, form="plain", leaf=1, group=0, steps=20),
        # a reference-style host loop on a small plasma, one call per step
        dict(name="small_dropin", kind="dropin", config="small", N=8193, form="fast", leaf=8, group=32),
        # the host program at its default flags, between two records
        dict(name="default_fast", kind="steps", config="default", N=150001, form="fast", leaf=16, group=32, steps=20),
        # and one of its record steps
        dict(name="default_record", kind="record", config="default", N=150001, form="fast", leaf=16, group=32),
        # the 1m benchmark plasma, both forms
        dict(name="1m_fast", kind="steps", config="1m", N=1000001, form="fast", leaf=16, group=32, steps=8),
        dict(name="1m_plain", kind="steps", config="1m", N=1000001, form="plain", leaf=1, group=0, steps=2),
        # the largest benchmark plasma: the 4m spheroid with a magnetic field
        dict(name="4m_spheroid_fast", kind="steps", config="4m", N=4000001, form="fast", leaf=16, group=64, steps=8),
        # an oblate grain in the reference's arithmetic, an odd size
        dict(name="oblate_plain", kind="steps", config="family", N=60003, form="plain", leaf=1, group=0, D=12.0,
             a_rel=0.3, A=0.5, bz=0.5, theta=0.4, te_ti=3.0, steps=4),
        # a host loop that keeps its particles and hands them over every step
        dict(name="1m_dropin", kind="dropin", config="1m", N=1000001, form="fast", leaf=16, group=32),
        # a parameter sweep: uneven runs advanced together between two looks at their charges
        dict(name="sweep", kind="sweep", runs=24, nmin=16000, nmax=256000, steps=20),
        # the other compile-time variants: two field evaluations per step, dipole cells, walls, no absorption
        dict(name="verlet_dipoles", kind="steps", config="family", N=30001, integrator=1, dipoles=True, bounce=1.0,
             grain=False, te_ti=3.0, mach=0.0, steps=4),
        # the potential profile of the 1m plasma: 2,200 points, the tree built for them
        dict(name="1m_phi", kind="phi", config="1m", N=1000001, form="fast", leaf=16, group=32, points=2200),
    ]


def _log_int(rng, lo, hi):
    """An odd size, spread over the logarithm (a grain and ion-electron pairs)."""
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "plain", "plain", "dropin", "record", "sweep", "variant", "phi"])
    plasma = dict(config="family", D=rng.uniform(5.0, 12.0), a_rel=math.exp(rng.uniform(math.log(0.05), 0.0)),
                  te_ti=rng.choice([1.0, 3.0, 10.0]), mach=rng.uniform(0.0, 1.0), theta=rng.choice([0.4, 0.5]),
                  soft=rng.choice([0.01, 0.02]))
    if kind == "steps":
        N = _log_int(rng, 8e3, 3e6)
        c = dict(kind="steps", N=N, leaf=rng.choice([8, 16, 16, 32]), group=64 if N > 2000000 else rng.choice([32, 32, 64]),
                 bz=rng.choice([0.0, 0.9]), A=rng.choice([0.0, 0.0, 3.0]), steps=8 if N > 500000 else 20)
    elif kind == "plain":
        N = _log_int(rng, 8e3, 8e5)
        c = dict(kind="steps", N=N, form="plain", leaf=1, group=0, A=rng.choice([0.0, 0.0, 0.5, 3.0]),
                 steps=2 if N > 100000 else 8)
    elif kind == "dropin":
        c = dict(kind="dropin", N=_log_int(rng, 8e3, 2e6), form=rng.choice(["fast", "fast", "plain"]))
    elif kind == "record":
        c = dict(kind="record", N=_log_int(rng, 8e3, 5e5), form=rng.choice(["fast", "plain"]))
    elif kind == "sweep":
        return dict(kind="sweep", runs=rng.randint(8, 32), nmin=8000, nmax=rng.choice([64000, 200000]), steps=10)
    elif kind == "variant":
        c = dict(kind="steps", N=_log_int(rng, 8e3, 6e4), integrator=rng.choice([1, 2]), dipoles=rng.random() < 0.5,
                 bounce=rng.choice([1.0, 0.8]), grain=False, steps=4)
        plasma.update(te_ti=3.0, mach=0.0)
    else:
        c = dict(kind="phi", N=_log_int(rng, 3e4, 2e6), points=rng.randint(50, 20000))
    if c.get("form") == "plain":
        c.update(leaf=1, group=0)
    return dict(plasma, **c)


# ---- the runs ---------------------------------------------------------------
def _family(c):
    """A plasma in Debye lengths: lambda follows from N, Te and D."""
    N = c["N"]
    lam = 3.0 * (N - 1) * QE * QE / (8.0 * PI * EPS0 * KB * TE * c["D"] ** 3)
    R = c["D"] * lam
    w_pe = math.sqrt((N - 1) / ((4.0 / 3.0) * PI * R ** 3) / 2.0 * QE * QE / (EPS0 * ME))
    return RunConfig(N=N, r=1000, mpp=R / 1000.0, a=c["a_rel"] * lam, soft=c["soft"] * lam, dt=c["dt_w"] / w_pe,
                     Te=TE, Ti=TE / c["te_ti"], x_drift=c["mach"] * math.sqrt(KB * TE / MI), theta=c["theta"],
                     B=(0.0, 0.0, c["bz"]), A=c["A"], integrator=c["integrator"], dipoles=c["dipoles"],
                     bounce=c["bounce"], disable_grain=not c["grain"])


def _run_config(case):
    if case["config"] == "default":  # the host program's own defaults, SI units
        return RunConfig(N=case["N"], r=1000, dt=1e-12, mpp=4e-7, soft=2e-8, Te=220.0, Ti=220.0, a=2.5e-6)
    if case["config"] == "family":
        return _family(dict(BASE, **case))
    return configs.run_config(case["config"], case["N"])


def _run(case, seed, init=True):
    c = dict(BASE, **case)
    r = Run(_run_config(case), form=c["form"], leaf_size=c["leaf"], group_size=c["group"], seed=seed, chi_cap=True)
    if init:
        r.init_particles()
    return r


def _records(N):
    """Page-locked particle records, as a program that owns its array has them."""
    return torch.zeros(N * PARTICLE_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(PARTICLE_DTYPE)


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _download(lib, handle, out):
    """pot_gpu_download into the program's own records."""
    rc = lib.pot_gpu_download(handle, _ptr(out), None)
    if rc:
        raise RuntimeError("pot_gpu_download: %s" % lib.pot_gpu_strerror(rc).decode())


def _state(parts):
    """The records as arrays of numbers (views)."""
    w = parts.view(np.float64).reshape(len(parts), 7)
    return dict(pos=w[:, 0:3], vel=w[:, 3:6], species=parts["species"])


def _plasma(cfg, seed, charge):
    """Particles of a quiet plasma with a charged grain at the centre."""
    rng = np.random.default_rng(seed)
    n, R = cfg.N - 1, cfg.r * cfg.mpp
    p = np.zeros(cfg.N, PARTICLE_DTYPE)
    u = rng.normal(size=(n, 3))
    u *= (R * (rng.random(n) * 0.999 + 1e-4) ** (1.0 / 3.0) / np.linalg.norm(u, axis=1))[:, None]
    p["species"][1:] = np.where(np.arange(n) < n // 2, 1, 2)
    s = np.where(p["species"][1:] == 1, math.sqrt(KB * cfg.Ti / MI), math.sqrt(KB * cfg.Te / ME))
    v = rng.normal(size=(n, 3)) * s[:, None]
    for k, a in enumerate("xyz"):
        p[a][0] = R
        p[a][1:] = R + u[:, k]
        p["v" + a][1:] = v[:, k]
    return p, dict(q=charge, m=1.67e-12, pos=(R, R, R))


def _sweep(case, seed):
    """The sweep's runs: size and grain log-uniform, temperature ratio and flow drawn."""
    rng = np.random.default_rng(seed)
    runs = []
    for k in range(case["runs"]):
        # the sizes do not depend on the seed: every sweep of a case is as much work
        N = int(case["nmin"] * (case["nmax"] / case["nmin"]) ** ((k + 0.5) / case["runs"])) | 1
        c = dict(BASE, N=N, a_rel=math.exp(rng.uniform(math.log(0.05), 0.0)),
                 te_ti=float(rng.choice([1.0, 3.0, 10.0, 30.0])), mach=float(rng.uniform(0.0, 2.0)))
        runs.append((_family(c), 16 if N < 100000 else 32))
    return runs


def _points(case, cfg, seed):
    rng = np.random.default_rng(seed)
    R = cfg.r * cfg.mpp
    u = rng.normal(size=(case["points"], 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    return R + u * (np.linspace(0.02, 1.0, case["points"]) * R)[:, None]


# bouncing walls and no absorption: a step without the sampler
def _is_variant(case):
    return case["kind"] == "steps" and dict(BASE, **case)["bounce"] > 0.0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        b = Batch()
        slots, bufs = [], []
        for k, (cfg, leaf) in enumerate(_sweep(case, seed)):
            slots.append(b.admit(cfg, leaf_size=leaf, group_size=32, seed=seed + 1000 + k, chi_cap=True))
            bufs.append(_records(cfg.N))
        return dict(kind=kind, batch=b, slots=slots, bufs=bufs, steps=case["steps"])
    if _is_variant(case):
        run = _run(case, seed, init=False)
        parts, grain = _plasma(run.cfg, seed, -200)
        run.upload(parts, grain)
    elif kind == "phi":
        run = _run(case, seed, init=False)
        parts, grain = _plasma(run.cfg, seed, -2000)
        run.upload(parts, grain)
        return dict(kind=kind, run=run, xyz=_points(case, run.cfg, seed))
    else:
        run = _run(case, seed)
    s = dict(kind=kind, run=run, steps=case.get("steps", 1))
    if kind in ("steps", "dropin", "record"):
        s["parts"] = _records(case["N"])
    if kind == "dropin":
        _download(run.lib, run.h, s["parts"])
        s["grain"] = run.grain()
    return s


def run(state):
    kind = state["kind"]
    if kind == "sweep":
        b = state["batch"]
        b.step(state["steps"])
        rows = b.summary()
        h = ctypes.c_void_p()
        out = []
        for slot, buf in zip(state["slots"], state["bufs"]):
            b.lib.pot_batch_ctx(b.h, slot, ctypes.byref(h))
            _download(b.lib, h, buf)
            w = buf.view(np.float64).reshape(len(buf), 7)
            out.append(w[:, 0:6])
        return dict(q=rows["grain_q"], t=rows["t_steps"], absorbed=rows["tot_absor_e"], state=out)
    r = state["run"]
    if kind == "steps":
        st = r.step(state["steps"])
        _download(r.lib, r.h, state["parts"])
        return dict(_state(state["parts"]), q=st["grain_q"], pushed=st["n_pushed"], cells=st["n_nodes"])
    if kind == "dropin":
        state["grain"], st = r.move_particles(state["parts"], state["grain"])
        return dict(_state(state["parts"]), q=st["grain_q"], pushed=st["n_pushed"], cells=st["n_nodes"])
    if kind == "record":
        st = r.step(1, epe=True)
        sums = r.macro()
        _download(r.lib, r.h, state["parts"])
        return dict(_state(state["parts"]), epe=st["epe"], sums=sums, q=st["grain_q"])
    cells = r.build_tree()
    return dict(phi=r.phi_at(state["xyz"]), cells=cells)


# ---- what a pass cannot do without ------------------------------------------
def _step_work(N, theta, fields=1):
    """One step: every particle's position and velocity read for the tree, the
    electrons' state read and written, and the terms of a walk (17 flops
    each), about 46 log2 N of them at an opening angle of 0.5."""
    due = (N - 1) / 2.0
    terms = 46.0 * math.log2(N) * (0.5 / theta) ** 2
    return 48.0 * N + 96.0 * due, 17.0 * terms * due * fields


def work(case):
    c = dict(BASE, **case)
    if c["kind"] == "sweep":
        b = f = 0.0
        for cfg, _ in _sweep(case, 1):
            sb, sf = _step_work(cfg.N, 0.5)
            b += sb * c["steps"] + 56.0 * cfg.N
            f += sf * c["steps"]
        return dict(bytes=b, flops=f)
    theta = _run_config(case).theta
    sb, sf = _step_work(c["N"], theta, 2 if c["integrator"] else 1)
    if c["kind"] == "steps":
        return dict(bytes=sb * c["steps"] + 56.0 * c["N"], flops=sf * c["steps"])
    if c["kind"] == "dropin":  # all records up, the electrons' back
        return dict(bytes=sb + 56.0 * 1.5 * c["N"], flops=sf)
    if c["kind"] == "record":  # the step, every particle's potential, the state for the sums and copied back
        return dict(bytes=sb + (48.0 + 56.0) * c["N"], flops=3.0 * sf)
    return dict(bytes=24.0 * c["N"] + 32.0 * c["points"],
                flops=8.0 * 46.0 * math.log2(c["N"]) * (0.5 / theta) ** 2 * c["points"])


# ---- the same in 64 bits, by direct sums ------------------------------------
def _direct_field(x, q, at, idx, soft):
    """Softened Coulomb field of charges q (elementary) at x, at the points
    `at`, each leaving out the source idx."""
    k = QE / (4.0 * PI * EPS0)
    out = torch.empty_like(at)
    step = max(1, 60000000 // len(x))
    for i in range(0, len(at), step):
        d = at[i:i + step, None, :] - x[None, :, :]
        r2 = (d * d).sum(-1) + soft * soft
        w = q[None, :] * r2 ** -1.5
        w[torch.arange(len(d), device=x.device), idx[i:i + step]] = 0.0
        out[i:i + step] = k * (w[:, :, None] * d).sum(1)
    return out


def _exact_variant(case, seed):
    """Velocity Verlet / midpoint steps between bouncing walls, no absorption."""
    cfg = _run_config(case)
    c = dict(BASE, **case)
    p, grain = _plasma(cfg, seed, -200)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(np.stack([p[a] for a in "xyz"], 1), device=dev)
    v = torch.tensor(np.stack([p["v" + a] for a in "xyz"], 1), device=dev)
    sp = torch.tensor(p["species"].astype(np.int64), device=dev)
    q = torch.where(sp == 1, 1.0, -1.0).double()
    q[0] = float(grain["q"])
    m = torch.where(sp == 1, MI, ME).double()
    R = cfg.r * cfg.mpp
    tss_i = int(math.sqrt(cfg.Te * MI / (cfg.Ti * ME)))
    for t in range(1, c["steps"] + 1):
        due = sp == 2
        if t % tss_i == 0:
            due |= sp == 1
        i = torch.nonzero(due)[:, 0]
        dt = torch.where(sp[i] == 1, cfg.dt * tss_i, cfg.dt).double()[:, None]
        qm = (QE * q[i] / m[i])[:, None]
        x0, v0 = x[i].clone(), v[i].clone()
        a1 = qm * _direct_field(x, q, x0, i, cfg.soft)
        vh = v0 + 0.5 * dt * a1
        xm = x0 + (0.5 * dt * v0 if c["integrator"] == 2 else dt * vh)
        xs = x.clone()
        xs[i] = xm
        a2 = qm * _direct_field(xs, q, xm, i, cfg.soft)
        if c["integrator"] == 2:
            xn, vn = x0 + dt * vh, v0 + dt * a2
        else:
            xn, vn = xm, vh + 0.5 * dt * a2
        # the wall turns the radial velocity of a leaving particle round and puts the particle back
        r = xn - R
        d = r.norm(dim=1, keepdim=True)
        n = r / d
        vr = (vn * n).sum(1, keepdim=True)
        hit = (d > R) & (vr > 0.0)
        vn = torch.where(hit, c["bounce"] * (vn - 2.0 * vr * n), vn)
        xn = torch.where(hit, x0, xn)
        x[i], v[i] = xn, vn
    return dict(pos=x.cpu().numpy(), vel=v.cpu().numpy(), species=p["species"].copy(), q=None, pushed=None, cells=None)


def _exact_phi(case, seed):
    """Softened Coulomb potential of every particle at the profile's points."""
    cfg = _run_config(case)
    p, grain = _plasma(cfg, seed, -2000)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(np.stack([p[a] for a in "xyz"], 1), device=dev)
    q = torch.tensor(np.where(p["species"] == 1, 1.0, -1.0), device=dev)
    q[0] = float(grain["q"])
    at = torch.tensor(_points(case, cfg, seed), device=dev)
    phi = torch.empty(len(at), dtype=torch.float64, device=dev)
    step = max(1, 60000000 // len(x))
    for i in range(0, len(at), step):
        r2 = ((at[i:i + step, None, :] - x[None, :, :]) ** 2).sum(-1) + cfg.soft ** 2
        phi[i:i + step] = (q[None, :] * r2 ** -0.5).sum(1) * (QE / (4.0 * PI * EPS0))
    return dict(phi=phi.cpu().numpy(), cells=None)


def exact(case, seed):
    # a reinjected particle comes from the library's own random streams, and a
    # magnetic field or large plasma is more than a direct sum can give quickly
    if _is_variant(case) and dict(BASE, **case)["bz"] == 0.0 and case["N"] < 70000:
        return _exact_variant(case, seed)
    if case["kind"] == "phi" and case["N"] * case["points"] < 4e9:
        return _exact_phi(case, seed)
    return None
