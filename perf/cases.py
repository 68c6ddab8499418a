"""The work that users of this framework have it do, as cases for timing.

A pass is a stretch of the time loop and what a program reads after it: the
running spectra of its monitors (into buffers it keeps) and, on the small
grids, a frame of one field.  The kinds:

  line      the 1D programs: a gold slab in vacuum with a soft source, or
            (tfsf) the layered stack of the 1D reference program with its
            incident line; slab PML at both ends
  plane     2D, TMz or TE: gold cylinders, a dielectric substrate on request,
            split-field PML on all faces, a line source, two line monitors.
            With host_loop the steps go through the per-procedure entry points,
            as a Fortran host program drives them
  program2  the 2D reference program (125 x 1266, TE, x periodic, y-slab PML)
  program3  the 3D reference program (125 x 1266 x 25)
  sphere    3D: a gold sphere, split-field PML on all faces, a plane source,
            the tangential fields on a box around the sphere
  column    3D, laterally periodic: a nonlinear graphene sheet, PML along z, the
            plane mean of the transmitted field
  serve     a server given a batch of small jobs: set-up, steps and results

Fields start from seeded wave packets (a restart, an initial-value problem),
so that every cell works on ordinary values from the first step.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, "fortran-mpi-fdtd_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from fdtd_gpu import Job, Server, abi, problems  # noqa: E402
from fdtd_gpu.spec import JobSpec, box, monitor_shape, spheres  # noqa: E402

EP0 = 8.85418781762039e-12
MU0 = math.pi * 4e-7
C0 = 1.0 / math.sqrt(EP0 * MU0)
GOLD = dict(eps_inf=1.1431, omega_d=1.3202e16, gamma_d=1.0805e14, amp=(0.26698, 3.0834), phi=(-1.2371, -1.0968),
            omega=(3.8711e15, 4.1684e15), gamma=(4.4642e14, 2.3555e15))
GOLD_PROGRAM = dict(GOLD, gamma=(4.4642e14, 2.4555e15))  # the reference programs' value of the second damping
GRAPHENE = dict(fermi_ev=0.4, tau=0.1e-12, temperature=300.0, chi3=1e-18, raman_frac=0.3, raman_freq=47.4e12,
                raman_tau=1e-12, thickness=2e-9, e_scale=1.0)
SUBSTRATE = 1.46 ** 2


def listed():
    return [
        # 1D: the 4000-cell gold slab line, and the reference's 13004-cell stack in its own precision
        {"name": "line_gold_f32", "kind": "line", "cells": 4000, "tfsf": False, "f64": False, "steps": 2048},
        {"name": "line_stack_f64", "kind": "line", "cells": 13004, "tfsf": True, "f64": True, "steps": 1024},
        # small 2D: one member of a parameter sweep; one frame of the 2D reference program (every 684 steps);
        # an odd-sized TE grid on a substrate; a host program's own loop, a procedure at a time
        {"name": "tm_256_f32", "kind": "plane", "te": False, "nx": 256, "ny": 256, "npml": 16, "cylinders": 6,
         "substrate": False, "f64": False, "steps": 512, "nfreq": 64, "host_loop": False},
        {"name": "te_program_f64", "kind": "program2", "f64": True, "steps": 684},
        {"name": "te_odd_f32", "kind": "plane", "te": True, "nx": 611, "ny": 407, "npml": 20, "cylinders": 8,
         "substrate": True, "f64": False, "steps": 200, "nfreq": 64, "host_loop": False},
        {"name": "host_loop_f32", "kind": "plane", "te": False, "nx": 512, "ny": 512, "npml": 16, "cylinders": 10,
         "substrate": False, "f64": False, "steps": 16, "nfreq": 64, "host_loop": True},
        # the benchmark's 2D workload, and the largest 2D grid
        {"name": "tm_2048_f32", "kind": "plane", "te": False, "nx": 2048, "ny": 2048, "npml": 32, "cylinders": 40,
         "substrate": False, "f64": False, "steps": 512, "nfreq": 100, "host_loop": False},
        {"name": "tm_8192_f32", "kind": "plane", "te": False, "nx": 8192, "ny": 8192, "npml": 32, "cylinders": 160,
         "substrate": False, "f64": False, "steps": 64, "nfreq": 32, "host_loop": False},
        # 3D: the benchmark's sphere (the largest grid) and graphene column, and the 3D reference program
        {"name": "sphere_512_f32", "kind": "sphere", "nx": 512, "ny": 512, "nz": 512, "npml": 16, "f64": False,
         "steps": 64, "nfreq": 16},
        {"name": "column_f32", "kind": "column", "nxy": 256, "nz": 384, "f64": False, "steps": 96, "nfreq": 128},
        {"name": "program3_f64", "kind": "program3", "f64": True, "steps": 64},
        # a batch of the serving mix
        {"name": "serve_batch_f32", "kind": "serve", "jobs2": 6, "jobs3": 1, "n2": 256, "n3": 96, "f64": False,
         "steps": 512, "nfreq": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("line", "line", "plane", "plane", "plane", "plane", "sphere", "sphere", "column", "program2",
                       "host", "serve"))
    f64 = rng.random() < 0.25
    if kind == "line":
        tfsf = rng.random() < 0.5
        return {"kind": "line", "cells": _log(rng, 1200, 20000), "tfsf": tfsf, "f64": rng.random() < 0.5,
                "steps": rng.randint(300, 2200)}
    if kind in ("plane", "host"):
        nx, ny = _log(rng, 160, 4096), _log(rng, 160, 4096)
        if rng.random() < 0.6:
            nx = max(160, nx // 4 * 4)
        host = kind == "host"
        cells = nx * ny * (4 if f64 else 1)
        return {"kind": "plane", "te": rng.random() < 0.4, "nx": nx, "ny": ny, "npml": rng.choice((10, 16, 20, 32)),
                "cylinders": rng.randint(1, 24), "substrate": rng.random() < 0.4, "f64": f64,
                "steps": rng.randint(4, 24) if host else max(40, min(rng.randint(200, 600), int(2e9 / cells))),
                "nfreq": rng.randint(16, 100), "host_loop": host}
    if kind == "sphere":
        top = 160 if f64 else 320
        return {"kind": "sphere", "nx": _log(rng, 72, top), "ny": _log(rng, 72, top),
                "nz": _log(rng, 72, top), "npml": rng.choice((8, 12, 16)), "f64": f64, "steps": rng.randint(40, 110),
                "nfreq": rng.randint(8, 32)}
    if kind == "column":
        return {"kind": "column", "nxy": _log(rng, 8, 200), "nz": rng.randint(96, 400), "f64": f64,
                "steps": rng.randint(40, 160), "nfreq": rng.randint(16, 128)}
    if kind == "program2":
        return {"kind": "program2", "f64": f64, "steps": rng.randint(100, 800)}
    return {"kind": "serve", "jobs2": rng.randint(2, 10), "jobs3": rng.randint(0, 2), "n2": _log(rng, 160, 480),
            "n3": rng.randint(64, 112), "f64": f64, "steps": rng.randint(200, 600), "nfreq": rng.randint(16, 48)}


# ---- geometry ----------------------------------------------------------------
def _sigma(npml, ds):
    return 4.0 * C0 * 16.0 / (2.0 * npml * ds)


def _omegas(lam_a, lam_b, nf):
    fa, fb = C0 / lam_b, C0 / lam_a
    return 2.0 * math.pi * (fa + (fb - fa) / nf * np.arange(nf))


def _pulse(lam, st, lead):
    return dict(t0=lead * st, st=st, w0=2.0 * math.pi * C0 / lam)


def _prec(case):
    return abi.F64 if case["f64"] else abi.F32


def _cylinders(rng, nx, ny, npml, count):
    out = []
    scale = min(nx, ny) / 2048.0
    rmax = max(6.0, 40.0 * min(1.0, 1.6 * scale))
    for _ in range(200 * count):
        if len(out) == count:
            break
        r = float(int(rng.uniform(4.0, rmax)))
        cx = float(rng.uniform(npml + r + 4, nx - npml - r - 4))
        cy = float(rng.uniform(npml + r + 24, ny - npml - r - 12))
        if all(math.hypot(cx - x, cy - y) > r + q + 2 for x, y, _, q in out):
            out.append((cx, cy, 0.0, r))
    return out


def _plane(case, rng):
    """A 2D job: its spec, with sources and monitors as the 2D benchmark has them."""
    nx, ny, npml, te = case["nx"], case["ny"], case["npml"], case["te"]
    ds = 1e-9
    spec = JobSpec(layout=abi.LAYOUT_2D_TE if te else abi.LAYOUT_2D_TM, n=(nx, ny, 1), ku=0.5, dt=0.5 * ds / C0, ds=ds,
                   precision=_prec(case), main_lo=(npml, npml, 0), main_hi=(nx - npml - 1, ny - npml - 1, 0))
    spec.add_dielectric(box((0, 0, 0), (nx - 1, ny - 1, 0)), 1.0)
    sub = ny - npml - ny // 4
    if case["substrate"]:
        spec.add_dielectric(box((npml, sub, 0), (nx - npml - 1, ny - npml - 1, 0)), SUBSTRATE)
    cyl = _cylinders(rng, nx, ny, npml, case["cylinders"])
    if cyl:
        spec.add_gold(spheres(cyl), GOLD)
    spec.pml = dict(mode=abi.PML_SPLIT, npml=((npml, npml), (npml, npml), (0, 0)), eps_lo=1.0,
                    sigma_max=_sigma(npml, ds), order=3.0)
    e, h = (abi.EX, abi.HZ) if te else (abi.EZ, abi.HX)
    ys, yin, yt = npml + 4, npml + 12, ny - npml - 5
    spec.sources.append(dict(component=e, lo=(0, ys, 0), hi=(nx - 1, ys, 0), amp=1.0, **_pulse(600e-9, 0.5e-15, 1.5)))
    om = _omegas(500e-9, 800e-9, case["nfreq"])
    for y in (yin, yt):
        spec.add_monitor((0, y, 0), (nx - 1, y, 0), (e, h), om)
    if case["host_loop"]:
        spec.add_probe((nx // 2, yin, 0), (e, h))
    return spec, dict(cyl=cyl, sub=sub if case["substrate"] else None, gold=GOLD)


def _line(case, rng):
    """A 1D job: a gold slab in vacuum, or the reference program's stack with its incident line."""
    n, tfsf = case["cells"], case["tfsf"]
    ds, npml = 1e-9, 10 if tfsf else 20
    spec = JobSpec(layout=abi.LAYOUT_1D, n=(1, n, 1), ku=0.99, dt=0.99 * ds / C0, ds=ds, main_lo=(0, npml, 0),
                   main_hi=(0, n - npml - 1, 0), precision=_prec(case))
    hi = n - npml - 1
    geo = dict(gold=GOLD, slab=None, layers=[(npml, hi, 1.0)], bd=-1, eps_hi=1.0)
    if tfsf:
        a = n - 100 - int(rng.integers(60, 120)) - n // 50
        b = a + n // 50
        geo["layers"] = [(npml, a - 1, 1.0), (a, b - 1, SUBSTRATE), (b, hi, 3.772 ** 2)]
        geo.update(bd=npml + 14, eps_hi=3.772 ** 2, spos=npml + 9)
        spec.tfsf = dict(boundary=geo["bd"], eps_lo=1.0, eps_hi=1.0)
    else:
        lo = n // 2 + int(rng.integers(-20, 20))
        geo["slab"] = (lo, lo + 49)
        geo["spos"] = 100
    for lo, up, ep in geo["layers"]:
        spec.add_dielectric(box((0, lo, 0), (0, up, 0)), ep)
    if geo["slab"]:
        spec.add_gold(box((0, geo["slab"][0], 0), (0, geo["slab"][1], 0)), GOLD)
    spec.pml = dict(mode=abi.PML_REFERENCE, npml=((0, 0), (npml, npml), (0, 0)), eps_lo=1.0, eps_hi=geo["eps_hi"],
                    sigma_max=_sigma(npml, ds), order=3.0)
    s = geo["spos"]
    spec.sources.append(dict(component=abi.EX_INC if tfsf else abi.EX, lo=(0, s, 0), hi=(0, s, 0), amp=1.0,
                             **_pulse(600e-9, 0.5e-15, 1.5)))
    if tfsf:
        om = _omegas(200e-9, 1000e-9, 100)
        spec.add_monitor((0, geo["bd"] - 5, 0), (0, geo["bd"] - 5, 0), (abi.EX_INC, abi.HZ_INC), om)
        spec.add_monitor((0, geo["bd"] + 5, 0), (0, geo["bd"] + 5, 0), (abi.EX, abi.HZ), om)
    else:
        om = _omegas(400e-9, 900e-9, 200)
        for y in (300, 3 * n // 4):
            spec.add_monitor((0, y, 0), (0, y, 0), (abi.EX, abi.HZ), om)
    return spec, geo


def _sphere(case, rng):
    """A 3D job: the benchmark's gold sphere, its source plane and the box of monitors."""
    n, npml, ds = (case["nx"], case["ny"], case["nz"]), case["npml"], 1e-9
    spec = JobSpec(layout=abi.LAYOUT_3D, n=n, ku=0.5, dt=0.5 * ds / C0, ds=ds, precision=_prec(case),
                   main_lo=(npml,) * 3, main_hi=tuple(x - npml - 1 for x in n))
    spec.add_dielectric(box((0, 0, 0), tuple(x - 1 for x in n)), 1.0)
    m = min(n)
    r = max(4.0, 40.0 * m / 512.0)
    c = [x / 2.0 + float(rng.uniform(-2.0, 2.0)) for x in n]
    spec.add_gold(spheres([(*c, r)]), GOLD)
    spec.pml = dict(mode=abi.PML_SPLIT, npml=((npml, npml),) * 3, eps_lo=1.0, sigma_max=_sigma(npml, ds), order=3.0)
    zs = npml + 4
    spec.sources.append(dict(component=abi.EX, lo=(0, 0, zs), hi=(n[0] - 1, n[1] - 1, zs), amp=1.0,
                             **_pulse(600e-9, 0.5e-15, 1.5)))
    h = int(70 * m / 512.0) + 4
    om = _omegas(500e-9, 800e-9, case["nfreq"])
    tang = ((abi.EY, abi.EZ, abi.HY, abi.HZ), (abi.EX, abi.EZ, abi.HX, abi.HZ), (abi.EX, abi.EY, abi.HX, abi.HY))
    mid = [x // 2 for x in n]
    for axis in range(3):
        for side in (-h, h):
            lo, hi = [x - h for x in mid], [x + h for x in mid]
            lo[axis] = hi[axis] = mid[axis] + side
            spec.add_monitor(tuple(lo), tuple(hi), tang[axis], om)
    return spec, dict(ball=(*c, r), gold=GOLD)


def _column(case):
    nxy, nz, npml, ds = case["nxy"], case["nz"], 10, 2e-9
    spec = JobSpec(layout=abi.LAYOUT_3D, n=(nxy, nxy, nz), ku=0.5, dt=0.5 * ds / C0, ds=ds, precision=_prec(case),
                   periodic=(1, 1, 0), main_lo=(0, 0, npml), main_hi=(nxy - 1, nxy - 1, nz - npml - 1))
    spec.add_dielectric(box((0, 0, 0), (nxy - 1, nxy - 1, nz - 1)), 1.0)
    zg = nz // 2
    spec.add_graphene(box((0, 0, zg), (nxy - 1, nxy - 1, zg)), GRAPHENE)
    spec.pml = dict(mode=abi.PML_SPLIT, npml=((0, 0), (0, 0), (npml, npml)), eps_lo=1.0, sigma_max=_sigma(npml, ds),
                    order=3.0)
    f0 = C0 / 1550e-9
    spec.sources.append(dict(component=abi.EX, lo=(0, 0, 20), hi=(nxy - 1, nxy - 1, 20), amp=1e8, t0=1.5e-15, st=1e-15,
                             w0=2.0 * math.pi * f0))
    zt = nz * 300 // 384
    om = 2.0 * math.pi * f0 * np.linspace(1.0, 3.0, case["nfreq"], endpoint=False)
    spec.add_monitor((0, 0, zt), (nxy - 1, nxy - 1, zt), (abi.EX, abi.EY, abi.HX, abi.HY), om, mean=True)
    return spec, dict(sheet=zg)


def _program(case, dim):
    spec, meta = (problems.reference_2d if dim == 2 else problems.reference_3d)(_prec(case))
    far = 2 ** 31 - 1
    for m in spec.monitors + spec.probes:  # a stretch in the middle of the run: every record is taken
        m.n_first, m.n_last = 1, far
    if dim == 2:
        spec.probes = []
    return spec, meta


def _jobs(case, seed):
    """Specs and geometry of a case's jobs, one but for a batch."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "line":
        return [_line(case, rng)]
    if kind == "plane":
        return [_plane(case, rng)]
    if kind == "sphere":
        return [_sphere(case, rng)]
    if kind == "column":
        return [_column(case)]
    if kind in ("program2", "program3"):
        return [_program(case, int(kind[-1]))]
    out = []
    for q in range(case["jobs2"]):
        c = dict(case, nx=case["n2"], ny=case["n2"] + (q % 3) * 32, npml=16, te=False, substrate=False,
                 cylinders=1 + int(rng.integers(1, 8)), host_loop=False)
        out.append(_plane(c, rng))
    for q in range(case["jobs3"]):
        out.append(_sphere(dict(case, nx=case["n3"], ny=case["n3"], nz=case["n3"], npml=12), rng))
    return out


def _start(case, spec, seed):
    """The starting values of the main E component, [nz, ny, nx]: a few wave packets inside the main range."""
    rng = np.random.default_rng(seed + 7919)
    lo = spec.main_lo
    hi = spec.main_hi
    amp = 1e8 if case["kind"] == "column" else 1.0
    out = None
    for _ in range(2):
        f = []
        for a in range(3):
            x = np.arange(spec.n[a], dtype=np.float64)
            length = hi[a] - lo[a] + 1
            if spec.n[a] == 1:
                f.append(np.ones(1))
                continue
            if spec.periodic[a]:
                g = 1.0 + 0.3 * np.cos(2.0 * math.pi * (x / spec.n[a] + rng.random()))
            else:
                t = (x - lo[a] + 0.5) / length
                g = np.where((t > 0) & (t < 1), np.sin(math.pi * np.clip(t, 0, 1)) ** 4, 0.0)
                g = g * np.cos(2.0 * math.pi * x / rng.uniform(24.0, 90.0) + rng.uniform(0, 6.28))
            f.append(g)
        w = amp * rng.uniform(0.4, 1.0) * f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
        out = w if out is None else out + w
    return out


def _main_comp(spec):
    return abi.EZ if spec.layout == abi.LAYOUT_2D_TM else abi.EX


def _frame(case):
    """Whether a pass ends with a frame of the field: the programs' and the small grids' do."""
    return case["kind"] in ("line", "program2") or (case["kind"] == "plane" and case["nx"] * case["ny"] <= 400000
                                                    and not case["host_loop"])


# ---- what a program holds, and a pass --------------------------------------------
def prepare(case, seed):
    jobs = _jobs(case, seed)
    bufs = []
    for spec, _ in jobs:
        mine = []
        for m in spec.monitors:
            count = int(np.prod(monitor_shape(m)))
            t = torch.empty(2, count, dtype=torch.float64, pin_memory=torch.cuda.is_available())
            t.zero_()
            mine.append((t[0].numpy(), t[1].numpy()))
        bufs.append(mine)
    state = dict(case=case, bufs=bufs)
    if case["kind"] == "serve":
        state["specs"] = [spec for spec, _ in jobs]
        state["server"] = Server(hbm_budget=16 << 30, max_active=16, chunk_steps=256)
        return state
    spec = jobs[0][0]
    job = Job(spec)
    job.set_field(_main_comp(spec), _start(case, spec, seed))
    job.sync()
    state["job"] = job
    return state


def run(state):
    case, out = state["case"], []
    if case["kind"] == "serve":
        server = state["server"]
        tickets = [server.submit(spec, case["steps"]) for spec in state["specs"]]
        for ticket, mine in zip(tickets, state["bufs"]):
            if server.wait(ticket) != 2:
                raise RuntimeError("a served job failed")
            job = server.job(ticket)
            for q, pair in enumerate(mine):
                out.append(job.get_monitor(q, out=pair))
            server.release(ticket)
        return out
    job = state["job"]
    if case.get("host_loop"):
        for n in range(job.n_done + 1, job.n_done + 1 + case["steps"]):
            job.step_procedures(n)
    else:
        job.run(case["steps"])
    for q, pair in enumerate(state["bufs"][0]):
        out.append(job.get_monitor(q, out=pair))
    if case.get("host_loop"):
        out.append(job.get_probe(0)[-case["steps"]:])
    if _frame(case):
        out.append(job.get_field(abi.HX if job.spec.layout == abi.LAYOUT_2D_TM else abi.HZ))
    return out


def _cells(spec):
    return float(spec.n[0]) * spec.n[1] * spec.n[2]


def work(case):
    """Each field read and written once a step (not the material ids), the
    dispersive state aside; the spectra and the frame once."""
    bytes_ = flops = 0.0
    for spec, _ in _jobs(case, 1):
        w = 8.0 if spec.precision == abi.F64 else 4.0
        fields = {abi.LAYOUT_1D: 2, abi.LAYOUT_2D_TE: 3, abi.LAYOUT_2D_TM: 3, abi.LAYOUT_3D: 6}[spec.layout]
        if case.get("tfsf"):
            fields = 4
        ops = {2: 6.0, 4: 12.0, 3: 14.0, 6: 36.0}[fields]
        bytes_ += _cells(spec) * 2.0 * fields * w * case["steps"]
        flops += _cells(spec) * ops * case["steps"]
        for m in spec.monitors:
            count = float(np.prod(monitor_shape(m)))
            bytes_ += 16.0 * count
            flops += 4.0 * count * case["steps"]
    return {"bytes": bytes_, "flops": flops}


# ---- the same in 64 bits, in plain torch --------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=_dev())


def _profile(length, lo, hi, ep, spec, npml=None):
    """f1, f2, g1, g2 along an axis: lo and hi graded cells at its two ends."""
    k = spec.dt * C0 / spec.ds
    sm, order = spec.pml["sigma_max"], spec.pml["order"]
    z0 = math.sqrt(MU0 / EP0)
    f1, f2, g1, g2 = np.ones(length), np.full(length, k / ep), np.ones(length), np.full(length, k)

    def e_cell(x, u, cells):
        s = ep * EP0 * sm * (u / cells) ** order
        f1[x] = math.exp(-s * spec.dt / (ep * EP0))
        f2[x] = (1.0 - f1[x]) / (z0 * s * spec.ds)

    def h_cell(x, u, cells):
        s = MU0 * sm * (u / cells) ** order
        g1[x] = math.exp(-s * spec.dt / MU0)
        g2[x] = z0 * (1.0 - g1[x]) / (s * spec.ds)

    for i in range(lo):
        e_cell(i, lo - 1 - i + 0.5, lo)
        if lo - 1 - i > 0:
            h_cell(i, lo - 1 - i, lo)
    for q in range(hi):
        if q > 0:
            e_cell(length - hi + q, q, hi)
        h_cell(length - hi + q, q + 0.5, hi)
    return [_t(x) for x in (f1, f2, g1, g2)]


class _Gold:
    """Drude and two critical points on the flagged cells of a few components."""

    def __init__(self, at, p, dt, comps):
        self.at = at
        z = torch.zeros(int(at.sum()), dtype=torch.float64, device=_dev())
        self.ha, self.hb = math.exp(-p["gamma_d"] * dt), p["omega_d"] ** 2 * dt / p["gamma_d"]
        self.gb = [complex(math.e) ** complex(-g * dt, w * dt) for g, w in zip(p["gamma"], p["omega"])]
        self.gc = [2j * dt * a * w * complex(math.cos(f), -math.sin(f)) for a, w, f in
                   zip(p["amp"], p["omega"], p["phi"])]
        self.ga = p["eps_inf"] - sum(self.gc)
        self.s = {c: [z.clone(), z.clone(), z.to(torch.complex128), z.to(torch.complex128)] for c in comps}

    def __call__(self, c, inc):
        q, s, g1, g2 = self.s[c]
        q = q + inc
        g1, g2 = self.gb[0] * g1, self.gb[1] * g2
        e = ((q + self.ha * s + g1 + g2) / self.ga).real
        self.s[c] = [q - self.hb * e, self.ha * s + self.hb * e, g1 + self.gc[0] * e, g2 + self.gc[1] * e]
        return e


class _Sheet:
    """The conducting graphene sheet with its instantaneous and delayed third order."""

    def __init__(self, p, dt, n):
        hbar, kt = 6.62607015e-34 / (2.0 * math.pi), 1.380649e-23 * p["temperature"]
        qe = 1.602176634e-19
        sig = 2.0 * qe * qe * kt * p["tau"] / (math.pi * hbar * hbar) * math.log(2.0 * math.cosh(p["fermi_ev"] * qe / (2 * kt)))
        self.ha, self.hb = math.exp(-dt / p["tau"]), sig / p["thickness"] * dt / EP0
        w, a = 2.0 * math.pi * p["raman_freq"], 0.5 / p["raman_tau"]
        b = math.sqrt(w * w - a * a)
        self.r0 = p["raman_frac"] * p["chi3"] * (w * w / b) * dt * math.exp(-a * dt) * math.sin(b * dt)
        sb = math.sin(0.5 * b * dt)
        c1 = 2.0 * (math.expm1(-a * dt) * math.cos(b * dt) - 2.0 * sb * sb)
        c2 = -math.expm1(-2.0 * a * dt)
        self.rv, self.rs = 1.0 - c2, c1 + c2
        self.kerr = (1.0 - p["raman_frac"]) * p["chi3"]
        z = torch.zeros(n, dtype=torch.float64, device=_dev())
        self.s = {c: [z.clone() for _ in range(4)] for c in (abi.EX, abi.EY)}

    def __call__(self, c, inc, old):
        q, s, sr, v = self.s[c]
        q = q + inc
        e = (q + self.ha * s + 2.0 * self.kerr * old ** 3) / (1.0 + sr + 3.0 * self.kerr * old * old)
        v = self.rv * v + self.rs * sr + self.r0 * e * e
        self.s[c] = [q - self.hb * e, self.ha * s + self.hb * e, sr + v, v]
        return e


def _shift(a, axis, step, wrap):
    """a at the cell `step` (+1 or -1) away along an axis (0 = x): wrapped, or zero outside."""
    d = a.dim() - 1 - axis
    r = torch.roll(a, -step, d)
    if not wrap:
        r.select(d, a.shape[d] - 1 if step > 0 else 0).zero_()
    return r


def _ids(spec, geo, case):
    """eps and the flag of dispersive cells, [nz, ny, nx]."""
    nx, ny, nz = spec.n
    eps = torch.ones(nz, ny, nx, dtype=torch.float64, device=_dev())
    gold = torch.zeros(nz, ny, nx, dtype=torch.bool, device=_dev())
    x = torch.arange(nx, device=_dev(), dtype=torch.float64) + 0.5
    y = torch.arange(ny, device=_dev(), dtype=torch.float64) + 0.5
    z = torch.arange(nz, device=_dev(), dtype=torch.float64) + 0.5
    if case["kind"] in ("program2", "program3"):
        for name, ep in (("air", 1.0), ("au", None), ("sio2", 1.46 ** 2), ("si", 3.88 ** 2)):
            m = geo.get(name)
            if m is None:  # the 3D program's regions: read them off the boxes of its materials
                reg = spec.materials[("air", "au", "sio2", "si").index(name)].region
                lo, hi = reg["lo"], reg["hi"]
            else:
                lo, hi = (m["x"][0] - 1, m["y"][0] - 1, 0), (m["x"][1] - 1, m["y"][1] - 1, nz - 1)
            part = (slice(lo[2], hi[2] + 1), slice(lo[1], hi[1] + 1), slice(lo[0], hi[0] + 1))
            gold[part] = ep is None
            eps[part] = ep or 1.0
        return eps, gold
    if geo.get("sub") is not None:
        npml = case["npml"]
        eps[:, geo["sub"]:ny - npml, npml:nx - npml] = SUBSTRATE
    for cx, cy, _, r in geo.get("cyl", ()):
        gold |= ((x[None, None, :] - cx) ** 2 + (y[None, :, None] - cy) ** 2 <= r * r)
    if geo.get("ball"):
        cx, cy, cz, r = geo["ball"]
        gold |= ((x[None, None, :] - cx) ** 2 + (y[None, :, None] - cy) ** 2 + (z[:, None, None] - cz) ** 2 <= r * r)
    return eps, gold


# E component -> ((axis of the derivative, H component, sign), ...) of its curl, backward differences;
# H component -> the same of its curl of E, forward differences (3D; 2D takes the terms it has)
_CURL_E = {abi.EX: ((1, abi.HZ, 1), (2, abi.HY, -1)), abi.EY: ((2, abi.HX, 1), (0, abi.HZ, -1)),
           abi.EZ: ((0, abi.HY, 1), (1, abi.HX, -1))}
_CURL_H = {abi.HX: ((1, abi.EZ, -1), (2, abi.EY, 1)), abi.HY: ((2, abi.EX, -1), (0, abi.EZ, 1)),
           abi.HZ: ((0, abi.EY, -1), (1, abi.EX, 1))}


def _gauss(s, t):
    a = (t - s["t0"]) / s["st"]
    return s["amp"] * math.exp(-0.5 * a * a) * math.sin(s["w0"] * t)


def _spectra(samples, spec, steps):
    """re, im of each monitor from its samples, [step][component][cell]."""
    t = _t(np.arange(steps) * spec.dt)
    out = []
    for m, rows in zip(spec.monitors, samples):
        v = torch.stack(rows)  # [step, comp, cell]
        ph = _t(m.omega)[:, None] * t[None, :]
        re = torch.einsum("fs,scx->cfx", torch.cos(ph), v) * spec.dt
        im = torch.einsum("fs,scx->cfx", torch.sin(ph), v) * spec.dt
        out.append((re.cpu().numpy(), im.cpu().numpy()))
    return out


class _Slabs:
    """The reference's PML of y-slabs: split fields of their own over the slab
    rows, joined to the grid at one row (2D: BERpmly_HzExEy, 3D: BERpmly)."""

    def __init__(self, spec, dim):
        nx, ny, nz = spec.n
        p = spec.pml
        self.dim, self.rows, self.ny = dim, p["npml"][1][0], ny
        names = ("exy", "exz", "eyz", "eyx", "ezx", "ezy", "hxy", "hxz", "hyz", "hyx", "hzx", "hzy")
        self.f = [{k: torch.zeros(nz, self.rows, nx, dtype=torch.float64, device=_dev()) for k in names} for _ in (0, 1)]
        self.prof = []
        for side in (0, 1):
            ep = (p["eps_lo"], p["eps_hi"])[side]
            x = _profile(nx, p["npml"][0][0], p["npml"][0][1], ep, spec)
            y = _profile(self.rows, self.rows if side == 0 else 0, self.rows if side else 0, ep, spec)
            z = _profile(nz, p["npml"][2][0], p["npml"][2][1], ep, spec)
            self.prof.append([[q[None, None, :] for q in x], [q[None, :, None] for q in y], [q[:, None, None] for q in z]])

    def e(self, F):
        for side in (0, 1):
            f, (px, py, pz) = self.f[side], self.prof[side]
            hx, hy, hz = f["hxy"] + f["hxz"], f["hyz"] + f["hyx"], f["hzx"] + f["hzy"]
            hzd, hxd = _shift(hz, 1, -1, False), _shift(hx, 1, -1, False)
            edge = self.rows - 1 if side == 0 else self.ny - self.rows
            if side == 1:  # the row below the slab is the grid's
                hzd[:, 0] = F[abi.HZ][:, edge - 1]
                if self.dim == 3:
                    hxd[:, 0] = F[abi.HX][:, edge - 1]
            hzc = hz
            if self.dim == 2 and side == 0:  # the 2D coupling row takes the grid's Hz
                hzc = hz.clone()
                hzc[:, -1] = F[abi.HZ][:, edge]
            f["exy"] = py[0] * f["exy"] + py[1] * (hzc - hzd)
            f["eyx"] = px[0] * f["eyx"] + px[1] * (_shift(hz, 0, -1, False) - hz)
            if self.dim == 3:
                f["exz"] = pz[0] * f["exz"] + pz[1] * (_shift(hy, 2, -1, False) - hy)
                f["eyz"] = pz[0] * f["eyz"] + pz[1] * (hx - _shift(hx, 2, -1, False))
                f["ezx"] = px[0] * f["ezx"] + px[1] * (hy - _shift(hy, 0, -1, False))
                f["ezy"] = py[0] * f["ezy"] + py[1] * (hxd - hx)
                F[abi.EX][:, edge] = f["exy"][:, -1 if side == 0 else 0]
                F[abi.EZ][:, edge] = f["ezy"][:, -1 if side == 0 else 0]
            else:
                at = slice(0, self.rows) if side == 0 else slice(edge, self.ny)
                F[abi.EX][:, at] = f["exy"]

    def h(self, F):
        for side in (0, 1):
            f, (px, py, pz) = self.f[side], self.prof[side]
            ex, ey, ez = f["exy"] + f["exz"], f["eyz"] + f["eyx"], f["ezx"] + f["ezy"]
            exu, ezu = _shift(ex, 1, 1, False), _shift(ez, 1, 1, False)
            if side == 0 and self.dim == 3:  # the row above the slab is the grid's
                exu[:, -1], ezu[:, -1] = F[abi.EX][:, self.rows], F[abi.EZ][:, self.rows]
            f["hzy"] = py[2] * f["hzy"] + py[3] * (exu - ex)
            f["hzx"] = px[2] * f["hzx"] + px[3] * (ey - _shift(ey, 0, 1, False))
            if self.dim == 3:
                f["hxy"] = py[2] * f["hxy"] + py[3] * (ez - ezu)
                f["hxz"] = pz[2] * f["hxz"] + pz[3] * (_shift(ey, 2, 1, False) - ey)
                f["hyz"] = pz[2] * f["hyz"] + pz[3] * (ex - _shift(ex, 2, 1, False))
                f["hyx"] = px[2] * f["hyx"] + px[3] * (_shift(ez, 0, 1, False) - ez)
                row, r = (self.rows - 1, -1) if side == 0 else (self.ny - self.rows, 0)
                F[abi.HX][:, row] = f["hxy"][:, r]
                F[abi.HZ][:, row] = f["hzy"][:, r]
            elif side == 0:
                F[abi.HZ][:, :self.rows - 1] = (f["hzy"] + f["hzx"])[:, :-1]
            else:
                F[abi.HZ][:, self.ny - self.rows:] = f["hzy"] + f["hzx"]


def _exact_grid(case, spec, geo, start):
    """2D and 3D: fields [nz, ny, nx] in 64 bits; returns the spectra, the fields and the probe's records."""
    nx, ny, nz = spec.n
    dim = 3 if spec.layout == abi.LAYOUT_3D else 2
    comps = {abi.LAYOUT_2D_TE: (abi.EX, abi.EY, abi.HZ), abi.LAYOUT_2D_TM: (abi.EZ, abi.HX, abi.HY),
             abi.LAYOUT_3D: range(6)}[spec.layout]
    F = {c: torch.zeros(nz, ny, nx, dtype=torch.float64, device=_dev()) for c in comps}
    if start is not None:
        F[_main_comp(spec)] = _t(start)
    eps, gold = _ids(spec, geo, case)
    idx = [torch.arange(n, device=_dev()).reshape([-1 if 2 - d == a else 1 for d in range(3)])
           for a, n in enumerate(spec.n)]
    inside = torch.ones(nz, ny, nx, dtype=torch.bool, device=_dev())
    for a in range(dim):
        inside &= (idx[a] >= spec.main_lo[a]) & (idx[a] <= spec.main_hi[a])
    split = spec.pml["mode"] == abi.PML_SPLIT
    slabs = None if split else _Slabs(spec, dim)
    if split:
        prof = []
        for a in range(dim):
            lo, hi = (0, 0) if spec.periodic[a] else spec.pml["npml"][a]
            prof.append([q.reshape([-1 if 2 - d == a else 1 for d in range(3)]) for q in
                         _profile(spec.n[a], lo, hi, 1.0, spec)])
        parts = {}
        gold &= inside
    es = [c for c in comps if c <= abi.EZ]
    hs = [c for c in comps if c > abi.EZ]
    ca = torch.where(inside, spec.ku / eps, torch.zeros_like(eps))
    cs = torch.where(inside, 1.0 / eps, torch.zeros_like(eps))
    metal = _Gold(gold, GOLD_PROGRAM if "program" in case["kind"] else geo["gold"], spec.dt, es) if bool(gold.any()) else None
    sheet = _Sheet(GRAPHENE, spec.dt, ny * nx) if case["kind"] == "column" else None
    src = spec.sources[0]
    at = tuple(slice(max(src["lo"][a], spec.main_lo[a]), min(src["hi"][a], spec.main_hi[a]) + 1) for a in (2, 1, 0))
    samples, record = [[] for _ in spec.monitors], []

    def half(c, curl, step, pick, coef):
        """The new values of component c: the split update outside the main range, else the plain one."""
        terms = [(a, sg * step * (_shift(F[o], a, step, bool(spec.periodic[a])) - F[o])) for a, o, sg in curl[c] if o in F and a < dim]
        total = sum(t for _, t in terms)
        new = F[c] + coef * total
        if split and any(a for a in range(dim)):
            both = None
            for a, t in terms:
                old = parts.get((c, a), 0.0)
                parts[(c, a)] = prof[a][pick] * old + prof[a][pick + 1] * t
                both = parts[(c, a)] if both is None else both + parts[(c, a)]
            new = torch.where(inside, new, both)
        return new, total

    for n in range(1, case["steps"] + 1):
        g = _gauss(src, (n - 1) * spec.dt)
        new = {}
        for c in es:
            v, total = half(c, _CURL_E, -1, 0, ca)
            inc = None
            if metal or sheet:
                inc = spec.ku * total
            if c == src["component"]:
                v[at] += cs[at] * g
                if inc is not None:
                    inc[at] += g
            if metal:
                v[gold] = metal(c, inc[gold])
            if sheet and c != abi.EZ:
                k = geo["sheet"]
                v[k] = sheet(c, inc[k].reshape(-1), F[c][k].reshape(-1)).reshape(ny, nx)
            new[c] = v
        F.update(new)
        if slabs:
            slabs.e(F)
        new = {c: half(c, _CURL_H, 1, 2, torch.where(inside, spec.ku, 0.0))[0] for c in hs}
        F.update(new)
        if slabs:
            slabs.h(F)
        for rows, m in zip(samples, spec.monitors):
            part = tuple(slice(m.lo[a], m.hi[a] + 1) for a in (2, 1, 0))
            v = torch.stack([F[c][part].reshape(-1) for c in sorted(m.comps)])
            rows.append(v.mean(1, keepdim=True) if m.mean else v)
        if case.get("host_loop"):
            i, j, k = spec.probes[0].cell
            record.append([float(F[c][k, j, i]) for c in sorted(spec.probes[0].comps)])
    return _spectra(samples, spec, case["steps"]), F, record


def _exact_line(case, spec, geo, start):
    n, bd = case["cells"], geo["bd"]
    lo, hi = spec.main_lo[1], spec.main_hi[1]
    rows = spec.pml["npml"][1][0]
    eps = np.ones(n)
    for a, b, ep in geo["layers"]:
        eps[a:b + 1] = ep
    eps = _t(eps)
    zero = lambda k: torch.zeros(k, dtype=torch.float64, device=_dev())  # noqa: E731
    lines = [dict(e=_t(start).reshape(-1), h=zero(n), ep=(1.0, geo["eps_hi"]))]
    if case["tfsf"]:
        lines.append(dict(e=zero(n), h=zero(n), ep=(1.0, 1.0)))
    for ln in lines:
        ln["slab"] = []
        for side in (0, 1):
            q = _profile(rows, rows if side == 0 else 0, rows if side else 0, ln["ep"][side], spec)
            ln["slab"].append(dict(e=zero(rows + 2), h=zero(rows + 2), p=q))
    gold = torch.zeros(n, dtype=torch.bool, device=_dev())
    if geo["slab"]:
        gold[geo["slab"][0]:geo["slab"][1] + 1] = True
    metal = _Gold(gold, geo["gold"], spec.dt, (abi.EX,)) if geo["slab"] else None
    main = slice(lo, hi + 1)
    src, samples = spec.sources[0], [[] for _ in spec.monitors]
    ku, s = spec.ku, geo["spos"]
    for step in range(case["steps"]):
        g = _gauss(src, step * spec.dt) / (src["amp"] if case["tfsf"] else 1.0)
        for q, ln in enumerate(lines):
            e, h = ln["e"], ln["h"]
            curl = h[main] - h[lo - 1:hi]
            extra = zero(n)
            if q == len(lines) - 1:
                extra[s] += g
            if q == 0 and bd >= 0:
                extra[bd] -= ku * lines[1]["h"][bd - 1]
            if q == 0:
                new = e[main] + (ku * curl + extra[main]) / eps[main]
                if metal:
                    inc = zero(n)
                    inc[main] = ku * curl + extra[main]
                    new[gold[main]] = metal(abi.EX, inc[gold])
            else:
                new = e[main] + ku * curl + extra[main]
            ln["new"] = new
        for ln in lines:
            ln["e"][main] = ln.pop("new")
            for side, sl in enumerate(ln["slab"]):
                f1, f2, _, _ = sl["p"]
                sl["e"][1:rows + 1] = f1 * sl["e"][1:rows + 1] + f2 * (sl["h"][1:rows + 1] - sl["h"][:rows])
                if side == 0:
                    sl["e"][rows + 1] = ln["e"][rows]
                    ln["e"][rows - 1] = sl["e"][rows]
                else:
                    sl["e"][0] = ln["e"][n - rows - 1]
                    ln["e"][n - rows] = sl["e"][1]
        for ln in lines:
            e, h = ln["e"], ln["h"]
            h[main] = h[main] + ku * (e[lo + 1:hi + 2] - e[main])
            for side, sl in enumerate(ln["slab"]):
                _, _, g1, g2 = sl["p"]
                sl["h"][1:rows + 1] = g1 * sl["h"][1:rows + 1] + g2 * (sl["e"][2:] - sl["e"][1:rows + 1])
                if side == 0:
                    sl["h"][rows + 1] = h[rows]
                    h[rows - 1] = sl["h"][rows]
                else:
                    sl["h"][0] = h[n - rows - 1]
                    h[n - rows] = sl["h"][1]
        if bd > 0:
            lines[0]["h"][bd - 1] -= ku * lines[1]["e"][bd]
        names = {abi.EX: (0, "e"), abi.HZ: (0, "h"), abi.EX_INC: (1, "e"), abi.HZ_INC: (1, "h")}
        for rec, m in zip(samples, spec.monitors):
            j = m.lo[1]
            rec.append(torch.stack([lines[names[c][0]][names[c][1]][j:j + 1] for c in sorted(m.comps)]))
    return _spectra(samples, spec, case["steps"]), lines[0]["h"]


def exact(case, seed):
    out = []
    for spec, geo in _jobs(case, seed):
        start = None if case["kind"] == "serve" else _start(case, spec, seed)
        if case["kind"] == "line":
            spectra, h = _exact_line(case, spec, geo, start)
            out += spectra + [h.cpu().numpy().reshape(1, case["cells"], 1)]
            continue
        spectra, fields, record = _exact_grid(case, spec, geo, start)
        out += spectra
        if case.get("host_loop"):
            out.append(np.array(record))
        if _frame(case):
            out.append(fields[abi.HX if spec.layout == abi.LAYOUT_2D_TM else abi.HZ].cpu().numpy())
    return out
