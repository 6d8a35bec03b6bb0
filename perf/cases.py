"""The work users have this framework do, as cases that can be timed one by one.

Kinds of case:
  step      a running simulation (one job, or a batch of jobs in one engine) advanced by a block
            of steps, then its potential and charge read into device tensors: what a simulation
            loop does between two looks at its fields
  request   one served request from nothing: job creation, particle load from device arrays,
            stream-ordered steps, diagnostics, results, job destroyed
  poisson   the stateless multigrid Poisson solve on caller-owned FP64 arrays, from phi = 0
  embedded  the embedded-boundary multigrid solve (electrodes and solid blocks in the domain)

Sizes and settings are those of the package's workloads (configs.py, batch.py, serve.py), of the
reference's solver call (5 levels, omega 1.25, 3/3/20 sweeps, 1e-5) and of the benchmark's
embedded-boundary problem.
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from pic_cuda_b200 import _lib as L
from pic_cuda_b200 import batch
from pic_cuda_b200 import configs as cf
from pic_cuda_b200.engine import Engine, solve_embedded_f64, solve_multigrid_f64

EPS0 = 8.8541878128e-12
DEV = "cuda"


def listed():
    return [
        # The smallest simulation (129^2, 1e5 + 1e5, collisionless): launches and latency count.
        dict(name="step_plain_129", kind="step", n=129, particles=100_000, mcc=False, deposit="f32", tol=1e-6,
             steps=20, jobs=1),
        # The collisional workload, 1025^2 with 1e7 + 1e7 in argon, FP32 deposit: an ordinary run.
        dict(name="step_mcc_1025", kind="step", n=1025, particles=10_000_000, mcc=True, deposit="f32", tol=1e-9,
             steps=10, jobs=1),
        # A collisionless run of middle size with an odd particle number, FP32 deposit.
        dict(name="step_plain_2049", kind="step", n=2049, particles=24_999_999, mcc=False, deposit="f32", tol=1e-9,
             steps=10, jobs=1),
        # The largest run, 4097^2 with 1e8 + 1e8 in argon, bit-reproducible int64 deposit.
        dict(name="step_mcc_4097", kind="step", n=4097, particles=100_000_000, mcc=True, deposit="i64", tol=1e-9,
             steps=10, jobs=1),
        # A batch of uneven jobs (sides 65 .. 513) stepped together.
        dict(name="step_batch_32", kind="step", n=0, particles=0, mcc=True, deposit="i64", tol=1e-6, steps=10,
             jobs=32),
        # A small served request with its particles read back by their ids.
        dict(name="request_257", kind="request", n=257, ppc=20, steps=20, export=True),
        # A large request of few steps: creation, load and the first sort weigh as much as the steps.
        dict(name="request_1025", kind="request", n=1025, ppc=10, steps=4, export=False),
        # The reference's solver call on its demo grid: one small solve, latency.
        dict(name="poisson_129", kind="poisson", n=129, levels=5, nu=3, nu_coarse=20, omega=1.25, tol=1e-5),
        # The Poisson solve of the two collisional workloads on its own.
        dict(name="poisson_1025", kind="poisson", n=1025, levels=0, nu=2, nu_coarse=2, omega=1.15, tol=1e-9),
        dict(name="poisson_4097", kind="poisson", n=4097, levels=0, nu=2, nu_coarse=2, omega=1.15, tol=1e-9),
        # An electrode geometry on a rectangular grid solved to a tolerance.
        dict(name="embedded_385x257", kind="embedded", nx=385, ny=257, levels=6, nu=2, tol=1e-8, cycles=100),
        # Five V-cycles on the large grid (a caller that cycles the solver itself).
        dict(name="embedded_4097", kind="embedded", nx=4097, ny=4097, levels=10, nu=2, tol=0.0, cycles=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "request", "poisson", "embedded"])
    if kind == "step":
        n = rng.choice([129, 257, 513, 1025, 2049, 4097])
        mcc = rng.random() < 0.6
        # int64 deposits over the whole range; FP32 with collisions up to the 1025^2 workload
        deposit = "f32" if (not mcc or (n <= 1025 and rng.random() < 0.7)) else "i64"
        top = min(100_000_000, 100 * n * n, 10_000_000 if mcc and deposit == "f32" else 50_000_000)
        return dict(kind=kind, n=n, particles=_log_int(rng, max(20_000, 2 * n * n), top), mcc=mcc, deposit=deposit,
                    tol=rng.choice([1e-6, 1e-9]), steps=rng.randint(5, 15), jobs=1)
    if kind == "request":
        n = rng.choice([129, 257, 513, 1025])
        return dict(kind=kind, n=n, ppc=_log_int(rng, 4, min(200, 20_000_000 // (n * n))), steps=rng.randint(2, 30),
                    export=n <= 257)
    if kind == "poisson":
        n = rng.choice([65, 129, 257, 513, 1025, 2049, 4097])
        if rng.random() < 0.3:
            return dict(kind=kind, n=n, levels=5, nu=3, nu_coarse=20, omega=1.25, tol=rng.choice([1e-5, 1e-6]))
        return dict(kind=kind, n=n, levels=0, nu=rng.choice([1, 2, 2, 3]), nu_coarse=rng.choice([2, 20]),
                    omega=rng.choice([1.0, 1.15]), tol=rng.choice([1e-7, 1e-8, 1e-9]))
    nx = _log_int(rng, 100, 4097)
    ny = max(65, min(4097, _log_int(rng, nx / 2, 2 * nx)))
    levels = max(2, int(math.log2(min(nx, ny))) - 2)
    return dict(kind=kind, nx=nx, ny=ny, levels=levels, nu=rng.choice([1, 2, 2, 3]), tol=0.0,
                cycles=rng.randint(2, 8))


# ------------------------------------------------------------------------------------ step
WARM = 2   # steps a simulation has run before the measured ones (its first sort among them)


def _domain(n):
    return 0.01 if n <= 129 else 0.05 * (n - 1) / 1024


def _job_cfg(case):
    dep = L.DEPOSIT_I64 if case["deposit"] == "i64" else L.DEPOSIT_F32
    kw = dict(tol=case["tol"], deposit=dep, warm_start=1, omega=1.0 if case["tol"] > 1e-7 else cf.MG_OMEGA_1E9)
    if case["mcc"]:
        kw["mcc"] = cf.argon_mcc(3.2e21)
    return cf.plasma(case["n"], _domain(case["n"]), case["particles"], **kw)


def _specs(case, seed):
    dep = L.DEPOSIT_I64 if case["deposit"] == "i64" else L.DEPOSIT_F32
    return batch.batched_specs(case["jobs"], seed=4, ppc_scale=0.05, deposit=dep), seed % 1_000_003


def _electrons_ions(case, seed):
    n, box = case["particles"], _domain(case["n"])
    return (cf.maxwellian_state(n, box, 2.0, cf.ME, seed, DEV),
            cf.maxwellian_state(n, box, 0.03, cf.M_AR, seed + 1, DEV))


def _grid(job, which):
    """A grid of a job in a device tensor (pic_job_get_grid)."""
    out = torch.empty((job.ny, job.nx), dtype=torch.float64, device=DEV)
    L.check(L.lib().pic_job_get_grid(job.engine.h, job.id, which, C.c_void_p(out.data_ptr()), L.MEM_DEVICE),
            "pic_job_get_grid")
    return out


def _prepare_step(case, seed):
    eng = Engine(0)
    jobs = []
    if case["jobs"] == 1:
        job = eng.add_job(_job_cfg(case))
        for s, a in enumerate(_electrons_ions(case, seed)):
            job.load_species(s, *a)
            del a
        jobs.append(job)
    else:
        specs, shift = _specs(case, seed)
        for s in specs:
            s.seed += shift
            s.tol = case["tol"]
            job = eng.add_job(batch.job_config(s))
            batch.load_job(job, s, device=DEV)
            jobs.append(job)
    eng.step_graph(WARM)
    eng.sync()
    return dict(case=case, engine=eng, jobs=jobs)


def _run_step(st):
    st["engine"].step_graph(st["case"]["steps"])
    if len(st["jobs"]) > 1:
        return [_grid(j, L.GRID_PHI) for j in st["jobs"]]
    job = st["jobs"][0]
    return {"phi": _grid(job, L.GRID_PHI), "rho": _grid(job, L.GRID_RHO)}


# --------------------------------------------------------------------------------- request
def _prepare_request(case, seed):
    spec = batch.JobSpec(n=case["n"], ppc=case["ppc"], Te=3.0, density=3.2e21, steps=case["steps"], seed=seed)
    n = spec.n_per_species
    eng = Engine(0)
    eng.reserve(2 * batch.bytes_needed(batch.job_config(spec)))   # a server maps its budget at start-up
    parts = [cf.maxwellian_state(n, spec.L, spec.Te, cf.ME, seed, DEV),
             cf.maxwellian_state(n, spec.L, spec.Ti, cf.M_AR, seed + 1, DEV)]
    return dict(case=case, engine=eng, spec=spec, parts=parts)


def _track_table(raw, rows):
    """Exported particles of every species by their ids: one column per id with its position in
    cells and its velocity (zeros where the particle is gone), as a track file wants them."""
    out = torch.zeros((5, rows), dtype=torch.float32, device=DEV)
    for p in raw:
        cell = p["cell"]
        out[:, p["pid"].long()] = torch.stack([(cell & 0xFFFF) + p["fx"], (cell >> 16) + p["fy"], p["vx"], p["vy"],
                                               p["vz"]])
    return out


def _run_request(st):
    eng, case = st["engine"], st["case"]
    job = eng.add_job(batch.job_config(st["spec"]))
    for s, a in enumerate(st["parts"]):
        job.load_species(s, *a)
    eng.step(case["steps"])
    d = job.diagnostics()
    out = {"phi": _grid(job, L.GRID_PHI), "count": d["count"]}
    if case["export"]:
        out["tracks"] = _track_table([job.export_raw(0), job.export_raw(1)], 3 * st["spec"].n_per_species)
    else:
        out["rho"] = _grid(job, L.GRID_RHO)
    job.destroy()
    return out


# ------------------------------------------------------------------------ Poisson, embedded
def _prepare_poisson(case, seed):
    n = case["n"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    # charge noise of a few dozen particles per cell on a smooth cloud
    t = torch.linspace(0, 1, n, dtype=torch.float64, device=DEV)
    cloud = torch.exp(-8.0 * ((t[:, None] - 0.45) ** 2 + (t[None, :] - 0.55) ** 2))
    rho = cloud + 0.2 * torch.randn((n, n), generator=g, dtype=torch.float64, device=DEV)
    return dict(case=case, rho=rho, h=1.0 / (n - 1))


def _run_poisson(st):
    c = st["case"]
    phi = torch.zeros_like(st["rho"])
    cycles, _, _ = solve_multigrid_f64(phi, st["rho"], c["n"], c["n"], c["levels"], st["h"], c["omega"], c["nu"],
                                       c["nu"], c["nu_coarse"], c["tol"])
    return {"phi": phi, "cycles": cycles}


EMB_OPTIONS = L.EMB_COARSEN_ANY | L.EMB_PROLONG_BILINEAR


def _prepare_embedded(case, seed):
    nx, ny = case["nx"], case["ny"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    mask = torch.zeros((ny, nx), dtype=torch.uint8, device=DEV)
    mask[ny // 4: ny // 2, nx // 4: nx // 2 + 1] = L.NODE_DIRICHLET
    mask[3 * ny // 5: 3 * ny // 4, 3 * nx // 5: 4 * nx // 5] = L.NODE_SOLID
    rhs = torch.randn((ny, nx), generator=g, dtype=torch.float64, device=DEV)
    bc = torch.where(mask == L.NODE_DIRICHLET, 2.5, 0.0).double().contiguous()
    return dict(case=case, rhs=rhs, mask=mask, bc=bc, h=1.0 / (nx - 1))


def _run_embedded(st):
    c = st["case"]
    phi = torch.zeros_like(st["rhs"])
    cycles, _, _ = solve_embedded_f64(phi, st["rhs"], st["mask"], st["bc"], c["levels"], st["h"], c["nu"], c["nu"],
                                      EMB_OPTIONS, tol=c["tol"], max_cycles=c["cycles"])
    return {"phi": phi, "cycles": cycles}


_PREPARE = {"step": _prepare_step, "request": _prepare_request, "poisson": _prepare_poisson,
            "embedded": _prepare_embedded}
_RUN = {"step": _run_step, "request": _run_request, "poisson": _run_poisson, "embedded": _run_embedded}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------ work
# Bytes one V-cycle of the FP32 correction cannot do without: per level the right-hand side read
# and the correction written (down), both and the coarser correction read and the result written
# (up); on the finest level the FP64 potential read and written, the charge read and the new
# defect written.  A step adds the initial defect and the field.
def _vcycle_bytes(n):
    b, a = 25.0 * n * n, n
    while a > 3:
        b += 24.0 * a * a
        a = (a + 1) // 2
    return b


def _cycles(tol, warm):
    return max(1, math.ceil(-math.log10(tol) / 1.6) - (2 if warm else 0))


def _step_bytes(n, particles, mcc, rho_bytes, tol):
    return 2.0 * particles * (44 if mcc else 40) + n * n * (32.0 + 2 * rho_bytes) + _cycles(tol, True) * _vcycle_bytes(n)


def work(case):
    k = case["kind"]
    if k == "step":
        rb = 8 if case["deposit"] == "i64" else 4
        if case["jobs"] > 1:
            specs, _ = _specs(case, 0)
            b = sum(_step_bytes(s.n, s.n_per_species, True, rb, case["tol"]) for s in specs)
            p = sum(2.0 * s.n_per_species for s in specs)
            nodes = sum(s.n * s.n for s in specs)
        else:
            b = _step_bytes(case["n"], case["particles"], case["mcc"], rb, case["tol"])
            p, nodes = 2.0 * case["particles"], case["n"] ** 2
        f = p * (180.0 if case["mcc"] else 80.0) + 60.0 * nodes * _cycles(case["tol"], True)
        return {"bytes": b * case["steps"] + 16.0 * nodes, "flops": f * case["steps"]}
    if k == "request":
        p = case["ppc"] * (case["n"] - 1) ** 2
        b = _step_bytes(case["n"], p, True, 4, 1e-6) * case["steps"]
        b += 2.0 * p * (40 + 28 + 56) + (2.0 * p * 56 if case["export"] else 0.0)   # load, first sort, read-back
        return {"bytes": b, "flops": (2.0 * p * 180 + 60.0 * case["n"] ** 2 * 4) * case["steps"]}
    if k == "poisson":
        n, c = case["n"], _cycles(case["tol"], False)
        return {"bytes": c * _vcycle_bytes(n) + 40.0 * n * n, "flops": c * n * n * (8.0 + 2 * 12 * case["nu"] + 20)}
    nodes = float(case["nx"] * case["ny"])
    c = case["cycles"] if case["tol"] == 0.0 else 20
    return {"bytes": c * nodes * 4 / 3 * (50 + 25 / 4.0), "flops": c * nodes * 4 / 3 * (24.0 * case["nu"] + 20)}


# ----------------------------------------------------------------------------------- exact
def _sine(a):
    """Discrete sine transform (type I) along the last axis."""
    z = torch.zeros_like(a[..., :1])
    return -0.5 * torch.fft.rfft(torch.cat([z, a, z, -a.flip(-1)], -1)).imag[..., 1:a.shape[-1] + 1]


def _poisson_exact(rhs, h):
    """The discrete solution of lap(phi) = rhs, phi = 0 on the boundary."""
    n = rhs.shape[0]
    k = torch.arange(1, n - 1, dtype=torch.float64, device=rhs.device)
    lam = -4.0 / (h * h) * torch.sin(math.pi * k / (2 * (n - 1))) ** 2
    a = _sine(_sine(rhs[1:-1, 1:-1]).T).T
    a = a / (lam[:, None] + lam[None, :])
    phi = torch.zeros_like(rhs)
    phi[1:-1, 1:-1] = _sine(_sine(a).T).T * (2.0 / (n - 1)) ** 2
    return phi


def _deposit(n, dx, x, y, q, rho):
    xi, yi = x / dx, y / dx
    i, j = xi.floor().clamp(0, n - 2), yi.floor().clamp(0, n - 2)
    fx, fy = xi - i, yi - j
    a = (j * n + i).long()
    flat = rho.view(-1)
    for off, w in ((0, (1 - fx) * (1 - fy)), (1, fx * (1 - fy)), (n, (1 - fx) * fy), (n + 1, fx * fy)):
        flat.index_add_(0, a + off, q * w)


def _gather(n, dx, x, y, field):
    xi, yi = x / dx, y / dx
    i, j = xi.floor().clamp(0, n - 2), yi.floor().clamp(0, n - 2)
    fx, fy = xi - i, yi - j
    a = (j * n + i).long()
    f = field.reshape(-1)
    return ((1 - fx) * (1 - fy) * f[a] + fx * (1 - fy) * f[a + 1] + (1 - fx) * fy * f[a + n] + fx * fy * f[a + n + 1])


def _step_exact(case, seed):
    """Collisionless steps in FP64: drift, absorption at the walls, deposit, field, kick."""
    n, box, dt = case["n"], _domain(case["n"]), 1e-11
    dx = box / (n - 1)
    w = 1e15 * box * box / case["particles"]
    sp = [dict(q=q, m=m, p=[a[k] for k in range(4)])
          for (q, m), a in zip(((-cf.QE, cf.ME), (cf.QE, cf.M_AR)), _electrons_ions(case, seed))]
    phi = rho = None
    for _ in range(WARM + case["steps"]):
        rho = torch.zeros((n, n), dtype=torch.float64, device=DEV)
        if phi is not None:
            ey, ex = (-g for g in torch.gradient(phi, spacing=dx))
        for s in sp:
            x, y, vx, vy = s["p"]
            if phi is not None:
                vx = vx + s["q"] / s["m"] * dt * _gather(n, dx, x, y, ex)
                vy = vy + s["q"] / s["m"] * dt * _gather(n, dx, x, y, ey)
            x, y = x + vx * dt, y + vy * dt
            live = (x >= 0) & (x < box) & (y >= 0) & (y < box)
            s["p"] = [a[live] for a in (x, y, vx, vy)]
            _deposit(n, dx, s["p"][0], s["p"][1], s["q"] * w, rho)
        phi = _poisson_exact(-rho / (EPS0 * dx * dx), dx)
    return {"phi": phi, "rho": rho}


def _embedded_exact(case, seed):
    """Conjugate gradients on the FLUID nodes to round-off."""
    st = _prepare_embedded(case, seed)
    fluid = st["mask"] == L.NODE_FLUID
    fluid[0, :] = fluid[-1, :] = False
    fluid[:, 0] = fluid[:, -1] = False
    inside = torch.zeros_like(fluid)
    inside[1:-1, 1:-1] = True
    fixed = torch.where((st["mask"] == L.NODE_DIRICHLET) & inside, st["bc"], torch.zeros_like(st["bc"]))

    def minus_lap(a):
        r = torch.zeros_like(a)
        r[1:-1, 1:-1] = 4 * a[1:-1, 1:-1] - a[:-2, 1:-1] - a[2:, 1:-1] - a[1:-1, :-2] - a[1:-1, 2:]
        return torch.where(fluid, r, torch.zeros_like(r))

    b = torch.where(fluid, -st["h"] ** 2 * st["rhs"], torch.zeros_like(fixed)) - minus_lap(fixed)
    u = torch.zeros_like(b)
    r = b.clone()
    p = r.clone()
    rr = (r * r).sum()
    stop = rr.item() * 1e-28
    for it in range(6000):
        ap = minus_lap(p)
        alpha = rr / (p * ap).sum()
        u += alpha * p
        r -= alpha * ap
        new = (r * r).sum()
        if it % 50 == 0 and new.item() <= stop:
            break
        p = r + (new / rr) * p
        rr = new
    return {"phi": u + fixed, "cycles": None}


def exact(case, seed):
    if case["kind"] == "poisson":
        st = _prepare_poisson(case, seed)
        return {"phi": _poisson_exact(st["rho"], st["h"]), "cycles": None}
    if case["kind"] == "step" and not case["mcc"]:
        return _step_exact(case, seed)
    if case["kind"] == "embedded" and case["tol"] > 0.0:
        return _embedded_exact(case, seed)
    # collisions follow FP32 random streams particle by particle; fixed numbers of V-cycles have
    # no closed form
    return None
