"""The work this package is measured on: one lab-loop step (or the calls of
one step) per pass, through the classes a lab program uses.

Kinds of case, each over a range of sizes:

* box2d     2D periodic box, one lab step: update_particles, update_fields,
            sort_particles every 20 steps (compaction on or off, charge output
            and current smoothing on or off, pipelined or synchronous calls);
* tracer2d  2D particles pushed in given fields and sorted by cell each step;
* box1d     1D periodic plain PIC, one lab step;
* batch2d   several uneven 2D boxes advanced together through Batch;
* batch1d   several 1D gap runs with pair injection, a few steps per call
            (the round of a served stream);
* logsph    the pulsar lab's step on a log-spherical grid;
* radiation the pulsar lab's photon emission and pair production;
* gap1d     the 1D gap lab's step.

A pass starts from where the last one on the same state ended, as a
simulation does, at the state's own step number.
"""
import dataclasses
import math

import numpy as np
import torch

from aperture3_b200 import Batch, SimData, SimEnvironment, ic, serve
from aperture3_b200 import sim

SORT_INTERVAL = 20
PTC = ("x1", "x2", "x3", "p1", "p2", "p3", "E", "weight", "cell", "id", "flag")


def listed():
    return [
        # the full-size box of the benchmark: particles far beyond L2
        {"name": "box2d_1024x64", "kind": "box2d", "N": 1024, "ppc": 64, "compact": 2,
         "smooth": 0, "rho": False, "sync": False},
        # a large grid with few particles per cell: field, current and order
        # passes weigh as much as the push
        {"name": "box2d_2048x4", "kind": "box2d", "N": 2048, "ppc": 4, "compact": 2,
         "smooth": 0, "rho": False, "sync": False},
        # a small box, where a step is launches and latency
        {"name": "box2d_64x16", "kind": "box2d", "N": 64, "ppc": 16, "compact": 0,
         "smooth": 0, "rho": False, "sync": False},
        # an odd grid with charge output and current smoothing every step and
        # the default synchronous calls, as a lab runs out of the box
        {"name": "box2d_193x30_rho", "kind": "box2d", "N": 193, "ppc": 30, "compact": 0,
         "smooth": 1, "rho": True, "sync": True},
        # test particles in given fields, sorted every step: the cell sort
        {"name": "tracer2d_512x32", "kind": "tracer2d", "N": 512, "ppc": 32},
        # the 1D configuration of the benchmark
        {"name": "box1d_4096x256", "kind": "box1d", "N": 4096, "n": 1 << 20, "sync": False},
        # a small 1D run
        {"name": "box1d_500x32", "kind": "box1d", "N": 500, "n": 16000, "sync": False},
        # uneven boxes in one batch (the batched mode's mix of sides and ppc)
        {"name": "batch2d_4", "kind": "batch2d", "runs": 4, "N_lo": 96, "N_hi": 384,
         "ppc_lo": 16, "ppc_hi": 96, "mix": 3},
        # a round of the served stream of 1D gap runs
        {"name": "batch1d_8", "kind": "batch1d", "runs": 8, "cells_lo": 512,
         "cells_hi": 16384, "ppc_lo": 32, "ppc_hi": 256, "steps": 4, "mix": 5},
        # the pulsar lab's step
        {"name": "logsph_1024x32", "kind": "logsph", "N": 1024, "ppc": 32},
        # its photon emission and pair production
        {"name": "radiation_512x64", "kind": "radiation", "N": 512, "ppc": 64},
        # the 1D gap lab's step
        {"name": "gap1d_8192x256", "kind": "gap1d", "N": 8192, "n": 1 << 21, "smooth": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box2d", "box2d", "tracer2d", "box1d", "batch2d", "batch1d", "logsph",
                       "radiation", "gap1d"])
    mix = rng.randrange(1, 1 << 20)
    if kind in ("box2d", "tracer2d"):
        N = _log_int(rng, 32, 1500)
        ppc = 2 * min(_log_int(rng, 2, 64), max(1, (1 << 24) // (N * N)))
        c = {"kind": kind, "N": N, "ppc": ppc}
        if kind == "box2d":
            c.update(compact=rng.choice([0, 2]), smooth=rng.choice([0, 0, 1, 2]),
                     rho=rng.random() < 0.3, sync=rng.random() < 0.3)
        return c
    if kind == "box1d":
        N = _log_int(rng, 256, 16384)
        n = 2 * _log_int(rng, 4 * N, min(256 * N, 1 << 21))
        return {"kind": kind, "N": N, "n": n, "sync": rng.random() < 0.3}
    if kind == "batch2d":
        lo = _log_int(rng, 64, 192)
        return {"kind": kind, "runs": rng.randint(2, 4), "N_lo": lo, "N_hi": 2 * lo,
                "ppc_lo": 16, "ppc_hi": 2 * rng.randint(16, 64), "mix": mix}
    if kind == "batch1d":
        return {"kind": kind, "runs": rng.randint(2, 8), "cells_lo": 512,
                "cells_hi": _log_int(rng, 1024, 16384), "ppc_lo": 32,
                "ppc_hi": 2 * rng.randint(32, 128), "steps": rng.choice([1, 4, 8]), "mix": mix}
    if kind in ("logsph", "radiation"):
        N = _log_int(rng, 128, 1024)
        return {"kind": kind, "N": N, "ppc": 2 * rng.randint(8, 32)}
    N = _log_int(rng, 512, 16384)
    return {"kind": "gap1d", "N": N, "n": _log_int(rng, 16 * N, min(256 * N, 1 << 21)),
            "smooth": rng.choice([0, 1, 2])}


# ---------------------------------------------------------------------------
# initial states


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _box2d_state(case, seed):
    params, fields, ptc = ic.box2d(seed=seed, N=case["N"], ppc=case["ppc"], device=_dev(),
                                   data_interval=1 if case.get("rho") else 100)
    params.current_smoothing = case.get("smooth", 0)
    return params, fields, ptc


def _box1d_state(case, seed):
    params, fields, ptc = ic.box1d(seed=seed, N=case["N"], num_particles=case["n"], device=_dev())
    params.data_interval = 100
    return params, fields, ptc


def _mix2d(case, seed):
    """(N, ppc) of each run of a batch; the states come from the seed."""
    rng = np.random.default_rng(case["mix"])
    return [{"N": int(rng.integers(case["N_lo"], case["N_hi"] + 1)),
             "ppc": 2 * int(rng.integers(case["ppc_lo"] // 2, case["ppc_hi"] // 2 + 1)),
             "seed": 1000 * seed + r} for r in range(case["runs"])]


def _mix1d(case, seed):
    rng = np.random.default_rng(case["mix"])
    out = []
    for r in range(case["runs"]):
        out.append(serve.GapRequest(
            rid=r, cells=int(rng.integers(case["cells_lo"], case["cells_hi"] + 1)),
            ppc=2 * int(rng.integers(case["ppc_lo"] // 2, case["ppc_hi"] // 2 + 1)),
            steps=1 << 30, ramp=float(rng.uniform(0.1, 10.0)), seed=1000 * seed + r + 1))
    return out


def _gap1d_state(case, seed):
    """A gap of unit length starting at the surface x = 0: E1 a smooth ramp,
    e- / e+ pairs with momenta of both signs, gamma from p1 and beta = x."""
    N, n, guard = case["N"], case["n"], 2
    dx = 1.0 / N
    params = sim.SimParams(N=(N, 1, 1), guard=(guard, 0, 0), lower=(0.0, 0.0, 0.0),
                           size=(1.0, 1.0, 1.0), delta_t=float(np.float32(0.5 * dx)), q_e=1.0,
                           num_species=2, periodic_boundary=(False, False, False),
                           current_smoothing=case["smooth"], max_ptc_number=n, B0=0.7,
                           coord_system="1dgap")
    dev = _dev()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    dims = N + 2 * guard
    x = (torch.arange(dims, device=dev, dtype=torch.float64) - guard + 0.5) / N
    E1 = (0.5 * torch.sin(6.0 * x) + 0.1).float()
    cells = torch.sort(torch.randint(guard + 2, N - 2, (n,), generator=g, device=dev)).values
    x1 = torch.rand(n, generator=g, device=dev)
    p1 = 3.0 * torch.randn(n, generator=g, device=dev)
    beta = (cells - guard + x1.double()) / N
    E = torch.sqrt(1.0 + p1.double() ** 2 + beta ** 2).float()
    zero = torch.zeros(n, device=dev)
    ptc = {"x1": x1, "x2": zero, "x3": zero, "p1": p1, "p2": zero, "p3": zero, "E": E,
           "weight": torch.ones(n, device=dev), "cell": cells,
           "id": torch.arange(n, device=dev),
           "flag": (torch.arange(n, device=dev) % 2) << 29}
    z = torch.zeros(dims, device=dev)
    return params, {"E": [E1, z, z], "B": [z, z, z]}, ptc


def _load(params, fields, ptc, capacity, **kw):
    env = SimEnvironment(params)
    data = SimData(env, capacity=capacity, **kw)
    data.set_fields_device(fields)
    data.set_particles_device(ptc)
    return env, data


def prepare(case, seed):
    k = case["kind"]
    st = {"kind": k, "case": case, "step": 0}
    if k in ("box2d", "tracer2d", "box1d", "gap1d"):
        make = {"box2d": _box2d_state, "tracer2d": _box2d_state, "box1d": _box1d_state,
                "gap1d": _gap1d_state}[k]
        params, fields, ptc = make(case, seed)
        n = ptc["x1"].numel()
        # compaction alternates between the halves of twice the particle count
        env, data = _load(params, fields, ptc, 2 * n if case.get("compact") else n)
        if case.get("compact"):
            env.set_compaction(case["compact"])
        env.set_sync(bool(case.get("sync", False)))
        cls = ((sim.ptc_updater_1dgap, sim.field_solver_1dgap) if k == "gap1d"
               else (sim.ptc_updater, sim.field_solver))
        st.update(env=env, data=data, dt=params.delta_t, pusher=cls[0](env), solver=cls[1](env))
    elif k == "batch2d":
        runs = []
        for spec in _mix2d(case, seed):
            params, fields, ptc = _box2d_state(spec, spec["seed"])
            env, data = _load(params, fields, ptc, 2 * ptc["x1"].numel())
            env.set_compaction(2)
            runs.append(data)
        st.update(runs=runs, batch=Batch(runs))
    elif k == "batch1d":
        runs = [serve.GapRun(req, _dev()) for req in _mix1d(case, seed)]
        st.update(held=runs, runs=[r.data for r in runs], batch=Batch([r.data for r in runs]))
    elif k == "logsph":
        params, fields, ptc = ic.logsph(seed=seed, N=case["N"], ppc=case["ppc"], device=_dev())
        env, data = _load(params, fields, ptc, _logsph_capacity(case))
        env.set_sync(False)
        st.update(env=env, data=data, dt=params.delta_t, omega=params.omega,
                  pusher=sim.ptc_updater_logsph(env), solver=sim.field_solver_logsph(env))
    elif k == "radiation":
        params, fields, ptc = ic.logsph(seed=seed, N=case["N"], ppc=case["ppc"], device=_dev())
        cap = 4 * _logsph_capacity(case)
        params = dataclasses.replace(params, create_pairs=True, rad_model="pulsar",
                                     max_photon_number=cap, max_ptc_number=cap, rad_seed=seed)
        env, data = _load(params, fields, ptc, cap)
        st.update(env=env, data=data, rt=sim.radiative_transfer(env))
    else:
        raise ValueError(k)
    torch.cuda.synchronize()
    return st


def _ptc(data, names=PTC):
    a, b = data.slot_range()
    return {n: data.particles[n][a:b] for n in names}


def _fields(data, rho=False, divs=True):
    out = {"E": list(data.E), "B": list(data.B), "J": list(data.J)}
    if divs:
        out.update(divE=data.divE, divB=data.divB)
    if rho:
        out["Rho"] = list(data.Rho)
    return out


def run(st):
    k, s = st["kind"], st["step"]
    st["step"] = s + 1
    if k in ("box2d", "box1d"):
        data, dt = st["data"], st["dt"]
        st["pusher"].update_particles(data, dt, s)
        st["solver"].update_fields(data, dt, s)
        if s % SORT_INTERVAL == 0 and s != 0:
            data.sort_particles()
        return {"ptc": _ptc(data), **_fields(data, rho=bool(st["case"].get("rho")))}
    if k == "tracer2d":
        data = st["data"]
        st["pusher"].update_particles(data, st["dt"], s)
        data.sort_particles()
        return {"ptc": _ptc(data), "J": list(data.J)}
    if k == "gap1d":
        data = st["data"]
        st["pusher"].update_particles(data, st["dt"], s)
        st["solver"].update_fields(data, st["dt"], s * st["dt"])
        return {"ptc": _ptc(data, ("x1", "p1", "E", "cell")), "E": list(data.E),
                "J": data.J[0], "Rho": list(data.Rho)}
    if k == "batch2d":
        st["batch"].update_particles(s)
        st["batch"].update_fields(s)
        if s % SORT_INTERVAL == 0 and s != 0:
            st["batch"].sort_particles()
        return [{"ptc": _ptc(d, ("x1", "x2", "p1", "p2", "p3", "cell", "id")), "E": list(d.E),
                 "B": list(d.B), "J": list(d.J)} for d in st["runs"]]
    if k == "batch1d":
        n = st["case"]["steps"]
        st["batch"].advance(s * n, n, SORT_INTERVAL, True)
        return [{"ptc": {m: d.particles[m] for m in ("x1", "p1", "p2", "E", "cell", "id")},
                 "E1": d.E[0], "J1": d.J[0]} for d in st["runs"]]
    if k == "logsph":
        data, dt = st["data"], st["dt"]
        st["pusher"].update_particles(data, dt, s)
        st["solver"].update_fields(data, dt, s * dt)
        st["solver"].apply_boundary(data, st["omega"], s * dt)
        if s % SORT_INTERVAL == 0 and s != 0:
            data.sort_particles()
        return {"ptc": dict(data.particles), **_fields(data)}
    # radiation
    data = st["data"]
    em = st["rt"].emit_photons(data)
    pr = st["rt"].produce_pairs(data)
    names = ("p1", "p2", "p3", "E", "cell", "id")
    return {"ptc": {n: data.particles[n] for n in names},
            "photons": {n: data.photons[n] for n in names},
            "photon_produced": data.photon_produced, "pair_produced": data.pair_produced,
            "emitted": em["written"], "pairs": pr["written"]}


# ---------------------------------------------------------------------------
# bytes and operations a pass cannot do without


def _box_work(n, cells, dim):
    # per particle: cell, x1..x3, p1..p3, weight, flag read, cell, x1..x3,
    # p1..p3, E written; per cell: E, B, background fields and J read once, E,
    # B, J and the divergences written once
    return n * 68.0 + cells * 4.0 * (12 + 11), n * (300.0 if dim == 2 else 200.0) + cells * 60.0


def work(case):
    k = case["kind"]
    if k == "box2d":
        cells = (case["N"] + 4) ** 2
        b, f = _box_work(case["N"] ** 2 * case["ppc"], cells, 2)
        # the sort of every 20th step reads and writes the whole record
        return {"bytes": b + case["N"] ** 2 * case["ppc"] * 96.0 / SORT_INTERVAL, "flops": f}
    if k == "tracer2d":
        n = case["N"] ** 2 * case["ppc"]
        return {"bytes": n * (68.0 + 96.0) + 36.0 * (case["N"] + 4) ** 2, "flops": 300.0 * n}
    if k == "box1d":
        b, f = _box_work(case["n"], case["N"] + 4, 1)
        return {"bytes": b + case["n"] * 96.0 / SORT_INTERVAL, "flops": f}
    if k == "gap1d":
        # x1, p1, E, cell, flag, weight read, x1, p1, E, cell written
        return {"bytes": case["n"] * 40.0 + case["N"] * 4.0 * 10, "flops": 60.0 * case["n"]}
    if k == "batch2d":
        b = f = 0.0
        for r in _mix2d(case, 0):
            n = r["N"] ** 2 * r["ppc"]
            x, y = _box_work(n, (r["N"] + 4) ** 2, 2)
            b, f = b + x + n * 96.0 / SORT_INTERVAL, f + y
        return {"bytes": b, "flops": f}
    if k == "batch1d":
        b = f = 0.0
        for r in _mix1d(case, 0):
            n = r.cells * r.ppc
            x, y = _box_work(n, r.cells + 4, 1)
            # injection reads cell and gamma of every particle
            b, f = b + x + n * (8.0 + 96.0 / SORT_INTERVAL), f + y
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    n = _logsph_count(case)
    cells = (case["N"] + 4) ** 2
    if k == "logsph":
        # as the box, and 13 metric coefficients per cell
        b, f = _box_work(n, cells, 2)
        return {"bytes": b + n * 96.0 / SORT_INTERVAL + cells * 4.0 * 13, "flops": f + 300.0 * n}
    # cell, flag, E, x1, x2 of each particle read
    return {"bytes": n * 20.0 + cells * 8.0, "flops": n * 40.0}


def _logsph_count(case):
    """Expected number of particles of ic.logsph: N x N cells, a Poisson number
    of pairs of mean ppc / 2 exp(-(r - 1) / 0.5)."""
    N = case["N"]
    r = np.exp((np.arange(N) + 0.5) * (math.log(50.0) / N))
    return float(N * case["ppc"] * np.exp(-(r - 1.0) / 0.5).sum())


def _logsph_capacity(case):
    """Slots for the particles of any seed (the count's spread is far below 2 %)."""
    return int(1.02 * _logsph_count(case)) + 4096


def tolerance(case):
    # 32-bit results, currents sums of 32-bit products (up to 4e-7 from the
    # 64-bit values), divergences differences of neighbouring 32-bit fields
    # over the cell size: 3e-6 in 2D, 2e-5 on a fine 1D grid
    return {"rel": 1e-4 if case["kind"] == "box1d" else 1e-5, "max": 1e-3, "differ": 1e-6}


# ---------------------------------------------------------------------------
# the same step in 64 bits (torch only)

D = torch.float64
STAG = [(0, 1), (1, 0), (1, 1), (1, 0), (0, 1), (0, 0)]  # E1..E3, B1..B3 (x, y)


def _cic(d):
    return torch.clamp(1.0 - d.abs(), min=0.0)


def _gather2(f, st, x1, x2, c1, c2):
    """CIC interpolation of one component: a node with stagger 1 sits at the
    upper edge of its cell, with stagger 0 at its centre."""
    acc = torch.zeros_like(x1)
    for dj in (-1, 0, 1):
        wy = _cic(dj + (1.0 if st[1] else 0.5) - x2)
        for di in (-1, 0, 1):
            acc += f[c2 + dj, c1 + di] * _cic(di + (1.0 if st[0] else 0.5) - x1) * wy
    return acc


def _gather1(f, st, x1, c1):
    acc = torch.zeros_like(x1)
    for di in (-1, 0, 1):
        acc += f[c1 + di] * _cic(di + (1.0 if st else 0.5) - x1)
    return acc


def _vay(p, e, b):
    """Vay's push; e and b carry the factor q dt / (2 m)."""
    g = torch.sqrt(1 + p[0] ** 2 + p[1] ** 2 + p[2] ** 2)
    cr = lambda u, w: (u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2],  # noqa: E731
                       u[0] * w[1] - u[1] * w[0])
    c = cr(p, b)
    up = [p[i] + 2 * e[i] + c[i] / g for i in range(3)]
    tt = sum(x * x for x in b)
    ut = sum(x * y for x, y in zip(up, b))
    sg = 1 + sum(x * x for x in up) - tt
    ig2 = 2 / (sg + torch.sqrt(sg * sg + 4 * (tt + ut * ut)))
    s = 1 / (1 + ig2 * tt)
    g = 1 / torch.sqrt(ig2)
    c = cr(up, b)
    return [(up[i] + b[i] * ut * ig2 + c[i] / g) * s for i in range(3)], g


def _fold(a, n0, n1, g):
    """The guard strips of one rank's periodic box added to the bulk images."""
    if n1 > 1:
        a[:, n0 - 2 * g:n0 - g] += a[:, 0:g]
        a[:, g:2 * g] += a[:, n0 - g:n0]
        low, up = a[0:g].clone(), a[n1 - g:n1].clone()
        a[n1 - 2 * g:n1 - g] += low
        a[g:2 * g] += up
    else:
        low, up = a[:, 0:g].clone(), a[:, n0 - g:n0].clone()
        a[:, n0 - 2 * g:n0 - g] += low
        a[:, g:2 * g] += up


def _images(a, g):
    n1, n0 = a.shape
    if n1 > 1:
        a[:, n0 - g:] = a[:, g:2 * g]
        a[:, :g] = a[:, n0 - 2 * g:n0 - g]
        a[n1 - g:] = a[g:2 * g]
        a[:g] = a[n1 - 2 * g:n1 - g]
    else:
        a[:, n0 - g:] = a[:, g:2 * g]
        a[:, :g] = a[:, n0 - 2 * g:n0 - g]


def _smooth2(a, g):
    n1, n0 = a.shape
    c = lambda dx, dy: a[g + dy:n1 - g + dy, g + dx:n0 - g + dx]  # noqa: E731
    v = (0.25 * c(0, 0) + 0.125 * (c(1, 0) + c(-1, 0) + c(0, 1) + c(0, -1))
         + 0.0625 * (c(1, 1) + c(-1, 1) + c(1, -1) + c(-1, -1)))
    a[g:n1 - g, g:n0 - g] = v
    _images(a, g)


def _push2(F, dt, dx, ptc, dims0):
    """Chunks of (pushed momenta, gamma, old and new offsets, cell moves)."""
    n = ptc["x1"].numel()
    for lo in range(0, n, 1 << 21):
        s = slice(lo, min(n, lo + (1 << 21)))
        x = [ptc[k][s].to(D) for k in ("x1", "x2", "x3")]
        p = [ptc[k][s].to(D) for k in ("p1", "p2", "p3")]
        q = torch.where((ptc["flag"][s] >> 29) == 0, -1.0, 1.0).to(D)
        c1, c2 = ptc["cell"][s] % dims0, ptc["cell"][s] // dims0
        f = [_gather2(F[k], STAG[k], x[0], x[1], c1, c2) * q * (0.5 * dt) for k in range(6)]
        p, gam = _vay(p, f[:3], f[3:])
        yield s, q * ptc["weight"][s].to(D), x, p, gam, c1, c2


def _exact_box2d(params, fields, ptc, rho, divs=True, step_fields=True):
    N, g = params.N[0], 2
    dims = N + 2 * g
    dt, dx = float(params.delta_t), 1.0 / N
    dev = ptc["x1"].device
    F = [f.to(D) for f in fields["E"] + fields["B"]]
    zero = lambda: torch.zeros((dims, dims), dtype=D, device=dev)  # noqa: E731
    J, R = [zero() for _ in range(3)], [zero(), zero()]
    out = {k: torch.empty_like(ptc["x1"], dtype=D) for k in ("x1", "x2", "x3", "p1", "p2", "p3",
                                                             "E")}
    for s, w, x, p, gam, c1, c2 in _push2(F, dt, dx, ptc, dims):
        v = [p[i] / gam for i in range(3)]
        n1, n2 = x[0] + v[0] * dt / dx, x[1] + v[1] * dt / dx
        d1, d2 = torch.floor(n1), torch.floor(n2)
        for i in range(3):
            out["p%d" % (i + 1)][s] = p[i]
        out["E"][s] = gam
        out["x1"][s], out["x2"][s], out["x3"][s] = n1 - d1, n2 - d2, x[2] + v[2] * dt
        # Esirkepov's decomposition over the nodes -2..1 around the old cell
        nodes = (-2, -1, 0, 1)
        sx0 = [_cic(i + 1 - x[0]) for i in nodes]
        sx1 = [_cic(i + 1 - n1) for i in nodes]
        sy0 = [_cic(j + 1 - x[1]) for j in nodes]
        sy1 = [_cic(j + 1 - n2) for j in nodes]
        at = c2 * dims + c1
        sp = (ptc["flag"][s] >> 29) == 1
        djy = [torch.zeros_like(w) for _ in nodes]
        for b, j in enumerate(nodes):
            djx = torch.zeros_like(w)
            for a, i in enumerate(nodes):
                o = at + j * dims + i
                djx = djx + (sx1[a] - sx0[a]) * 0.5 * (sy0[b] + sy1[b])
                djy[a] = djy[a] + (sy1[b] - sy0[b]) * 0.5 * (sx0[a] + sx1[a])
                c = (2 * sx1[a] * sy1[b] + sx0[a] * sy1[b] + sx1[a] * sy0[b]
                     + 2 * sx0[a] * sy0[b]) / 6
                if i < 1:
                    J[0].view(-1).index_add_(0, o + 1, -w * djx)
                if j < 1:
                    J[1].view(-1).index_add_(0, o + dims, -w * djy[a])
                J[2].view(-1).index_add_(0, o, w * v[2] * c)
                if rho:
                    r = w * sx1[a] * sy1[b]
                    for k in range(2):
                        R[k].view(-1).index_add_(0, o, torch.where(sp == bool(k), r, 0.0))
    for a in J + R:
        _fold(a, dims, dims, g)
    for _ in range(params.current_smoothing):
        for a in J + R:
            _smooth2(a, g)
    res = {"ptc": {**{k: None for k in PTC}, **out}, "J": J}
    if not step_fields:
        return res
    E, B = F[:3], F[3:]
    id_ = 1.0 / dx
    c = lambda a, dx_=0, dy=0: a[g + dy:dims - g + dy, g + dx_:dims - g + dx_]  # noqa: E731

    def upd_e(h):
        new = [c(E[0]) + h * ((c(B[2], 0, 1) - c(B[2])) * id_ - c(J[0])),
               c(E[1]) + h * ((c(B[2]) - c(B[2], 1)) * id_ - c(J[1])),
               c(E[2]) + h * ((c(B[1], 1) - c(B[1])) * id_ + (c(B[0]) - c(B[0], 0, 1)) * id_
                              - c(J[2]))]
        for a, v in zip(E, new):
            c(a).copy_(v)
            _images(a, g)

    upd_e(0.5 * dt)
    new = [c(B[0]) - dt * (c(E[2]) - c(E[2], 0, -1)) * id_,
           c(B[1]) - dt * (c(E[2], -1) - c(E[2])) * id_,
           c(B[2]) - dt * ((c(E[1]) - c(E[1], -1)) * id_ + (c(E[0], 0, -1) - c(E[0])) * id_)]
    for a, v in zip(B, new):
        c(a).copy_(v)
        _images(a, g)
    upd_e(dt)
    res.update(E=E, B=B)
    if divs:
        dE, dB = zero(), zero()
        c(dE).copy_((c(E[0], 1) - c(E[0])) * id_ + (c(E[1], 0, 1) - c(E[1])) * id_)
        c(dB).copy_((c(B[0]) - c(B[0], -1)) * id_ + (c(B[1]) - c(B[1], 0, -1)) * id_)
        res.update(divE=dE, divB=dB)
    if rho:
        res["Rho"] = R
    return res


def _exact_box1d(params, fields, ptc):
    N, g = params.N[0], 2
    dims = N + 2 * g
    dt, dx = float(params.delta_t), 1.0 / N
    dev = ptc["x1"].device
    F = [f.reshape(-1).to(D) for f in fields["E"] + fields["B"]]
    x = [ptc[k].to(D) for k in ("x1", "x2", "x3")]
    p = [ptc[k].to(D) for k in ("p1", "p2", "p3")]
    q = torch.where((ptc["flag"] >> 29) == 0, -1.0, 1.0).to(D)
    w, c1 = q * ptc["weight"].to(D), ptc["cell"]
    f = [_gather1(F[k], STAG[k][0], x[0], c1) * q * (0.5 * dt) for k in range(6)]
    p, gam = _vay(p, f[:3], f[3:])
    v = [p[i] / gam for i in range(3)]
    n1 = x[0] + v[0] * dt / dx
    J = [torch.zeros((1, dims), dtype=D, device=dev) for _ in range(3)]
    djx = torch.zeros_like(w)
    for i in (-2, -1, 0, 1):
        s0, s1 = _cic(i + 1 - x[0]), _cic(i + 1 - n1)
        djx = djx + s1 - s0
        if i < 1:
            J[0].view(-1).index_add_(0, c1 + i + 1, -w * djx)
        for k in (1, 2):
            J[k].view(-1).index_add_(0, c1 + i, w * v[k] * 0.5 * (s0 + s1))
    for a in J:
        _fold(a, dims, 1, g)
    out = {"p1": p[0], "p2": p[1], "p3": p[2], "E": gam, "x1": n1 - torch.floor(n1),
           "x2": x[1] + v[1] * dt, "x3": x[2] + v[2] * dt}
    E, B = [a.reshape(1, -1) for a in F[:3]], [a.reshape(1, -1) for a in F[3:]]
    id_ = 1.0 / dx
    c = lambda a, s=0: a[:, g + s:dims - g + s]  # noqa: E731

    def upd_e(h):
        new = [c(E[0]) - h * c(J[0]), c(E[1]) + h * ((c(B[2]) - c(B[2], 1)) * id_ - c(J[1])),
               c(E[2]) + h * ((c(B[1], 1) - c(B[1])) * id_ - c(J[2]))]
        for a, u in zip(E, new):
            c(a).copy_(u)
            _images(a, g)

    upd_e(0.5 * dt)
    new = [c(B[1]) - dt * (c(E[2], -1) - c(E[2])) * id_,
           c(B[2]) - dt * (c(E[1]) - c(E[1], -1)) * id_]
    for a, u in zip(B[1:], new):
        c(a).copy_(u)
        _images(a, g)
    _images(B[0], g)
    upd_e(dt)
    dE, dB = torch.zeros_like(J[0]), torch.zeros_like(J[0])
    c(dE).copy_((c(E[0], 1) - c(E[0])) * id_)
    c(dB).copy_((c(B[0]) - c(B[0], -1)) * id_)
    return {"ptc": {**{k: None for k in PTC}, **out}, "E": E, "B": B, "J": J, "divE": dE,
            "divB": dB}


def _exact_gap1d(params, fields, ptc):
    N, g = params.N[0], 2
    dims = N + 2 * g
    dt, dx = float(params.delta_t), 1.0 / N
    dev = ptc["x1"].device

    def smooth(a):
        for _ in range(params.current_smoothing):
            z = torch.cat([a.new_zeros(1), a, a.new_zeros(1)])
            up, dn = z[2:].clone(), z[:-2].clone()
            up[dims - g - 1] = a[dims - g - 1]
            dn[g] = a[g]
            a = 0.5 * a + 0.25 * up + 0.25 * dn
        return a

    E1 = fields["E"][0].to(D).reshape(-1)
    E3 = smooth(E1)
    x, p, gam, c1 = (ptc[k].to(D) for k in ("x1", "p1", "E", "cell"))
    c1 = ptc["cell"]
    q = torch.where((ptc["flag"] >> 29) == 0, -1.0, 1.0).to(D)
    p = p + _gather1(E3, 0, x, c1) * q * dt
    beta = (c1 - g + x) * dx
    p = p + beta / gam * ((gam - p) / (1 + beta * beta)) ** 2 * dt
    vr = (p / torch.sqrt(1 + p * p + beta * beta) + beta * beta) / (1 + beta * beta)
    n1 = x + vr * dt / dx
    d1 = torch.floor(n1)
    bn = (c1 + d1 - g + n1 - d1) * dx
    J = torch.zeros(dims, dtype=D, device=dev)
    R = [torch.zeros(dims, dtype=D, device=dev) for _ in range(2)]
    w = q * ptc["weight"].to(D)
    sp = (ptc["flag"] >> 29) == 1
    dj = torch.zeros_like(w)
    for i in (-2, -1, 0, 1):
        s0, s1 = _cic(i + 1 - x), _cic(i + 1 - n1)
        dj = dj + s1 - s0
        if i < 1:
            J.index_add_(0, c1 + i + 1, -w * dj * dx / dt)
        for k in range(2):
            R[k].index_add_(0, c1 + i, torch.where(sp == bool(k), w * s1, 0.0))
    J, R = smooth(J), [smooth(a) for a in R]
    En = E1.clone()
    s = slice(g + 1, dims - g - 1)
    En[s] += (1.6 * float(np.float32(params.B0)) - J[s]) * dt
    row = lambda a: a.reshape(1, -1)  # noqa: E731
    return {"ptc": {"x1": n1 - d1, "p1": p, "E": torch.sqrt(1 + p * p + bn * bn), "cell": None},
            "E": [row(En), None, row(E3)], "J": row(J), "Rho": [row(a) for a in R]}


def _exact_logsph_particles(params, fields, ptc, capacity):
    """The particles of the log-spherical step: Vay's push, the move in
    Cartesian space, the reflection at the axis. Fields and currents of that
    grid have no plain form here."""
    N, g = params.N[0], 2
    dims = N + 2 * g
    dt = float(params.delta_t)
    d1, d2 = (float(np.float32(np.float32(params.size[i]) / np.float32(N))) for i in range(2))
    F = [f.to(D) for f in fields["E"] + fields["B"]]
    # slots past the particles hold zeros
    out = {k: torch.zeros(capacity, dtype=D, device=F[0].device) for k in ("p1", "p2", "p3", "E")}
    for s, w, x, p, gam, c1, c2 in _push2(F, dt, d1, ptc, dims):
        r, th = torch.exp((c1 - g + x[0]) * d1), (c2 - g + x[1]) * d2
        gam = torch.sqrt(1 + p[0] ** 2 + p[1] ** 2 + p[2] ** 2)
        v = [a / gam for a in p]
        st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(x[2]), torch.cos(x[2])
        vx = v[0] * st * cp + v[1] * ct * cp - v[2] * sp
        vy = v[0] * st * sp + v[1] * ct * sp + v[2] * cp
        vz = v[0] * ct - v[1] * st
        X, Y, Z = r * st * cp + vx * dt, r * st * sp + vy * dt, r * ct + vz * dt
        rn = torch.sqrt(X * X + Y * Y + Z * Z)
        tn, pn = torch.acos(Z / rn), torch.atan2(Y, X)
        st, ct, sp, cp = torch.sin(tn), torch.cos(tn), torch.sin(pn), torch.cos(pn)
        q1 = vx * st * cp + vy * st * sp + vz * ct
        q2 = vx * ct * cp + vy * ct * sp - vz * st
        q3 = -vx * sp + vy * cp
        out["p1"][s], out["p2"][s], out["p3"][s] = q1 * gam, q2 * gam, q3 * gam
        out["E"][s] = gam
    return {"ptc": {**{k: None for k in PTC}, **out}, "E": None, "B": None, "J": None,
            "divE": None, "divB": None}


def exact(case, seed):
    k = case["kind"]
    if k == "box2d":
        st = _box2d_state(case, seed)
        return _exact_box2d(*st, rho=bool(case.get("rho")))
    if k == "tracer2d":
        # the sorted order has no 64-bit counterpart; the current has
        r = _exact_box2d(*_box2d_state(case, seed), rho=False, step_fields=False)
        return {"ptc": {n: None for n in PTC}, "J": r["J"]}
    if k == "box1d":
        return _exact_box1d(*_box1d_state(case, seed))
    if k == "gap1d":
        return _exact_gap1d(*_gap1d_state(case, seed))
    if k == "batch2d":
        out = []
        for spec in _mix2d(case, seed):
            r = _exact_box2d(*_box2d_state(spec, spec["seed"]), rho=False)
            out.append({"ptc": {n: (r["ptc"][n] if n not in ("cell", "id") else None)
                                for n in ("x1", "x2", "p1", "p2", "p3", "cell", "id")},
                        "E": r["E"], "B": r["B"], "J": r["J"]})
        return out
    if k == "logsph":
        st = ic.logsph(seed=seed, N=case["N"], ppc=case["ppc"], device=_dev())
        return _exact_logsph_particles(*st, _logsph_capacity(case))
    # batch1d and radiation: random draws decide which particles appear
    return None
