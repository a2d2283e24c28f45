"""The work that a user of armon_gb300 has it do, as cases that can be timed and compared.

A case names a public entry point (`kind`), a domain or a set of domains, the options of the step and a
number of cycles.  The kinds:

  solver   a `Solver` kept over many solves; a solve starts from init_test (`state` "circ": the circular Sod
           problem of the benchmark) or from fields that the caller holds (`state` "flow": a smooth flow that
           moves everywhere, as a restart from a developed field is), and its fields are what comes back.
           FP64 callers copy their device fields into the solver's arrays; FP32 solvers have no FP64 device
           arrays, so their callers upload and download pinned host arrays.
  host     `armon_solve_host`'s call: host arrays in, host arrays out, nothing kept.
  batch    a `Batch` kept over many sets of domains: the set joins, runs to its end, is read and leaves.
  serve    a `Server` kept over many requests: requests are submitted, rounds run until all are done, the
           results are read and released.
  stages   the reference's own kernel entry points, one by one, as a host program that drives the step
           itself calls them.

`exact` is the reference's step written in plain torch operations in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "armon-kokkos_gb300"))

import armon_gb300 as A  # noqa: E402
from armon_gb300 import workloads as W  # noqa: E402

FIELDS = ("rho", "umat", "vmat", "Emat")
GHOSTS = 5


def case(name, kind, nx=0, ny=0, precision=64, cycles=0, state="circ", scheme="GAD", projection="euler_2nd",
         limiter="Minmod", splitting="Sequential", domains=0, t_end=0.0, largest=0):
    c = dict(kind=kind, nx=nx, ny=ny, precision=precision, cycles=cycles, state=state, scheme=scheme,
             projection=projection, limiter=limiter, splitting=splitting, domains=domains, t_end=t_end,
             largest=largest)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest solves: a smoke or unit test, where launches and latency are all there is
        case("solver_f64_96x64", "solver", 96, 64, 64, 20),
        # the reference's own problem size (its tests run 100 x 100), with its symmetric splitting
        case("solver_f64_100x100", "solver", 100, 100, 64, 100, splitting="SequentialSym"),
        # one call with host arrays, nothing kept: a script's use of the library
        case("host_f64_512x300", "host", 512, 300, 64, 60, state="flow"),
        # odd sizes with the cheap scheme and a flow that moves everywhere
        case("solver_f64_1001x573_godunov", "solver", 1001, 573, 64, 40, state="flow", scheme="Godunov",
             projection="euler"),
        # a restart: every cell differs from its neighbours, so every position is computed
        case("solver_f64_2048_flow", "solver", 2048, 2048, 64, 24, state="flow"),
        # the benchmark: circular Sod, 200 cycles
        case("solver_f64_4096_circ", "solver", 4096, 4096, 64, 200),
        # the FP32 variant at its benchmark size
        case("solver_f32_8192_circ", "solver", 8192, 8192, 32, 100),
        # FP32, a moving flow, odd sizes, the third limiter and the three-pass splitting
        case("solver_f32_1777x1291_flow", "solver", 1777, 1291, 32, 40, state="flow", limiter="Superbee",
             splitting="Strang"),
        # uneven domains advanced together (the batched benchmark's mix, a sixteenth of it)
        case("batch_f64_mixed16", "batch", precision=64, domains=16, t_end=0.05, largest=1024),
        # many small FP32 domains, a parameter study
        case("batch_f32_small48", "batch", precision=32, domains=48, cycles=80, largest=256),
        # a burst of requests in both precisions through the server
        case("serve_mixed24", "serve", precision=0, domains=24, t_end=0.03, largest=1024),
        # the reference's kernel ABI, a host program driving every stage
        case("stages_f64_1500x1000", "stages", 1500, 1000, 64, 4, state="flow"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    scheme = rng.choice(["GAD", "GAD", "GAD", "Godunov"])
    opts = dict(scheme=scheme, projection=rng.choice(["euler_2nd", "euler_2nd", "euler"]),
                limiter=rng.choice(["Minmod", "Minmod", "Superbee", "None"]),
                splitting=rng.choice(["Sequential", "Sequential", "SequentialSym", "Strang"]))
    kind = rng.choice(["solver"] * 6 + ["host", "batch", "batch", "serve", "stages"])
    if kind == "solver" or kind == "host":
        cells = log(4e3, 1.6e7 if kind == "solver" else 1e6)
        aspect = math.exp(rng.uniform(-1.2, 1.2))
        nx = max(16, int(math.sqrt(cells * aspect)))
        ny = max(16, int(cells / nx))
        state = rng.choice(["circ", "flow"]) if kind == "solver" else "flow"
        cycles = max(4, min(log(20, 200), int(2.4e8 / cells) if state == "flow" else int(1.6e9 / cells)))
        precision = rng.choice([64, 64, 32]) if kind == "solver" else 64
        return case(None, kind, nx, ny, precision, cycles, state, **opts)
    if kind == "stages":
        return case(None, kind, log(64, 2000), log(64, 2000), 64, rng.randint(1, 8), "flow", scheme=scheme,
                    limiter=opts["limiter"])
    largest = rng.choice([128, 256, 512, 1024])
    domains = rng.randint(8, 20 if largest > 256 else 60)
    if kind == "serve":
        return case(None, kind, precision=0, domains=domains, t_end=round(rng.uniform(0.01, 0.04), 4), largest=largest)
    if rng.random() < 0.5:
        return case(None, kind, precision=64, domains=domains, t_end=round(rng.uniform(0.02, 0.05), 4),
                    largest=largest)
    return case(None, kind, precision=rng.choice([32, 64]), domains=domains, cycles=rng.randint(20, 120),
                largest=largest)


# ---- inputs ----

def step_case(c, nx, ny, **more):
    # the fields of a flow are the caller's, so the mirrored band covers every ghost cell that is read
    return A.Case(test="Sod_circ", scheme=c["scheme"], projection=c["projection"], limiter=c["limiter"],
                  splitting=c["splitting"], nghost=GHOSTS, nx=nx, ny=ny, stencil=GHOSTS, cfl=0.6, **more)


def circ_radius2(seed):
    # the benchmark's squared radius is 0.04, the reference's 0.09
    return float(np.random.default_rng(seed).uniform(0.035, 0.06))


def flow_fields(c, seed):
    """A smooth periodic-looking flow of a few Fourier modes: density and pressure within a factor of three,
    Mach numbers up to about one half, no two neighbouring cells alike.  Device FP64, ghosts included."""
    r = np.random.default_rng(seed)
    col, row = c["ny"] + 2 * GHOSTS, c["nx"] + 2 * GHOSTS
    y = ((torch.arange(col, dtype=torch.float64, device="cuda") - GHOSTS + 0.5) / c["ny"])[:, None]
    x = ((torch.arange(row, dtype=torch.float64, device="cuda") - GHOSTS + 0.5) / c["nx"])[None, :]

    def modes(amplitude):
        f = torch.zeros(col, row, dtype=torch.float64, device="cuda")
        for _ in range(4):
            kx, ky, ph = r.integers(1, 7), r.integers(1, 7), r.uniform(0, 2 * math.pi)
            f += torch.sin(2 * math.pi * (kx * x + ky * y) + ph) * (amplitude / 4 * r.uniform(0.5, 1.5))
        return f

    rho = torch.exp(modes(0.5))
    p = torch.exp(modes(0.4))
    u, v = modes(0.5), modes(0.5)
    E = p / (0.4 * rho) + 0.5 * (u * u + v * v)
    return dict(zip(FIELDS, (rho, u, v, E)))


def specs(c, seed):
    """The domains of a batch or of a burst of requests: the benchmark mixes' draws.  The sizes belong to the
    case, the states to the seed."""
    sizes = np.random.default_rng(c["domains"] * 7919 + c["largest"])
    r = np.random.default_rng(seed)
    sides = [s for s in W.SIDES if s <= c["largest"]]
    out = []
    for k in range(c["domains"]):
        if c["kind"] == "serve":   # square, any multiple of 16, a heavy tail
            nx = ny = max(128, int(min(sizes.lognormal(5.8, 0.6), c["largest"])) // 16 * 16)
        else:
            nx, ny = int(sizes.choice(sides)), int(sizes.choice(sides))
        precision = c["precision"] or (64 if sizes.random() < 0.5 else 32)
        out.append(W.DomainSpec(nx=nx, ny=ny, kind="planar" if r.random() < 0.5 else "circular",
                                pos=float(r.uniform(0.3, 0.7)), angle=float(r.uniform(0, np.pi)),
                                rho_l=float(r.uniform(0.5, 2.0)), rho_r=float(r.uniform(0.05, 0.3)),
                                p_l=float(r.uniform(0.5, 2.0)), p_r=float(r.uniform(0.05, 0.3)),
                                t_end=c["t_end"], precision=precision, splitting=c["splitting"]))
    return out


def spec_params(c, spec):
    ends = dict(max_cycles=c["cycles"], max_time=1e9) if c["cycles"] else dict(max_cycles=1_000_000, max_time=c["t_end"])
    return A.make_params(step_case(c, spec.nx, spec.ny, **ends))


class DeviceArray:
    """A device array of a solver, for torch.as_tensor: the tensor keeps this object, which keeps the solver
    and so the memory."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": None}


def device_view(solver, name):
    p = solver.params
    return torch.as_tensor(DeviceArray(solver, solver.device_array(name), p.nb_cells),
                           device="cuda").view(p.col_length, p.row_length)


def real(t, c):
    return t.view(c["ny"] + 2 * GHOSTS, c["nx"] + 2 * GHOSTS)[GHOSTS:-GHOSTS, GHOSTS:-GHOSTS]


def prepare(c, seed):
    return {"solver": prepare_solver, "host": prepare_host, "batch": prepare_batch, "serve": prepare_serve,
            "stages": prepare_stages}[c["kind"]](c, seed)


def run(state):
    return {"solver": run_solver, "host": run_host, "batch": run_batch, "serve": run_serve,
            "stages": run_stages}[state["case"]["kind"]](state)


# ---- solver ----

def prepare_solver(c, seed):
    option = circ_radius2(seed) if c["state"] == "circ" else 0.04
    stream = torch.cuda.Stream()
    s = A.Solver(step_case(c, c["nx"], c["ny"], max_cycles=c["cycles"], max_time=1e9, test_option=option),
                 precision=c["precision"], stream=stream.cuda_stream)
    st = {"case": c, "solver": s, "stream": stream}
    if c["state"] == "flow":
        s.init_test()
        st["fields"] = flow_fields(c, seed)
        if c["precision"] == 32:
            st["fields"] = {k: f.cpu().pin_memory() for k, f in st["fields"].items()}
    if c["precision"] == 32:
        st["out"] = {k: torch.empty(s.params.nb_cells, dtype=torch.float64, pin_memory=True) for k in FIELDS + ("pmat",)}
    else:
        # a solve ends with its fields in these arrays
        st["out"] = {k: device_view(s, k) for k in FIELDS + ("pmat",)}
    torch.cuda.synchronize()
    return st


def run_solver(st):
    c, s = st["case"], st["solver"]
    L, h = A.lib(), s._h
    if c["state"] == "circ":
        s.init_test()
    else:
        for k, f in st["fields"].items():
            if c["precision"] == 32:
                A.check(L.armon_solver_upload(h, A.ARRAYS.index(k), f.data_ptr()))
            else:
                with torch.cuda.stream(st["stream"]):
                    st["out"][k].copy_(f)
        s.begin_loop()
    s.run()
    p, _ = s.state()
    out = {"time": p.time, "dt": p.next_cycle_dt, "cycles": p.cycle}
    for k in FIELDS + ("pmat",):
        if c["precision"] == 32:
            A.check(L.armon_solver_download(h, A.ARRAYS.index(k), st["out"][k].data_ptr()))
        out[k] = real(st["out"][k], c)
    return out


# ---- host arrays in, host arrays out ----

def prepare_host(c, seed):
    return {"case": c, "inputs": {k: f.reshape(-1).cpu().numpy() for k, f in flow_fields(c, seed).items()},
            "step": step_case(c, c["nx"], c["ny"], max_cycles=c["cycles"], max_time=1e9)}


def run_host(st):
    c = st["case"]
    p, out = A.solve_host(st["step"], st["inputs"])
    r = {k: A.real_cells(p, a) for k, a in out.items()}
    return {**r, "time": p.time, "dt": p.next_cycle_dt, "cycles": p.cycle}


# ---- batch ----

def prepare_batch(c, seed):
    return {"case": c, "batch": A.Batch(precision=c["precision"]),
            "domains": [(spec_params(c, s), s.sod_interface()) for s in specs(c, seed)]}


def run_batch(st):
    b = st["batch"]
    ids = [b.add_sod(p, i) for p, i in st["domains"]]
    b.run()
    out = {"rho": [], "time": [], "cycles": []}
    for k in ids:
        p, _ = b.state(k)
        out["rho"].append(A.real_cells(b.params[k], b.download(k, "rho")).ravel())
        out["time"].append(p.time)
        out["cycles"].append(p.cycle)
        b.remove(k)
    return {"rho": np.concatenate(out["rho"]), "time": np.array(out["time"]), "cycles": np.array(out["cycles"])}


# ---- server ----

def prepare_serve(c, seed):
    return {"case": c, "server": A.Server(),
            "requests": [(spec_params(c, s), s.precision, s.sod_interface()) for s in specs(c, seed)]}


def run_serve(st):
    srv = st["server"]
    ids = [srv.submit(p, prec, i) for p, prec, i in st["requests"]]
    got = {}
    while len(got) < len(ids):
        srv.step()
        while (r := srv.next_done()) is not None:
            info = srv.info(r)
            got[r] = (A.real_cells(srv.params[r], srv.download(r, "rho")).ravel(), info.time)
            srv.release(r)
    out = {}
    for prec in (64, 32):
        mine = [got[r] for r, q in zip(ids, st["requests"]) if q[1] == prec]
        if mine:
            out[f"rho{prec}"] = np.concatenate([m[0] for m in mine])
            out[f"time{prec}"] = np.array([m[1] for m in mine])
    return out


# ---- the reference's kernels, one by one ----

ARRAYS16 = ("rho", "umat", "vmat", "Emat", "pmat", "cmat", "gmat", "ustar", "pstar", "work_array_1", "work_array_2",
            "work_array_3", "work_array_4", "domain_mask")


def prepare_stages(c, seed):
    n = (c["nx"] + 2 * GHOSTS) * (c["ny"] + 2 * GHOSTS)
    t = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k in ARRAYS16}
    real(t["domain_mask"], c).fill_(1.0)
    K = A.lib()
    P, I, F = C.c_void_p, C.c_int64, C.c_double
    K.perfect_gas_EOS.argtypes = [P, P, F] + [P] * 7
    K.boundary_conditions.argtypes = [P, P, I, I, F, F] + [P] * 7
    K.acoustic.argtypes = [P, P, I] + [P] * 6
    K.acoustic_GAD.argtypes = [P, P, I, F, F] + [P] * 6 + [C.c_int32]
    K.cell_update.argtypes = [P, P, I, F, F] + [P] * 5
    K.advection_second_order.argtypes = [P, P, I, F, F] + [P] * 9
    K.euler_projection.argtypes = [P, P, I, F, F] + [P] * 9
    K.dt_CFL.argtypes = [P, P, F, F] + [P] * 4
    torch.cuda.synchronize()
    return {"case": c, "t": t, "v": {k: A.View(x.data_ptr(), n, None) for k, x in t.items()},
            "fields": {k: f.reshape(-1) for k, f in flow_fields(c, seed).items()}}


def run_stages(st):
    c, K = st["case"], A.lib()
    nx, ny, R = c["nx"], c["ny"], c["nx"] + 2 * GHOSTS
    v = {k: C.byref(x) for k, x in st["v"].items()}
    K.armon_kernels_set_stream(torch.cuda.current_stream().cuda_stream)
    for k, f in st["fields"].items():
        st["t"][k].copy_(f)

    def box(axis, lo, hi):
        # the real cells, widened by lo and hi positions along the axis
        i0, i1 = (-lo, nx + hi) if axis == 0 else (0, nx)
        j0, j1 = (-lo, ny + hi) if axis == 1 else (0, ny)
        return (C.byref(A.Range(0, (i1 - i0) * (j1 - j0))),
                C.byref(A.InnerRange2D((j0 + GHOSTS) * R, R, i0 + GHOSTS, i1 - i0)))

    def eos():
        K.perfect_gas_EOS(*box(0, 0, 0), 1.4, v["rho"], v["Emat"], v["umat"], v["vmat"], v["pmat"], v["cmat"], v["gmat"])

    first = GHOSTS * R + GHOSTS
    work = [v["work_array_%d" % k] for k in (1, 2, 3, 4)]
    time = dt = 0.0
    eos()
    for _ in range(c["cycles"]):
        local = K.dt_CFL(C.byref(A.Range(0, R * ny - 2 * GHOSTS)), C.byref(A.InnerRange1D(first, 1)), 1.0 / nx, 1.0 / ny,
                         v["umat"], v["vmat"], v["cmat"], v["domain_mask"])
        new = 0.6 * local if dt == 0 else min(0.6 * local, 1.05 * dt)
        dt, cur = new, (dt or new)
        for axis in (0, 1):
            s, dx, u = (1, 1.0 / nx, v["umat"]) if axis == 0 else (R, 1.0 / ny, v["vmat"])
            eos()
            n, step, far = (ny, R, nx) if axis == 0 else (nx, 1, ny)
            for start, disp in ((first - s, s), (first + far * s, -s)):
                K.boundary_conditions(C.byref(A.Range(0, n)), C.byref(A.InnerRange1D(start, step)), GHOSTS, disp,
                                      -1.0 if axis == 0 else 1.0, -1.0 if axis == 1 else 1.0, v["rho"], v["umat"],
                                      v["vmat"], v["pmat"], v["cmat"], v["gmat"], v["Emat"])
            if c["scheme"] == "GAD":
                K.acoustic_GAD(*box(axis, 2, 3), s, cur, dx, v["ustar"], v["pstar"], v["rho"], u, v["pmat"], v["cmat"],
                               A.LIMITERS[c["limiter"]])
            else:
                K.acoustic(*box(axis, 2, 3), s, v["ustar"], v["pstar"], v["rho"], u, v["pmat"], v["cmat"])
            K.cell_update(*box(axis, 2, 2), s, dx, cur, v["ustar"], v["pstar"], v["rho"], u, v["Emat"])
            K.advection_second_order(*box(axis, 0, 1), s, dx, cur, v["ustar"], v["rho"], v["umat"], v["vmat"], v["Emat"],
                                     *work)
            K.euler_projection(*box(axis, 0, 0), s, dx, cur, v["ustar"], v["rho"], v["umat"], v["vmat"], v["Emat"], *work)
        time += cur
    return {"time": time, "dt": dt, **{k: real(st["t"][k], c) for k in FIELDS + ("pmat",)}}


# ---- what a pass cannot do without ----

def cell_updates(c):
    """Cell-updates of a pass; for domains that run to a time, by the interface states' typical dt."""
    if c["kind"] in ("batch", "serve"):
        total = 0.0
        for s in specs(c, 1):
            side = max(s.nx, s.ny)
            total += s.nx * s.ny * (c["cycles"] or max(1.0, c["t_end"] * side * 2.5 / 0.6))
        return total
    return float(c["nx"]) * c["ny"] * c["cycles"]


def work(c):
    # a cycle reads and writes rho, u, v, E once; two axis passes of about 190 operations a cell
    size = {64: 8, 32: 4, 0: 6}[c["precision"]]
    n = cell_updates(c)
    return {"bytes": 8 * size * n, "flops": 380 * n}


# ---- the step in plain 64-bit torch ----

class Sim:
    """The reference's time loop on the real cells of one domain with reflecting walls."""

    def __init__(self, c, nx, ny, fields):
        self.c, self.nx, self.ny = c, nx, ny
        self.f = dict(zip(FIELDS, (t.clone() for t in fields)))
        self.cycle, self.time, self.dt = 0, 0.0, 0.0

    @staticmethod
    def eos(rho, u, v, E):
        p = (1.4 - 1) * rho * (E - 0.5 * (u * u + v * v))
        return p, torch.sqrt(1.4 * p / rho)

    def limit(self, num, den):
        r = num / den
        if self.c["limiter"] == "Minmod":
            return r.clamp(0.0, 1.0)
        if self.c["limiter"] == "Superbee":
            return torch.maximum((2 * r).clamp(0.0, 1.0), r.clamp(0.0, 2.0))
        return torch.ones_like(r)

    def axis_pass(self, axis, dt):
        c = self.c
        n = (self.nx, self.ny)[axis]
        dx = 1.0 / n
        dim = 1 - axis
        H = 5

        def cut(t, lo, hi):      # positions lo .. hi - 1 of a field that starts at position t[1]
            return t[0].narrow(dim, lo - t[1], hi - lo)

        def pad(t, sign):
            lo, hi = t.narrow(dim, 0, H).flip(dim), t.narrow(dim, n - H, H).flip(dim)
            return torch.cat([sign * lo, t, sign * hi], dim), -H

        a, o = ("umat", "vmat") if axis == 0 else ("vmat", "umat")
        rho, ua, uo, E = pad(self.f["rho"], 1), pad(self.f[a], -1), pad(self.f[o], 1), pad(self.f["Emat"], 1)
        p, cs = self.eos(rho[0], ua[0], uo[0], E[0])
        self.p = cut((p, -H), 0, n)
        rc = rho[0] * cs
        lo, hi = -H + 1, n + H   # faces lo .. hi - 1, face i between cells i - 1 and i

        def left(t):
            return t.narrow(dim, 0, t.shape[dim] - 1)

        def right(t):
            return t.narrow(dim, 1, t.shape[dim] - 1)

        rcl, rcr, ul, ur, pl, pr = left(rc), right(rc), left(ua[0]), right(ua[0]), left(p), right(p)
        us = (rcl * ul + rcr * ur + (pl - pr)) / (rcl + rcr)
        ps = (rcr * pl + rcl * pr + rcl * rcr * (ul - ur)) / (rcl + rcr)
        if c["scheme"] == "GAD":
            au, bu, ap, bp = us - ul, ur - us, ps - pl, pr - ps

            def at(t, k):        # the value of the face k after this one, for faces lo + 1 .. hi - 2
                return t.narrow(dim, 1 + k, t.shape[dim] - 2)

            rum = self.limit(at(au, 1), at(au, 0) + 1e-6)
            rpm = self.limit(at(ap, 1), at(ap, 0) + 1e-6)
            rup = self.limit(at(bu, -1), at(bu, 0) + 1e-6)
            rpp = self.limit(at(bp, -1), at(bp, 0) + 1e-6)
            dm = rho[0] * dx
            Dm = (at(left(dm), 0) + at(right(dm), 0)) / 2
            theta = 0.5 * (1 - at(rcl + rcr, 0) / 2 * (dt / Dm))
            us, ps = (at(us, 0) + theta * (rup * at(bu, 0) - rum * at(au, 0)),
                      at(ps, 0) + theta * (rpp * at(bp, 0) - rpm * at(ap, 0)))
            lo, hi = lo + 1, hi - 1
        F, P = (us, lo), (ps, lo)
        # Lagrangian cells lo .. hi - 2
        j0, j1 = lo, hi - 1
        dm = cut(rho, j0, j1) * dx
        width = dx + dt * (cut(F, j0 + 1, j1 + 1) - cut(F, j0, j1))
        pu = ps * us
        lr = dm / width
        lua = cut(ua, j0, j1) + dt / dm * (cut(P, j0, j1) - cut(P, j0 + 1, j1 + 1))
        lE = cut(E, j0, j1) + dt / dm * (cut((pu, lo), j0, j1) - cut((pu, lo), j0 + 1, j1 + 1))
        luo = cut(uo, j0, j1)
        q = [(t, j0) for t in (lr, lr * lua, lr * luo, lr * lE)]
        w = (width, j0)
        disp = dt * cut(F, 0, n + 1)
        up = disp > 0
        adv = []
        if c["projection"] == "euler":
            for t in q:
                adv.append(disp * torch.where(up, cut(t, -1, n), cut(t, 0, n + 1)))
        else:
            def pick(t, k):      # cell k from the upwind cell of each face
                return torch.where(up, cut(t, k - 1, k + n), cut(t, k, k + n + 1))

            d = (dt * us, lo)
            Dx = torch.where(up, -(dx - cut(d, -1, n)), dx + cut(d, 1, n + 2))
            wl = pick(w, 0)
            rm, rp = 2 * wl / (wl + pick(w, -1)), 2 * wl / (wl + pick(w, 1))
            for t in q:
                u0 = pick(t, 0)
                dp, dmm = rp * (pick(t, 1) - u0), rm * (u0 - pick(t, -1))
                sgn = torch.copysign(torch.ones_like(dp), dp)
                slope = sgn * torch.minimum(sgn * dp, sgn * dmm).clamp(min=0.0)
                adv.append(disp * (u0 - slope * (Dx / (2 * wl))))
        dX = cut(w, 0, n)
        new = [(dX * cut(t, 0, n) - (right(f) - left(f))) / dx for t, f in zip(q, adv)]
        self.f["rho"], self.f[a], self.f[o], self.f["Emat"] = new[0], new[1] / new[0], new[2] / new[0], new[3] / new[0]
        self.c_last = cut((cs, -H), 0, n)

    def run(self, cycles, t_end):
        f = self.f
        cs = self.eos(f["rho"], f["umat"], f["vmat"], f["Emat"])[1]
        while self.cycle < cycles and self.time < t_end:
            sx = torch.maximum((f["umat"] + cs).abs(), (f["umat"] - cs).abs()).max().item()
            sy = torch.maximum((f["vmat"] + cs).abs(), (f["vmat"] - cs).abs()).max().item()
            new = 0.6 * min(1.0 / self.nx / sx, 1.0 / self.ny / sy)
            if self.dt:
                new = min(new, 1.05 * self.dt)
            cur = self.dt or new
            self.dt = new
            first = 1 if self.cycle % 2 == 0 else 0
            order = {"Sequential": ((0, 1.0), (1, 1.0)), "SequentialSym": ((first, 1.0), (1 - first, 1.0)),
                     "Strang": ((first, 0.5), (1 - first, 1.0), (first, 0.5))}[self.c["splitting"]]
            for axis, factor in order:
                self.axis_pass(axis, cur * factor)
            cs = self.c_last
            self.time += cur
            self.cycle += 1
        return self


def centres(n):
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    return i / float(n) + 1.0 / (2 * n)


def interface(c, s):
    x, y = centres(s.nx)[None, :] - 0.5, centres(s.ny)[:, None] - 0.5
    if s.kind == "planar":
        high = x * float(np.cos(s.angle)) + y * float(np.sin(s.angle)) <= s.pos - 0.5
    else:
        high = x * x + y * y <= (s.pos / 2) ** 2
    h = high.double()
    rho = h * s.rho_l + (1 - h) * s.rho_r
    E = h * (s.p_l / ((1.4 - 1) * s.rho_l)) + (1 - h) * (s.p_r / ((1.4 - 1) * s.rho_r))
    z = torch.zeros_like(rho)
    return rho, z, z, E


def exact(c, seed):
    if c["kind"] in ("batch", "serve"):
        out, times, counts = [], [], []
        for s in specs(c, seed):
            if c["kind"] == "serve" and s.precision == 32:
                continue
            m = Sim(c, s.nx, s.ny, interface(c, s)).run(c["cycles"] or 1_000_000, c["t_end"] or 1e9)
            out.append(m.f["rho"].reshape(-1).cpu().numpy())
            times.append(m.time)
            counts.append(m.cycle)
        if c["kind"] == "serve":   # an FP32 request may end a cycle apart from its FP64 solve
            got = {"rho64": np.concatenate(out), "time64": np.array(times)} if out else {}
            if any(s.precision == 32 for s in specs(c, seed)):
                got.update(rho32=None, time32=None)
            return got
        return {"rho": np.concatenate(out), "time": np.array(times), "cycles": np.array(counts)}
    nx, ny = c["nx"], c["ny"]
    if c["state"] == "flow":
        fields = [real(f, c).contiguous() for f in flow_fields(c, seed).values()]
    else:
        if nx * ny * c["cycles"] > 4e9:
            return None
        x, y = centres(nx)[None, :] - 0.5, centres(ny)[:, None] - 0.5
        high = x * x + y * y <= circ_radius2(seed)
        z = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
        fields = [torch.where(high, 1.0, 0.125).double(), z, z, torch.where(high, 2.5, 2.0).double()]
    m = Sim(c, nx, ny, fields).run(c["cycles"], 1e9)
    out = {k: m.f[k] for k in FIELDS}
    out.update(pmat=m.p, time=m.time, dt=m.dt)
    if c["kind"] != "stages":
        out["cycles"] = m.cycle
    return out
