"""What a user of this framework has it do, as measurable cases.

Five kinds of work, each through the public entry points a program calls:

  engine     a forecast in the member engine: the initial states go up as one
             state image, the members take some large steps together, the
             states come back (EngineRun, Engine.upload_image_async / step /
             download_image_async: one output interval of HostPipeline);
  plain      the same large steps of one run through the per-operation entry
             points (ResidentRun), its substep count re-derived every step;
  acoustic   the batched acoustic loop on device arrays
             (Context.acoustic_batched), or dispatched on host arrays as the
             reference's program does (CudaComputeBackend);
  transport  the WENO5 scalar transport (Context.scalar_transport);
  moist      the Kessler tendencies and the EOS projection;
  sgs        the Smagorinsky closure (Context.smagorinsky_fused).

`exact` gives the same results from plain torch in 64 bits.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from nimbus_b200 import cuda, initial
from nimbus_b200.run import POSITIVE, PROGNOSTIC, SCALARS, EngineRun, ResidentRun
from nimbus_b200.sgs import SgsConfig

# Boundary sets (W, E, S, N, bottom, top): the open supercell box of every
# workload here, a doubly periodic channel, and closed walls.
BOUNDARIES = {
    "open": (1, 1, 1, 1, 1, 0),
    "periodic": (0, 0, 0, 0, 0, 2),
    "walls": (2, 3, 4, 3, 1, 1),
}
BLOCK_FIELDS = 7  # members whose fields are returned one by one; more come as one block a member


def listed():
    return [
        # The smallest served run (32x32x40): a minute of it between two output frames; latency and launches.
        dict(name="served_run_32", kind="engine", fp32=True, members=1, nx=32, ny=32, nz=40, dx=500.0, dt=3.0,
             steps=20, bc="open"),
        # A few requests of the serving stream in flight at once: ragged sizes, a frame every 12 s.
        dict(name="serving_mix", kind="engine", fp32=True, members=6, nx=0, ny=32, nz=256, dx=500.0, dt=3.0, steps=4,
             bc="open"),
        # A ragged forecast ensemble (48..192 squared, 40..64 levels), the framework's main load.
        dict(name="ensemble_24", kind="engine", fp32=True, members=24, nx=0, ny=48, nz=192, dx=500.0, dt=3.0,
             steps=10, bc="open"),
        # One storm at 250 m (256x256x80).
        dict(name="supercell_250m", kind="engine", fp32=True, members=1, nx=256, ny=256, nz=80, dx=250.0, dt=1.5,
             steps=10, bc="open"),
        # An ensemble in the arithmetic that equals the CPU solver's bit for bit, odd sizes among its members.
        dict(name="ensemble_7_reference", kind="engine", fp32=False, members=7, nx=0, ny=48, nz=192, dx=500.0, dt=3.0,
             steps=4, bc="open"),
        # The 1 km supercell (64x64x40, dt 6 s) operation by operation, reference precision: what a host program
        # that keeps its own loop pays.
        dict(name="plain_1km_reference", kind="plain", fp32=False, nx=64, ny=64, nz=40, dx=1000.0, dt=6.0, steps=4,
             bc="open"),
        # The acoustic loop of the largest single run (100 m storm, 512x512x128).
        dict(name="acoustic_100m", kind="acoustic", host=False, fp32=True, nx=512, ny=512, nz=128, dx=100.0, dt=0.6,
             substeps=10, bc="open"),
        # The same loop in reference precision on an odd, doubly periodic grid with an open top.
        dict(name="acoustic_odd_reference", kind="acoustic", host=False, fp32=False, nx=131, ny=97, nz=53, dx=500.0,
             dt=3.0, substeps=7, bc="periodic"),
        # The loop dispatched on host arrays, the reference program's contract (95x95x50, the ensemble's median run).
        dict(name="acoustic_host_dispatch", kind="acoustic", host=True, fp32=False, nx=95, ny=95, nz=50, dx=500.0,
             dt=3.0, substeps=7, bc="open"),
        # Transport of theta and three waters, reference precision, 250 m storm.
        dict(name="transport_reference", kind="transport", fp32=False, nx=256, ny=256, nz=80, dx=250.0, dt=1.5,
             scalars=4, bc="open"),
        # Warm rain and the pressure projection on their own, reference precision.
        dict(name="moist_reference", kind="moist", fp32=False, nx=193, ny=161, nz=61, dx=500.0, dt=3.0, bc="open"),
        # The turbulence closure of a 250 m run, reference precision.
        dict(name="closure_reference", kind="sgs", fp32=False, nx=320, ny=320, nz=64, dx=250.0, dt=1.5, bc="open"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["engine", "engine", "engine", "plain", "acoustic", "acoustic", "transport", "moist", "sgs"])
    case = dict(kind=kind, fp32=rng.random() < 0.6, dx=500.0, dt=3.0, bc="open")
    if kind == "engine":
        if rng.random() < 0.5:  # one run
            n = _log(rng, 32, 288)
            case.update(members=1, nx=n, ny=max(8, n + rng.randint(-9, 9)), nz=rng.randint(40, 84),
                        steps=rng.randint(2, 12))
        else:  # ragged members between two sizes
            lo = _log(rng, 32, 96)
            case.update(members=rng.randint(2, 24), nx=0, ny=lo, nz=min(192, 2 * lo + rng.randint(0, 9)),
                        steps=rng.randint(2, 8))
    else:
        n = _log(rng, 24, 320)
        case.update(nx=n, ny=max(8, n + rng.randint(-9, 9)), nz=rng.randint(24, 96))
        case["bc"] = rng.choice(["open", "open", "periodic", "walls"]) if kind == "acoustic" else "open"
        if kind == "plain":
            case.update(steps=rng.randint(1, 4))
        elif kind == "acoustic":
            case.update(host=n < 100 and rng.random() < 0.25)
            case["substeps"] = _substeps(case, _run_case(case, _grids(case)[0])) + rng.randint(0, 2)
            case["fp32"] = case["fp32"] and not case["host"]
        elif kind == "transport":
            case.update(scalars=rng.choice([1, 3, 4, 4, 5]))
    return case


# ---- sizes and inputs ------------------------------------------------------


def _grids(case):
    """The member grids of a case; ragged ones between ny and nz squared, 40 to 64 levels."""
    if case["nx"]:
        return [(case["nx"], case["ny"], case["nz"])]
    lo, hi = case["ny"], case["nz"]
    rng = random.Random(1000 * lo + hi + case["members"])
    out = []
    for _ in range(case["members"]):
        u = rng.random()
        n = int(round(lo * (hi / lo) ** u))
        out.append((n, n, int(round(40 * 1.6 ** u))))
    return out


def _run_case(case, grid):
    nx, ny, nz = grid
    dz = 20000.0 / nz
    return initial.Case(nx, ny, nz, case["dx"], case["dx"], dz, case["dt"], bc=BOUNDARIES[case["bc"]])


def _base(rc):
    b = initial.sounding(rc)
    return {k: np.ascontiguousarray(b[k], np.float64) for k in ("rho0", "p0", "qv0", "u0", "v0", "theta0", "z")}


def _storm(rc, base, seed):
    """A developing storm on the sounding, float32 on the GPU: smooth winds around the hodograph, a warm moist
    updraft holding cloud and rain, small-scale theta noise near the ground, pressure near balance."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = dict(device="cuda", dtype=torch.float64)
    nx, ny, nz = rc.shape
    x = torch.arange(nx, **d).view(-1, 1, 1) / nx
    y = torch.arange(ny, **d).view(1, -1, 1) / ny
    z = torch.arange(nz, **d).view(1, 1, -1) / nz
    col = {k: torch.from_numpy(v).to("cuda").view(1, 1, -1) for k, v in base.items()}
    cx, cy, ph = (torch.rand(8, generator=g, **d) for _ in range(3))

    def waves(m):
        a = torch.zeros(1, 1, 1, **d)
        for q in range(2):
            a = a + torch.sin(2 * math.pi * (((q + 1) * x) + cx[m + q])) * torch.cos(2 * math.pi * (y + cy[m + q])) \
                * torch.sin(math.pi * (z + 0.2 * ph[m + q]))
        return a

    r = torch.sqrt(((x - 0.3 - 0.4 * cx[7]) / 0.22) ** 2 + ((y - 0.3 - 0.4 * cy[7]) / 0.22) ** 2
                   + ((z - 0.25) / 0.2) ** 2)
    core = torch.where(r < 1, torch.cos(0.5 * math.pi * r.clamp(max=1.0)) ** 2, torch.zeros_like(r))
    noise = torch.rand(rc.shape, generator=g, device="cuda") - 0.5
    near = (z < 0.08).double()
    theta = col["theta0"] + 3.0 * core + 0.4 * near * noise + 0.3 * waves(0)
    p = col["p0"] * (1 + 2e-5 * waves(2))
    rho = (p / initial.P00) ** (1.0 / initial.GAMMA) * initial.P00 / (initial.R_D * theta)
    rim = (1 - (z * (1 - z) * 4 - 1).abs())
    st = dict(u=col["u0"] + 2.0 * waves(1), v=col["v0"] + 2.0 * waves(3),
              w=(8.0 * core + 0.5 * waves(4)) * rim, rho=rho, p=p, theta=theta,
              qv=col["qv0"] * (1 + 0.25 * core + 0.1 * noise * near),
              qc=2.5e-3 * (core - 0.2).clamp(min=0), qr=4e-3 * (core - 0.35).clamp(min=0))
    return {k: v.expand(rc.shape).to(torch.float32).contiguous() for k, v in st.items()}


def _precision(case):
    return cuda.PRECISION_FP32 if case["fp32"] else cuda.PRECISION_REFERENCE


def _grid_of(rc):
    return (rc.dx, rc.dy, rc.dz)


def _loop_inputs(case, rc, base, seed):
    st = _storm(rc, base, seed)
    return {k: st[k] for k in ("u", "v", "w", "rho", "p", "theta")}


def _transport_inputs(case, rc, base, seed):
    """Scalars, densities and retained fluxes as a large step leaves them."""
    st = _storm(rc, base, seed)
    up = {a: torch.cat([st["rho"].narrow(a, 1, rc.shape[a] - 1), st["rho"].narrow(a, rc.shape[a] - 1, 1)], a)
          for a in range(3)}
    mf = [0.5 * (st["rho"] + up[a]) * st[k] for a, k in enumerate(("u", "v", "w"))]
    mf[2][:, :, -1] = 0
    names = ["theta", "qv", "qc", "qr", "theta"][:case["scalars"]]
    return dict(q=[st[k].clone() for k in names], pd=[0 if k == "theta" else 1 for k in names],
                rho_begin=st["rho"], rho_end=(st["rho"] * (1 + 1e-4 * torch.sin(st["u"]))).contiguous(), mf=mf)


# ---- prepare and run -------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    ctx = cuda.Context()
    ctx.set_precision(_precision(case))
    state = dict(kind=kind, ctx=ctx, case=case)
    if kind == "engine":
        grids = _grids(case)
        floats = [9 * nx * ny * nz for nx, ny, nz in grids]
        first = torch.empty(sum(floats), dtype=torch.float32, pin_memory=True)
        run_ = EngineRun(ctx, _precision(case))
        at = 0
        for m, grid in enumerate(grids):
            rc = _run_case(case, grid)
            base = _base(rc)
            st = _storm(rc, base, 7919 * seed + m)
            block = first[at:at + floats[m]].view(9, *grid)
            for f, k in enumerate(PROGNOSTIC):
                block[f].copy_(st[k])
            run_.admit(rc, {k: block[f].numpy() for f, k in enumerate(PROGNOSTIC)}, base)
            at += floats[m]
        out = torch.empty_like(first, pin_memory=True)
        views, at = [], 0
        for m, grid in enumerate(grids):
            block = out[at:at + floats[m]].view(9, *grid)
            views.append({k: block[f] for f, k in enumerate(PROGNOSTIC)} if len(grids) <= BLOCK_FIELDS else block)
            at += floats[m]
        state.update(run=run_, first=first.view(torch.uint8).numpy(), out=out.view(torch.uint8).numpy(), views=views)
        return state
    rc = _run_case(case, _grids(case)[0])
    base = _base(rc)
    state["prof"] = {k: torch.from_numpy(base[k]).to("cuda") for k in ("rho0", "p0")}
    if kind == "plain":
        st = _storm(rc, base, seed)
        state["first"] = st
        state["run"] = ResidentRun(ctx, rc, {k: v.cpu().numpy() for k, v in st.items()}, base, autotune=False,
                                   precision=_precision(case))
    elif kind == "acoustic":
        st = _loop_inputs(case, rc, base, seed)
        n = case["substeps"]
        if case["host"]:
            backend = cuda.CudaComputeBackend()
            if not backend.initialize():
                raise RuntimeError(backend.last_error)
            host = {k: v.cpu().numpy() for k, v in st.items()}
            mf = [np.zeros(rc.shape, np.float32) for _ in range(3)]
            wave = np.zeros(2 * (rc.nx + rc.ny) * rc.nz, np.float32)
            state.update(backend=backend, host=host, mf=mf, wave=wave, rc=rc, base=base)
        else:
            mf = [torch.zeros_like(st["u"]) for _ in range(3)]
            wave = torch.zeros(2 * (rc.nx + rc.ny) * rc.nz, device="cuda")
            begin = torch.zeros_like(st["u"])
            args = cuda.batched_args(st, state["prof"]["rho0"], state["prof"]["p0"], rc.dt / n, n, _grid_of(rc), rc.bc,
                                     *mf, 1.0 / n, None, wave, begin, memory=cuda.MEMORY_DEVICE)
            state.update(args=args, st=st, mf=mf, begin=begin,
                         stream=torch.cuda.ExternalStream(ctx.stream, device=st["u"].device))
    elif kind == "transport":
        t = _transport_inputs(case, rc, base, seed)
        outs = [torch.empty_like(q) for q in t["q"]]
        state.update(args=cuda.transport_args(t["q"], outs, t["pd"], t["rho_end"], t["rho_begin"], *t["mf"], rc.dt,
                                              _grid_of(rc), memory=cuda.MEMORY_DEVICE), outs=outs)
    elif kind == "moist":
        st = _storm(rc, base, seed)
        outs = tuple(torch.empty_like(st["u"]) for _ in range(4))
        state.update(kessler=cuda.kessler_args(st, rc.dz, rc.dt, outputs=outs, memory=cuda.MEMORY_DEVICE),
                     eos=cuda.eos_args(st["p"], st["rho"], st["theta"], st["qv"], st["qc"], st["qr"],
                                       memory=cuda.MEMORY_DEVICE, p0=state["prof"]["p0"]), outs=outs, p=st["p"])
    else:
        st = _storm(rc, base, seed)
        args = cuda.smagorinsky_args(st, np.full(rc.nz, rc.dz), _grid_of(rc), SgsConfig.from_bc(rc.bc),
                                     memory=cuda.MEMORY_DEVICE)
        state["args"] = args
    return state


def run(state):
    kind, ctx, case = state["kind"], state["ctx"], state["case"]
    if kind == "engine":
        engine = state["run"].engine
        engine.upload_image_async(state["first"])
        state["run"].step(case["steps"])
        engine.download_image_async(state["out"])
        return state["views"]
    if kind == "plain":
        r = state["run"]
        with torch.cuda.stream(r.torch_stream):
            for k, v in state["first"].items():
                r.fields[k].copy_(v)
        for _ in range(case["steps"]):
            r.step()
        return r.fields
    if kind == "acoustic" and case["host"]:
        st, rc, base, n = state["host"], state["rc"], state["base"], case["substeps"]
        for m in state["mf"]:
            m.fill(0.0)
        if not state["backend"].dispatch_acoustic_substeps_batched_cartesian_cgrid(
                st, base["rho0"], base["p0"], rc.dt / n, n, _grid_of(rc), rc.bc, *state["mf"], 1.0 / n, None,
                state["wave"]):
            raise RuntimeError(state["backend"].last_error)
        return dict({k: st[k] for k in ("u", "v", "w", "rho", "p")}, mf=state["mf"])
    if kind == "acoustic":
        with torch.cuda.stream(state["stream"]):
            for m in state["mf"]:
                m.zero_()
        ctx.check(ctx.acoustic_batched(state["args"]))
        return dict({k: state["st"][k] for k in ("u", "v", "w", "rho", "p")}, mf=state["mf"], begin=state["begin"])
    if kind == "transport":
        ctx.check(ctx.scalar_transport(state["args"]))
        return state["outs"]
    if kind == "moist":
        ctx.check(ctx.kessler_tendencies(state["kessler"]))
        ctx.check(ctx.eos_projection(state["eos"]))
        return dict(rates=state["outs"], p=state["p"])
    ctx.check(ctx.smagorinsky_fused(state["args"]))
    return state["args"].outputs


# ---- work ------------------------------------------------------------------

# Per cell, each input read once and each output written once: an acoustic
# substep reads rho, theta, u, v, w and the three retained fluxes and writes
# rho, p, u, v, w and the fluxes (with u, v, w read again after the pressure);
# the rest of a large step is the Heun slow step (112), transport (20 + 8 a
# scalar), Kessler (40) and the projection (12).
_SUBSTEP_B, _SUBSTEP_F = 68, 75
_STEP_B, _STEP_F = 216, 1900


def _substeps(case, rc):
    b = initial.sounding(rc)
    c = math.sqrt(float(np.max(initial.GAMMA * b["p0"] / b["rho0"])))
    return initial.resolve_substep_count(rc.dt, c, rc.dx, rc.dy, rc.dz)


def work(case):
    total_b = total_f = 0.0
    for grid in _grids(case):
        rc = _run_case(case, grid)
        kind = case["kind"]
        if kind in ("engine", "plain"):
            n = _substeps(case, rc)
            b, f = case["steps"] * (n * _SUBSTEP_B + _STEP_B) + 72, case["steps"] * (n * _SUBSTEP_F + _STEP_F)
        elif kind == "acoustic":
            b, f = case["substeps"] * _SUBSTEP_B, case["substeps"] * _SUBSTEP_F
        elif kind == "transport":
            b, f = 20 + 8 * case["scalars"], 300 * case["scalars"]
        elif kind == "moist":
            b, f = 24 + 16 + 12, 300
        else:
            b, f = 24 + 32, 450
        total_b += b * rc.cells
        total_f += f * rc.cells
    return {"bytes": total_b, "flops": total_f}


# ---- the same in 64 bits ---------------------------------------------------

_RD, _CP, _P00, _GAMMA = 287.0, 1004.0, 100000.0, 1004.0 / (1004.0 - 287.0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "engine":
        views = []
        grids = _grids(case)
        for m, grid in enumerate(grids):
            rc = _run_case(case, grid)
            base = _base(rc)
            s = _steps64(_double(_storm(rc, base, 7919 * seed + m)), rc, _columns(base), case["steps"])
            views.append(s if len(grids) <= BLOCK_FIELDS else torch.stack([s[k] for k in PROGNOSTIC]))
        return views
    rc = _run_case(case, _grids(case)[0])
    base = _base(rc)
    col = _columns(base)
    if kind == "plain":
        return _steps64(_double(_storm(rc, base, seed)), rc, col, case["steps"])
    if kind == "acoustic":
        s = _double(_loop_inputs(case, rc, base, seed))
        begin = s["rho"].clone()
        mf = _loop64(s, rc, col, case["substeps"])
        out = dict({k: s[k] for k in ("u", "v", "w", "rho", "p")}, mf=mf)
        return out if case["host"] else dict(out, begin=begin)
    if kind == "transport":
        t = _transport_inputs(case, rc, base, seed)
        return [_transport64(q.double(), pd, t["rho_begin"].double(), t["rho_end"].double(),
                             [m.double() for m in t["mf"]], rc) for q, pd in zip(t["q"], t["pd"])]
    s = _double(_storm(rc, base, seed))
    if kind == "moist":
        return dict(rates=_kessler64(s, rc), p=_eos64(s["rho"], s["theta"]))
    return _closure64(s, rc)


def _double(st):
    return {k: v.double() for k, v in st.items()}


def _columns(base):
    return {k: torch.from_numpy(v).to("cuda").view(1, 1, -1) for k, v in base.items()}


def _eos64(rho, theta):
    return (_P00 * (rho * _RD * theta / _P00) ** _GAMMA).clamp(1000.0, 200000.0)


def _closure(s, rc, hist, dt_rad):
    """The boundary closure W, E, S, N, top and bottom, in place; hist holds the KW78 face memory."""
    def radiate(prev, sign, gradient, inv):
        phase = prev + sign * 30.0
        new = prev - dt_rad * phase * gradient * inv
        return torch.where((phase >= 0) if sign < 0 else (phase <= 0), prev, new)

    for ax, n, lo_bc, hi_bc, inv in ((0, rc.nx, rc.bc[0], rc.bc[1], 1 / rc.dx), (1, rc.ny, rc.bc[2], rc.bc[3], 1 / rc.dy)):
        normal, cross = ("u", "v") if ax == 0 else ("v", "u")
        at = lambda f, i: s[f].select(ax, i)  # noqa: E731
        if lo_bc == 0:
            for f in ("u", "v", "w", "rho", "p"):
                at(f, 0).copy_(at(f, n - 2))
        else:
            if lo_bc == 1:
                if dt_rad > 0:
                    prev = hist[2 * ax]
                    hist[2 * ax] = radiate(prev, -1, at(normal, 1) - prev, inv)
                    at(normal, 0).copy_(hist[2 * ax])
            elif lo_bc == 4:
                at(normal, 0).copy_(at(normal, 1))
            else:
                at(normal, 0).zero_()
            for f in (cross, "w"):
                at(f, 0).zero_() if lo_bc == 2 else at(f, 0).copy_(at(f, 1))
            for f in ("rho", "p"):
                at(f, 0).copy_(at(f, 1))
        if hi_bc == 0:
            for f in ("u", "v", "w", "rho", "p"):
                at(f, n - 1).copy_(at(f, 1))
        else:
            if hi_bc in (2, 3):
                at(normal, n - 2).zero_()
            if hi_bc == 1 and dt_rad > 0:
                prev = hist[2 * ax + 1]
                hist[2 * ax + 1] = radiate(prev, 1, prev - at(normal, n - 3), inv)
                at(normal, n - 2).copy_(hist[2 * ax + 1])
            elif hi_bc == 4:
                at(normal, n - 2).copy_(at(normal, n - 3))
            at(normal, n - 1).copy_(at(normal, n - 2)) if hi_bc in (1, 4) else at(normal, n - 1).zero_()
            for f in (cross, "w"):
                at(f, n - 1).zero_() if hi_bc == 2 else at(f, n - 1).copy_(at(f, n - 2))
            for f in ("rho", "p"):
                at(f, n - 1).copy_(at(f, n - 2))
    if rc.bc[4] == 0:
        s["u"][:, :, 0] = 0
        s["v"][:, :, 0] = 0
    s["w"][:, :, -1] = s["w"][:, :, -2] if rc.bc[5] == 2 else 0
    s["u"][:, :, -1] = s["u"][:, :, -2]
    s["v"][:, :, -1] = s["v"][:, :, -2]


def _seed(s, rc):
    return [s["u"][0].clone(), s["u"][rc.nx - 2].clone(), s["v"][:, 0].clone(), s["v"][:, rc.ny - 2].clone()]


def _loop64(s, rc, col, n):
    """n acoustic substeps in place; the retained mass fluxes."""
    dt = rc.dt / n
    hist = _seed(s, rc)
    mf = [torch.zeros_like(s["u"]) for _ in range(3)]
    open_top = rc.bc[5] == 2
    ij = (slice(1, -1), slice(1, -1))
    for _ in range(n):
        rho, u, v, w = s["rho"], s["u"], s["v"], s["w"]
        fx, fy, fz = torch.zeros_like(rho), torch.zeros_like(rho), torch.zeros_like(rho)
        fx[:-1] = 0.5 * (rho[:-1] + rho[1:]) * u[:-1]
        fy[:, :-1] = 0.5 * (rho[:, :-1] + rho[:, 1:]) * v[:, :-1]
        fz[:, :, :-1] = 0.5 * (rho[:, :, :-1] + rho[:, :, 1:]) * w[:, :, :-1]
        fz[:, :, -1] = rho[:, :, -1] * w[:, :, -1]
        for q, f in enumerate((fx, fy, fz)):
            mf[q] += f / n
        if not open_top:
            mf[2][:, :, -1] = 0
        div = torch.zeros_like(rho)
        div[1:-1] = (fx[1:-1] - fx[:-2]) / rc.dx
        div[:, 1:-1] += (fy[:, 1:-1] - fy[:, :-2]) / rc.dy
        div += torch.cat([fz[:, :, :1], fz[:, :, 1:] - fz[:, :, :-1]], 2) / rc.dz
        new = rho.clone()
        new[ij] -= dt * div[ij]
        rho = s["rho"] = new.clamp(0.05, 2.0)
        p = s["p"] = _eos64(rho, s["theta"])
        k = (*ij, slice(0, -1))
        dp0 = (col["p0"][:, :, 1:] - col["p0"][:, :, :-1]) / rc.dz
        pc, rc_ = p[k], rho[k]
        u[k] -= dt * (p[2:, 1:-1, :-1] - pc) / rc.dx / (0.5 * (rc_ + rho[2:, 1:-1, :-1]))
        v[k] -= dt * (p[1:-1, 2:, :-1] - pc) / rc.dy / (0.5 * (rc_ + rho[1:-1, 2:, :-1]))
        w[k] -= dt * ((p[1:-1, 1:-1, 1:] - pc) / rc.dz - dp0) / (0.5 * (rc_ + rho[1:-1, 1:-1, 1:]))
        u.clamp_(-180.0, 180.0)
        v.clamp_(-180.0, 180.0)
        w.clamp_(-120.0, 120.0)
        _closure(s, rc, hist, dt)
    return mf


def _upwind(f, ax, n, a, d):
    """Upwind derivative of f along ax with wind a: fifth, third or first order by distance from the edge."""
    sh = lambda o: torch.roll(f, -o, ax)  # noqa: E731
    pos = a >= 0
    idx = torch.arange(n, device=f.device)
    half = torch.minimum(idx, n - 1 - idx).view([-1 if q == ax else 1 for q in range(3)])
    m1, p1, m2, p2, m3, p3 = sh(-1), sh(1), sh(-2), sh(2), sh(-3), sh(3)
    d5 = torch.where(pos, -2 * m3 + 15 * m2 - 60 * m1 + 20 * f + 30 * p1 - 3 * p2,
                     2 * p3 - 15 * p2 + 60 * p1 - 20 * f - 30 * m1 + 3 * m2) / 60
    d3 = torch.where(pos, 2 * p1 + 3 * f - 6 * m1 + m2, -p2 + 6 * p1 - 3 * f - 2 * m1) / 6
    d1 = torch.where(pos, f - m1, p1 - f)
    return torch.where(half >= 3, d5, torch.where(half == 2, d3, torch.where(half == 1, d1, torch.zeros_like(f)))) / d


def _slow64(s, rc, col):
    """The slow tendencies of u, v, w and p."""
    u, v, w, p, rho = (s[k] for k in ("u", "v", "w", "p", "rho"))
    r = lambda f, i, j, k: torch.roll(f, (-i, -j, -k), (0, 1, 2))  # noqa: E731
    below = r(w, 0, 0, -1)
    uy_u = 0.25 * (r(v, 0, -1, 0) + v + r(v, 1, -1, 0) + r(v, 1, 0, 0))
    ux_v = 0.25 * (r(u, -1, 0, 0) + u + r(u, -1, 1, 0) + r(u, 0, 1, 0))
    wx = 0.25 * (below + w + r(below, 1, 0, 0) + r(w, 1, 0, 0))
    wy = 0.25 * (below + w + r(below, 0, 1, 0) + r(w, 0, 1, 0))
    wx[:, :, 0] = 0.25 * (w + r(w, 1, 0, 0))[:, :, 0]
    wy[:, :, 0] = 0.25 * (w + r(w, 0, 1, 0))[:, :, 0]
    ux_w = 0.25 * (r(u, -1, 0, 0) + u + r(u, -1, 0, 1) + r(u, 0, 0, 1))
    uy_w = 0.25 * (r(v, 0, -1, 0) + v + r(v, 0, -1, 1) + r(v, 0, 0, 1))
    out = []
    for f, ax, ay, az in ((u, u, uy_u, wx), (v, ux_v, v, wy), (w, ux_w, uy_w, w)):
        dz = _upwind(f, 2, rc.nz, az, rc.dz)
        up = (f[:, :, 1] - f[:, :, 0]) / rc.dz
        own = f[:, :, 0] / rc.dz if f is w else torch.zeros_like(up)
        dz[:, :, 0] = torch.where(az[:, :, 0] >= 0, own, up)
        out.append(-ax * _upwind(f, 0, rc.nx, ax, rc.dx) - ay * _upwind(f, 1, rc.ny, ay, rc.dy) - az * dz)
    face = lambda f: 0.5 * (f + r(f, 0, 0, 1))  # noqa: E731
    rf = face(rho)
    out[2] = out[2] - 9.81 * (rf - face(col["rho0"])) / rf + 9.81 * 0.608 * (face(s["qv"]) - face(col["qv0"])) \
        - 9.81 * face(s["qc"] + s["qr"])
    grad = lambda ax, d: (torch.roll(p, -1, ax) - torch.roll(p, 1, ax)) / (2 * d)  # noqa: E731
    dp = -0.5 * (u + r(u, -1, 0, 0)) * grad(0, rc.dx) - 0.5 * (v + r(v, 0, -1, 0)) * grad(1, rc.dy) \
        - 0.5 * (w + below) * grad(2, rc.dz)
    dp[:, :, 0] = 0
    res = []
    for t in (*out, dp):
        z = torch.zeros_like(t)
        z[1:-1, 1:-1, :-1] = t[1:-1, 1:-1, :-1]
        res.append(z)
    return res


def _weno64(a, b, c, d, e):
    p0, p1, p2 = a / 3 - 7 * b / 6 + 11 * c / 6, -b / 6 + 5 * c / 6 + d / 3, c / 3 + 5 * d / 6 - e / 6
    b0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    big = torch.stack([t * t for t in (a, b, c, d, e)]).amax(0)
    eps = 1e-6 * big + 1e-40
    w0, w1, w2 = 0.1 / (eps + b0) ** 2, 0.6 / (eps + b1) ** 2, 0.3 / (eps + b2) ** 2
    # A stencil of zeros would be 0 / 0: its face is the donor value.
    total = w0 + w1 + w2
    face = (w0 * p0 + w1 * p1 + w2 * p2) / total
    return torch.where(torch.isfinite(face), face, c)


def _faces64(q, ax, m):
    """Flux through the upper face of each cell along ax (zero at the last): WENO5 where its stencil fits, else the
    MC-limited slope."""
    n = q.shape[ax]
    sh = lambda o: torch.roll(q, -o, ax)  # noqa: E731
    idx = torch.arange(n, device=q.device).view([-1 if x == ax else 1 for x in range(3)])

    def mc(l, c, h):
        a, b, g = 0.5 * (h - l), 2 * (h - c), 2 * (c - l)
        lo = torch.minimum(a, torch.minimum(b, g))
        hi = torch.maximum(a, torch.maximum(b, g))
        return torch.where(lo > 0, lo, torch.where(hi < 0, hi, torch.zeros_like(a)))

    zero = torch.zeros_like(q)
    up = torch.where((idx >= 2) & (idx + 2 <= n - 1), _weno64(sh(-2), sh(-1), q, sh(1), sh(2)),
                     q + 0.5 * torch.where(idx >= 1, mc(sh(-1), q, sh(1)), zero))
    dn = torch.where((idx >= 1) & (idx + 3 <= n - 1), _weno64(sh(3), sh(2), sh(1), q, sh(-1)),
                     sh(1) - 0.5 * torch.where(idx + 1 <= n - 2, mc(q, sh(1), sh(2)), zero))
    return torch.where(idx <= n - 2, m * torch.where(m >= 0, up, dn), zero)


def _transport64(q, pd, rho_b, rho_e, mf, rc):
    f = [_faces64(q, ax, mf[ax]) for ax in range(3)]
    if rc.bc[5] == 2:
        f[2][:, :, -1] = mf[2][:, :, -1] * q[:, :, -1]
    inv = (1 / rc.dx, 1 / rc.dy, 1 / rc.dz)

    def lower(t, ax):
        t = torch.roll(t, 1, ax)
        t.select(ax, 0).zero_()
        return t

    if pd:
        out = sum((f[a].clamp(min=0) - lower(f[a], a).clamp(max=0)) * inv[a] for a in range(3))
        ratio = rho_b * q.clamp(min=0) / rc.dt / out
        r = torch.where((out > 0) & (ratio < 1), ratio * (1 - 32 * 2.0 ** -23), torch.ones_like(q))
        f = [f[a] * torch.where(f[a] > 0, r, torch.roll(r, -1, a)) for a in range(3)]
    div = sum((f[a] - lower(f[a], a)) * inv[a] for a in range(3))
    new = q.clone()
    ij = (slice(1, -1), slice(1, -1))
    new[ij] = ((rho_b * q - rc.dt * div) / rho_e.clamp(min=0.05))[ij]
    return new


def _qvs64(T, p):
    tc = T.clamp(150.0, 400.0) - 273.15
    e = 611.21 * torch.exp((18.678 - tc / 234.5) * tc / (257.14 + tc))
    ps = p.clamp(100.0, 200000.0)
    return (0.62198 * e / (ps - e).clamp(min=1.0)).clamp(0.0, 0.2)


def _slope64(T, sat, p):
    tc = T - 273.15
    den, num = 257.14 + tc, (18.678 - tc / 234.5) * tc
    lps = ((18.678 - 2 * tc / 234.5) * den - num) / den ** 2
    vapour = sat * p / (0.62198 + sat)
    g = sat * p / (p - vapour).clamp(min=1.0) * lps
    return torch.where((sat > 0) & (sat < 0.2), g, torch.zeros_like(g))


def _adjust64(T, p, qv, qc):
    """Saturation adjustment: vapour condensed (positive) or cloud evaporated so that qv is saturated."""
    L = 2.5e6 / 1004.0
    qvs = _qvs64(T, p)
    cond = qv > qvs
    hi = torch.where(cond, qv, torch.zeros_like(qv))
    lo = torch.where(~cond & (qv < qvs), -qc, torch.zeros_like(qc))
    x = ((qv - qvs) / (1 + L * _slope64(T, qvs, p))).clamp(lo, hi)
    for _ in range(60):  # bisection keeps what Newton's step would leave
        sat = _qvs64(T + L * x, p)
        value = qv - x - sat
        lo, hi = torch.where(value > 0, x, lo), torch.where(value > 0, hi, x)
        step = x + value / (1 + L * _slope64(T + L * x, sat, p))
        x = torch.where((step > lo) & (step < hi), step, 0.5 * (lo + hi))
    return x


def _kessler64(s, rc):
    """Warm-rain tendencies of theta, qv, qc and qr."""
    th, qv, qc, qr, p, rho, dt = s["theta"], s["qv"], s["qc"], s["qr"], s["p"], s["rho"], rc.dt
    L = 2.5e6 / 1004.0
    exner = (p / 1e5) ** (287.0 / 1004.0)
    x = _adjust64(th * exner, p, qv, qc)
    T, qv_a, qc_a = th * exner + L * x, qv - x, qc + x
    factor = 1 / (1 + 2.2 * dt * qr.clamp(min=0) ** 0.875)
    prod = torch.minimum((qc_a * (1 - factor) + factor * 1e-3 * dt * (qc_a - 1e-3).clamp(min=0)).clamp(min=0), qc_a) / dt
    sat = _qvs64(T, p)
    have = qr + prod * dt
    rain = 1e-3 * rho * have
    vent = (1.6 + 124.9 * rain ** 0.2046) * rain ** 0.525
    raw = vent / (2.55e8 / (p * sat) + 5.4e5) * (sat - qv_a) / (1e-3 * rho * sat)
    bound = (sat - qv_a) / (1 + 2.5e6 ** 2 * sat / (1004.0 * 461.5 * T * T))
    evap = torch.minimum(raw.clamp(min=0), torch.minimum(bound, have) / dt)
    evap = torch.where((have > 0) & (qv_a < sat), evap, torch.zeros_like(evap))
    fall = torch.where(qr < 1e-9, torch.zeros_like(qr), 36.34 * (1e-3 * rho * qr.clamp(min=1e-12)) ** 0.1346)
    flux = (fall * torch.sqrt(1.2 / rho)).clamp(max=20.0) * qr
    above = torch.zeros_like(flux)
    above[:, :, :-1] = (rho * flux)[:, :, 1:] / rho[:, :, :-1]
    rates = ((L * (x / dt - evap)) / exner, evap - x / dt, x / dt - prod, prod - evap + (above - flux) / rc.dz)
    res = []
    for t in rates:
        z = torch.zeros_like(t)
        z[1:-1, 1:-1] = t[1:-1, 1:-1]
        res.append(z)
    return res


def _steps64(s, rc, col, steps):
    for _ in range(steps):
        c2 = max(float((_GAMMA * s["p"] / s["rho"]).max()), float((_GAMMA * col["p0"] / col["rho0"]).max()))
        n = initial.resolve_substep_count(rc.dt, math.sqrt(c2), rc.dx, rc.dy, rc.dz)
        k1 = _slow64(s, rc, col)
        mid = dict(s)
        for f, t in zip(("u", "v", "w", "p"), k1):
            mid[f] = s[f] + rc.dt * t
        for f, a, b in zip(("u", "v", "w", "p"), k1, _slow64(mid, rc, col)):
            s[f] = s[f] + rc.dt * 0.5 * (a + b)
        _closure(s, rc, None, 0.0)
        begin = s["rho"].clone()
        mf = _loop64(s, rc, col, n)
        new = {f: _transport64(s[f], pd, begin, s["rho"], mf, rc) for f, pd in zip(SCALARS, POSITIVE)}
        s.update(new)
        for f, t in zip(SCALARS, _kessler64(s, rc)):
            inner = (s[f] + rc.dt * t).clamp(200.0, 700.0) if f == "theta" else (s[f] + rc.dt * t).clamp(0.0, 0.05)
            s[f] = s[f].clone()
            s[f][1:-1, 1:-1] = inner[1:-1, 1:-1]
        s["p"] = _eos64(s["rho"], s["theta"])
    return {k: s[k] for k in PROGNOSTIC}


def _closure64(s, rc):
    """Smagorinsky coefficients and tendencies on a level of uniform layers with open lateral faces."""
    u, v, w, rho = s["u"], s["v"], s["w"], s["rho"]
    dx, dy, dz = rc.dx, rc.dy, rc.dz

    def sh(f, ax, o):  # neighbour, the edge repeated
        n = f.shape[ax]
        idx = (torch.arange(n, device=f.device) + o).clamp(0, n - 1)
        return f.index_select(ax, idx)

    def ground(f):  # the face below, zero at the ground
        g = sh(f, 2, -1).clone()
        g[:, :, 0] = 0
        return g

    inner = torch.ones(1, 1, rc.nz, dtype=torch.float64, device=u.device)
    inner[:, :, -1] = 0  # edges between layers exist below the top layer only
    dudy, dvdx = (sh(u, 1, 1) - u) / dy, (sh(v, 0, 1) - v) / dx
    dudz, dwdx = inner * (sh(u, 2, 1) - u) / dz, (sh(w, 0, 1) - w) / dx
    dvdz, dwdy = inner * (sh(v, 2, 1) - v) / dz, (sh(w, 1, 1) - w) / dy
    s12 = 0.5 * (dudy + dvdx)
    s13, s23 = 0.5 * (dudz + inner * dwdx), 0.5 * (dvdz + inner * dwdy)
    w_b = ground(w)
    sq = 2 * (((u - sh(u, 0, -1)) / dx) ** 2 + ((v - sh(v, 1, -1)) / dy) ** 2 + ((w - w_b) / dz) ** 2)

    def corners(e, a, b, lower):
        e = e * e
        t = e + sh(e, a, -1)
        return 0.25 * (t + (ground(t) if lower else sh(t, b, -1)))

    # At a lateral edge the lower corner repeats the edge row itself: the difference across it is of that row.
    sq = sq + 4 * (corners(s12, 0, 1, False) + corners(s13, 0, 2, True) + corners(s23, 1, 2, True))
    strain = torch.sqrt(sq)
    delta = (dx * dy * dz) ** (1.0 / 3.0)
    nu = (0.18 ** 2 * delta ** 2 * strain).clamp(max=1000.0)
    kt = (3.0 * nu).clamp(max=1000.0)
    mu = rho * nu
    t12 = 2 * 0.25 * (mu + sh(mu, 0, 1) + sh(mu, 1, 1) + sh(sh(mu, 0, 1), 1, 1)) * s12
    pair = lambda ax: 0.5 * (0.5 * (mu + sh(mu, ax, 1)) + 0.5 * sh(mu + sh(mu, ax, 1), 2, 1))  # noqa: E731
    t13, t23 = pair(0) * (dudz + dwdx), pair(1) * (dvdz + dwdy)
    t11, t22 = 2 * mu * (u - sh(u, 0, -1)) / dx, 2 * mu * (v - sh(v, 1, -1)) / dy
    t33 = 2 * mu * (w - w_b) / dz
    du = ((sh(t11, 0, 1) - t11) / dx + (t12 - sh(t12, 1, -1)) / dy + (t13 - ground(t13)) / dz) / (0.5 * (rho + sh(rho, 0, 1)))
    dv = ((sh(t22, 1, 1) - t22) / dy + (t12 - sh(t12, 0, -1)) / dx + (t23 - ground(t23)) / dz) / (0.5 * (rho + sh(rho, 1, 1)))
    dw = ((sh(t33, 2, 1) - t33) + dz * (t13 - sh(t13, 0, -1)) / dx + dz * (t23 - sh(t23, 1, -1)) / dy) \
        / (0.5 * dz * (rho + sh(rho, 2, 1)))

    def scalar(f):
        tr = rho * kt
        flux = lambda ax, d: 0.5 * (tr + sh(tr, ax, 1)) * (sh(f, ax, 1) - f) / d  # noqa: E731
        fx, fy, fz = flux(0, dx), flux(1, dy), inner * flux(2, dz)
        return ((fx - sh(fx, 0, -1)) / dx + (fy - sh(fy, 1, -1)) / dy + (fz - ground(fz)) / dz) / rho

    def keep(t, i, j, k):
        z = torch.zeros_like(t)
        at = (slice(1, i), slice(1, j), slice(0, k))
        z[at] = t[at]
        return z

    return dict(nu_t=nu, K_theta=kt, K_q=kt, dudt=keep(du, -2, -1, -1), dvdt=keep(dv, -1, -2, -1),
                dwdt=keep(dw, -1, -1, -1), dthdt=keep(scalar(s["theta"]), -1, -1, None),
                dqvdt=keep(scalar(s["qv"]), -1, -1, None))
