"""The calls whose speed is tracked: what a user of the framework has it do.

Five families, each through the package's public entry points:

  level     a periodic level stepped with Level.advance (the drop-in path of a
            host driver): state handed over and taken back on the device, a
            run of steps between two outputs;
  ensemble  realisations of a parameter scan stepped together
            (Ensemble.step), written from and read into pinned host arrays
            that the program keeps (sh_ensemble_read of the C interface);
  spectrum  the gravitational-wave spectrum of a level (Level.gw_spectrum);
  amr       a refined run (Amr.step) with its regrids, from a host array to
            the levels' states on the device;
  server    requests of a parameter scan drained by a Server.

Initial data are those of the framework's workloads: Gaussian random fields
with flat power up to |k| = 1 for the axion strings (unit variance), tanh
bubble walls plus weak tensor modes for the phase transition, a network of
strings for the refined runs.  A pass starts from its inputs again, so it can
be repeated.
"""
import ctypes
import math

import numpy as np
import torch

import sledgehamr_gb300 as sh

DX = 0.25          # grid spacing of the uniform workloads
ETA0 = 0.1         # conformal time at which the axion runs start
LAP_ORDER = {"AxionStringsLap1": 1, "AxionStringsLap2": 2, "AxionStringsLap3": 3,
             "AxionStrings": 2, "NextToMinimalExample": 2, "MinimalExample": 2}
INTEGRATOR = {"rkn4": sh.RKN4, "rkn5": sh.RKN5, "ssprk3": sh.LSSSPRK3, "leapfrog": sh.LEAPFROG}
PRECISION = {"fp64": sh.PREC_FP64, "fp32k": sh.PREC_FP32_KAHAN, "fp32": sh.PREC_FP32}
FAMILY = {"lap1": sh.FAMILY_AXION_LAP1, "lap2": sh.FAMILY_AXION_LAP2, "fopt": sh.FAMILY_FOPT_GW}


def _level(name, project, N, integrator, steps, precision="fp64", max_grid=0, ko=0, gw=False):
    return {"name": name, "kind": "level", "project": project, "N": N, "integrator": integrator,
            "steps": steps, "precision": precision, "max_grid": max_grid, "ko": ko, "gw": gw}


def _ensemble(name, family, precision, sizes, steps):
    return {"name": name, "kind": "ensemble", "family": family, "precision": precision,
            "sizes": sizes, "steps": steps}


def _spectrum(name, N, pad, projection, unbinned, max_grid):
    return {"name": name, "kind": "spectrum", "N": N, "pad": pad, "projection": projection,
            "unbinned": unbinned, "max_grid": max_grid}


def _amr(name, precision, N0, steps, te_crit=1e-3):
    return {"name": name, "kind": "amr", "precision": precision, "N0": N0, "steps": steps,
            "te_crit": te_crit}


def _server(name, precision, nreq, sizes, levels):
    return {"name": name, "kind": "server", "precision": precision, "nreq": nreq, "sizes": sizes,
            "levels": levels}


def listed():
    return [
        # a small box of a test run or a scan: launches and latency
        _level("level small", "AxionStringsLap1", 32, "rkn4", 50),
        # the framework's single-level workload: one box, 7-point Laplacian
        _level("level one box", "AxionStringsLap1", 128, "rkn4", 50),
        # the drop-in project on a level chopped as a host driver chops it
        _level("level boxes", "AxionStrings", 256, "rkn4", 6, max_grid=32),
        # an odd size with the other integrator and dissipation switched on
        _level("level odd ssprk3", "NextToMinimalExample", 99, "ssprk3", 20, ko=2),
        # phase transition with the tensor modes, plain path
        _level("level fopt gw", "FirstOrderPhaseTransition", 160, "leapfrog", 10, max_grid=80,
               gw=True),
        # the precision form on a chopped level
        _level("level fp32", "AxionStringsLap2", 256, "rkn4", 12, precision="fp32k", max_grid=64),
        # a parameter scan of uneven boxes, batched, over the workload's steps
        _ensemble("ensemble axion", "lap1", "fp32k", "32,48,64,64,96,96,128,128", 200),
        # the phase transition's precision form
        _ensemble("ensemble fopt", "fopt", "fp32k", "160", 300),
        # its spectrum, between two runs of steps
        _spectrum("spectrum", 256, 1, 2, False, 128),
        # refined runs, plain and precision form
        _amr("amr", "fp64", 64, 8),
        _amr("amr fp32", "fp32k", 96, 8),
        # a burst of requests
        _server("server", "fp32k", 6, "64,96,128", "0,0,0,1,0,0"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["level", "level", "level", "level32", "fopt", "ensemble", "ensemble",
                       "spectrum", "amr", "server"])
    if kind == "level":
        N = _log(rng, 16, 224)
        project = rng.choice(["AxionStringsLap1", "AxionStringsLap2", "AxionStringsLap3",
                              "AxionStrings", "NextToMinimalExample", "MinimalExample"])
        integrator = rng.choice(["rkn4", "rkn4", "rkn4", "rkn5", "ssprk3"])
        c = _level("", project, N, integrator, max(2, min(50, int(8e7 / N ** 3))),
                   max_grid=rng.choice([0, 0, 32, 64]), ko=rng.choice([0, 0, 0, 2, 3]))
    elif kind == "level32":
        N = _log(rng, 24, 256)
        c = _level("", rng.choice(["AxionStringsLap1", "AxionStringsLap2"]), N, "rkn4",
                   max(2, min(50, int(1.5e8 / N ** 3))), precision="fp32k",
                   max_grid=rng.choice([0, 32, 64]))
    elif kind == "fopt":
        N = _log(rng, 24, 160)
        c = _level("", "FirstOrderPhaseTransition", N, "leapfrog",
                   max(2, min(40, int(4e7 / N ** 3))), precision=rng.choice(["fp64", "fp32k"]),
                   max_grid=rng.choice([0, 64, 80]), gw=rng.random() < 0.7)
    elif kind == "ensemble":
        family = rng.choice(["lap1", "lap1", "lap2", "fopt"])
        top = 144
        sizes = [_log(rng, 24, top) for _ in range(rng.randint(1, 8 if family != "fopt" else 2))]
        cells = sum(n ** 3 for n in sizes)
        c = _ensemble("", family, rng.choice(["fp32k", "fp32k", "fp32", "fp64"]),
                      ",".join(str(n) for n in sizes),
                      max(40, min(200, int((1.2e9 if family != "fopt" else 8e8) / cells))))
    elif kind == "spectrum":
        N = _log(rng, 32, 224)
        pad = 2 if N <= 100 and rng.random() < 0.4 else 1
        c = _spectrum("", N, pad, rng.choice([1, 2, 3]), rng.random() < 0.5,
                      rng.choice([0, 64, 128]))
    elif kind == "amr":
        c = _amr("", rng.choice(["fp64", "fp32k"]), 8 * rng.randint(6, 10), rng.randint(4, 8),
                 round(math.exp(rng.uniform(math.log(1e-3), math.log(5e-3))), 5))
    else:
        n = rng.randint(2, 5)
        c = _server("", "fp32k", n, ",".join(str(rng.choice([48, 64, 80, 96, 112]))
                                            for _ in range(n)),
                    ",".join(str(rng.choice([0, 0, 1])) for _ in range(n)))
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _gauss(N, L, kmax, g, tilt=0.0):
    """Real N^3 Gaussian field, power ~ |k|^tilt up to kmax, unit variance."""
    H = N // 2 + 1
    amp = torch.randn(2, N, N, H, generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.fftfreq(N, d=1.0 / N, device="cuda", dtype=torch.float64) ** 2
    h = torch.arange(H, device="cuda", dtype=torch.float64) ** 2
    k = 2 * math.pi / L * (f[:, None, None] + f[None, :, None] + h[None, None, :]).sqrt()
    keep = (k > 0) & (k <= max(kmax, 2.01 * math.pi / L))
    a = torch.complex(amp[0], amp[1]) * torch.where(keep, k.clamp_min(1e-9) ** (tilt / 2), 0 * k)
    x = torch.fft.irfftn(a, s=(N, N, N))
    return x / x.std()


def _strings(N, L, seed):
    """Psi1, Psi2, Pi1, Pi2 of a string network (cores where both fields
    cross zero), at rest."""
    g = _generator(seed)
    s = torch.zeros(4, N, N, N, device="cuda", dtype=torch.float64)
    s[0], s[1] = _gauss(N, L, 1.0, g), _gauss(N, L, 1.0, g)
    r = (s[0] ** 2 + s[1] ** 2 + 0.05).sqrt()
    s[:2] /= r
    return s


def _axion(N, L, seed):
    g = _generator(seed)
    s = torch.zeros(4, N, N, N, device="cuda", dtype=torch.float64)
    s[0], s[1] = _gauss(N, L, 1.0, g), _gauss(N, L, 1.0, g)
    return s


def _bubbles(N, L, g, count):
    """Field of tanh bubbles at random centres (periodic distance)."""
    x = torch.arange(N, device="cuda", dtype=torch.float64) * (L / N)
    c = torch.rand(count, 3, generator=g, device="cuda", dtype=torch.float64) * L
    phi = torch.zeros(N, N, N, device="cuda", dtype=torch.float64)
    for b in range(count):
        d = [((x - c[b, a] + L / 2) % L - L / 2) ** 2 for a in range(3)]
        r = (d[2][:, None, None] + d[1][None, :, None] + d[0][None, None, :]).sqrt()
        phi += 0.5 * (1 - torch.tanh(r - L / 8))
    return phi


def _fopt(N, L, seed, gw):
    """Phi, dPhi (u_ij, du_ij): bubbles, and the tensor modes of a run under
    way (weak, red)."""
    g = _generator(seed)
    s = torch.zeros(14 if gw else 2, N, N, N, device="cuda", dtype=torch.float64)
    s[0] = _bubbles(N, L, g, 4)
    for c in range(2, s.shape[0]):
        s[c] = 1e-3 * _gauss(N, L, 4.0, g, -2.0)
    return s


def _lambda_bar_params(lb):
    n = 3.0 + math.sqrt(9.0 - 8.0 * lb)
    return [-1.0, 3.0 * n / (4.0 * lb), -n * n / (8.0 * lb)]


def _couplings(n, seed):
    return np.exp(np.random.default_rng(seed).uniform(math.log(0.5), math.log(2.0), n))


def _level_params(project):
    if project == "FirstOrderPhaseTransition":
        return [0.0, *_lambda_bar_params(0.8)]
    return {"AxionStrings": [], "MinimalExample": [], "NextToMinimalExample": [1.0]}.get(
        project, [1.0, 0.0])


def _requests(case, seed):
    """Two-bubble collisions: separation d, wall Lorentz factor, thick or
    thin wall; box d + 24, run to t = d."""
    rng = np.random.default_rng(seed)
    out = []
    for n, lev in zip(case["sizes"].split(","), case["levels"].split(",")):
        d, gamma = rng.uniform(8.0, 20.0), rng.uniform(1.0, 4.0)
        N, m = int(n), int(lev)
        Nb = N >> m
        L = d + 24.0
        wc, dx = 1.0 / gamma, L / Nb
        lcut = 4.0 + 10.0 * wc
        r = np.arange(int(lcut * 16.0) + 2) / 16.0
        x = (r - 4.0) / wc
        prof = np.stack([0.5 * (1 - np.tanh(x)),
                         0.5 * math.sqrt(1 - 1 / gamma ** 2) / wc / np.cosh(x) ** 2])
        c = np.array([[L / 2 - d / 2, L / 2, L / 2], [L / 2 + d / 2, L / 2, L / 2]])
        lb = (0.6, 1.0)[int(rng.integers(0, 2))]
        out.append(dict(N=Nb, dx=dx, dt=0.2 * dx, t_end=d, params=[*_lambda_bar_params(lb), 0.0],
                        centres=c, profile=prof, inv_dx=16.0, Lcut=lcut, max_level=m,
                        te_crit=(1e-2, 1e-2), regrid_dt=8 * 0.2 * dx))
    return out


def prepare(case, seed):
    kind = case["kind"]
    ctx = sh.Context(0)
    if kind == "level":
        N = case["N"]
        fopt = case["project"] == "FirstOrderPhaseTransition"
        order = LAP_ORDER.get(case["project"], 2)
        nghost = max(order, case["ko"], 1)
        lev = sh.Level.periodic(ctx, case["project"], N, nghost, max_grid=case["max_grid"],
                                with_gw=case["gw"], precision=PRECISION[case["precision"]])
        state = _fopt(N, N * DX, seed, case["gw"]) if fopt else _axion(N, N * DX, seed)
        out = torch.empty_like(state)
        torch.cuda.synchronize()
        return dict(kind=kind, ctx=ctx, lev=lev, state=state, out=out, steps=case["steps"],
                    integrator=INTEGRATOR[case["integrator"]], t0=0.0 if fopt else ETA0,
                    dt=0.2 * DX if fopt else 0.25 * DX, params=_level_params(case["project"]),
                    ko=case["ko"], ko_strength=[0.05] * lev.ncomp if case["ko"] else None)
    if kind == "ensemble":
        Ns = [int(n) for n in case["sizes"].split(",")]
        fopt = case["family"] == "fopt"
        params = ([[*_lambda_bar_params(0.8), 0.0]] * len(Ns) if fopt else
                  [[x, 0, 0, 0] for x in _couplings(len(Ns), seed)])
        E = sh.Ensemble(ctx, FAMILY[case["family"]], PRECISION[case["precision"]], Ns,
                        [DX] * len(Ns), params)
        make = (lambda n, s: _fopt(n, n * DX, s, True)) if fopt else \
            (lambda n, s: _axion(n, n * DX, s))
        states = []
        for r, n in enumerate(Ns):
            host = torch.empty(E.ncomp, n, n, n, dtype=torch.float64).pin_memory()
            host.copy_(make(n, 1000 * seed + r))
            states.append(host.numpy())
        torch.cuda.synchronize()
        dt = 0.2 * DX if fopt else 0.25 * DX
        E.tune(dt, tile_nz=16)
        E.set_graph(True)
        out = [torch.empty(E.ncomp, n, n, n, dtype=torch.float64).pin_memory() for n in Ns]
        return dict(kind=kind, ctx=ctx, E=E, states=states, out=out, t0=0.0 if fopt else ETA0,
                    dt=dt, steps=case["steps"])
    if kind == "spectrum":
        N = case["N"]
        lev = sh.Level.periodic(ctx, "FirstOrderPhaseTransition", N, 2, max_grid=case["max_grid"],
                                with_gw=True)
        state = _fopt(N, N * DX, seed, True)
        torch.cuda.synchronize()
        lev.write_device(state.data_ptr())
        ctx.synchronize()
        return dict(kind=kind, ctx=ctx, lev=lev, pad=case["pad"], projection=case["projection"],
                    unbinned=case["unbinned"])
    if kind == "amr":
        N0 = case["N0"]
        cfg = sh.amr_config("AxionStringsLap2", precision=PRECISION[case["precision"]], N0=N0,
                            L=N0 * DX, cfl=0.25, t_start=4.0, nghost=2, max_level=2,
                            blocking_factor=8, max_grid_size=32, n_error_buf=2, regrid_dt=0.25,
                            te_crit=[case["te_crit"]] * 4, params=[1.0, 0.0],
                            string_width_threshold=1.5)
        host = _strings(N0, N0 * DX, seed).cpu().numpy()
        # room for every level's boxes and cells (their number is the run's)
        out = [(np.zeros((8192, 2, 3), dtype=np.int64),
                torch.zeros(4 * (N0 << q) ** 3, device="cuda", dtype=torch.float64))
               for q in range(3)]
        torch.cuda.synchronize()
        return dict(kind=kind, ctx=ctx, cfg=cfg, host=host, out=out, steps=case["steps"])
    srv = sh.Server(ctx, PRECISION[case["precision"]],
                    2 * sum(int(n) ** 3 for n in case["sizes"].split(",")))
    return dict(kind=kind, ctx=ctx, srv=srv, requests=_requests(case, seed))


def run(s):
    kind = s["kind"]
    if kind == "level":
        lev = s["lev"]
        lev.write_device(s["state"].data_ptr())
        lev.set_time(s["t0"])
        for _ in range(s["steps"]):
            lev.advance(s["integrator"], s["dt"], DX, params=s["params"], ko_order=s["ko"],
                        ko_strength=s["ko_strength"])
        lev.read_device(s["out"].data_ptr())
        return s["out"]
    if kind == "ensemble":
        E = s["E"]
        for r, host in enumerate(s["states"]):
            E.write(r, host)
        E.set_time(s["t0"])
        E.step(s["dt"], s["steps"])
        for r, host in enumerate(s["out"]):
            E.check(s["ctx"].lib.sh_ensemble_read(E.h, r, ctypes.c_void_p(host.data_ptr())), "read")
        return s["out"]
    if kind == "spectrum":
        bins, ks = s["lev"].gw_spectrum(s["pad"], s["projection"], s["unbinned"])
        return {"bins": bins, "ks": ks}
    if kind == "amr":
        sim = sh.Amr(s["ctx"], s["cfg"], s["host"])
        sim.step(s["steps"])
        for lev in range(sim.info()["finest"] + 1):
            view = sim.level(lev)
            boxes, state = s["out"][lev]
            boxes[:len(view.boxes)] = view.boxes
            sh.Level.read_device(view, state.data_ptr(), sh.SH_NEW, 1)
        sim.close()
        return s["out"]
    ids = [s["srv"].submit(**r) for r in s["requests"]]
    while True:
        running, queued, _ = s["srv"].step()
        if running == 0 and queued == 0:
            break
    return [dict(zip(("bins", "ks"), s["srv"].result(i))) for i in ids]


# ---- bytes and operations that a pass cannot do without -----------------------

def _rhs_ops(project, gw):
    """Adds and multiplies of one evaluation of the equations per cell."""
    order = LAP_ORDER.get(project, 2)
    lap = 6 * order + order + 2
    if project == "FirstOrderPhaseTransition":
        return lap + 6 + (6 * (lap + 2) + 3 * 7 if gw else 0)
    return 2 * lap + 16


def work(case):
    """Every step reads its state and writes the next one; operations are
    those of the equations and the integrator's combinations."""
    kind = case["kind"]
    if kind == "level":
        cells = case["N"] ** 3
        ncomp = (14 if case["gw"] else 2) if case["project"] == "FirstOrderPhaseTransition" else 4
        evals = {"rkn4": 3, "rkn5": 4, "ssprk3": 3, "leapfrog": 2}[case["integrator"]]
        word = 8  # FP64, or an FP32 value and its FP32 compensation
        return {"bytes": cells * ncomp * (2 * word * case["steps"] + 16.0),
                "flops": cells * case["steps"] * evals *
                (_rhs_ops(case["project"], case["gw"]) + 3.0 * ncomp)}
    if kind == "ensemble":
        cells = sum(int(n) ** 3 for n in case["sizes"].split(","))
        fopt = case["family"] == "fopt"
        ncomp, evals = (14, 2) if fopt else (4, 3)
        word = 4 if case["precision"] == "fp32" else 8
        ops = _rhs_ops("FirstOrderPhaseTransition", True) if fopt else \
            _rhs_ops("AxionStringsLap1" if case["family"] == "lap1" else "AxionStringsLap2", False)
        return {"bytes": cells * ncomp * (2.0 * word * case["steps"] + 16.0),
                "flops": cells * case["steps"] * evals * (ops + 3.0 * ncomp)}
    if kind == "spectrum":
        P = case["N"] * case["pad"]
        return {"bytes": 6.0 * 8 * case["N"] ** 3,
                "flops": 6 * 2.5 * P ** 3 * math.log2(P ** 3) + 67.0 * P ** 3 / 2}
    if kind == "amr":
        # level 0 and about as many cells again on each finer level, which
        # takes two and four steps for one of level 0
        cells = case["N0"] ** 3 * (1 + 2 + 4) * case["steps"]
        return {"bytes": 4.0 * 16 * cells, "flops": 3.0 * (2 * 16 + 28) * cells}
    req = _requests(case, 0)
    up = sum(r["N"] ** 3 * math.ceil(14.0 / r["dt"]) for r in req)
    return {"bytes": 14.0 * 16 * up,
            "flops": 2.0 * (_rhs_ops("FirstOrderPhaseTransition", True) + 42) * up}


# ---- the same in 64 bits with plain torch -------------------------------------

def _shift(x, d, ax):
    return torch.roll(x, -d, ax)


def _lap(x, order, dx):
    ring = [sum(_shift(x, d, ax) for ax in (-1, -2, -3) for d in (r, -r))
            for r in range(1, order + 1)]
    if order == 1:
        return (ring[0] - 6 * x) / dx ** 2
    if order == 2:
        return (16 * ring[0] - ring[1] - 90 * x) / (12 * dx ** 2)
    return (270 * ring[0] - 27 * ring[1] + 2 * ring[2] - 1470 * x) / (180 * dx ** 2)


def _grad(x, ax, dx):
    return (8 * (_shift(x, 1, ax) - _shift(x, -1, ax)) -
            (_shift(x, 2, ax) - _shift(x, -2, ax))) / (12 * dx)


def _axion_accel(y, p, eta, order, lam, c):
    v = lam * (eta * eta * (y[0] ** 2 + y[1] ** 2 - 1.0) + c)
    return torch.stack([_lap(y[q], order, DX) - 2.0 / eta * p[q] - y[q] * v for q in (0, 1)])


def _dissipation(u, order, strength):
    if order == 0:
        return 0.0
    w = {2: {0: 6, 1: -4, 2: 1}, 3: {0: -20, 1: 15, 2: -6, 3: 1}}[order]
    s = sum(3 * m * u if d == 0 else
            sum(m * (_shift(u, d, ax) + _shift(u, -d, ax)) for ax in (-1, -2, -3))
            for d, m in w.items())
    return -strength * s / 16 / DX if order == 2 else strength * s / 64 / DX


def _exact_axion(state, t, dt, steps, integrator, order, lam, c, ko):
    y, p = state[:2].clone(), state[2:].clone()

    def a(y, p, eta):
        return _axion_accel(y, p, eta, order, lam, c) + _dissipation(p, ko, 0.05)

    def f(u, eta):
        return torch.cat([u[2:] + _dissipation(u[:2], ko, 0.05), a(u[:2], u[2:], eta)])

    for _ in range(steps):
        if integrator == "ssprk3":
            u0 = torch.cat([y, p])
            k = f(u0, t)
            k = f(u0 + dt * k, t + dt) + k
            k = f(u0 + dt / 4 * k, t + dt / 2) + 0.25 * k
            u1 = u0 + dt * 2.0 / 3 * k
            y, p = u1[:2], u1[2:]
        else:
            k0 = a(y, p, t)
            k1 = a(y + 0.5 * dt * p + dt * dt / 8 * k0, p, t + 0.5 * dt)
            k2 = a(y + dt * p + dt * dt / 2 * k1, p, t + dt)
            y, p = (y + dt * p + dt * dt * (k0 / 6 + k1 / 3),
                    p + dt * (k0 / 6 + 2 * k1 / 3 + k2 / 6))
        t += dt
    return torch.cat([y, p])


def _exact_fopt(state, dt, steps, q):
    def accel(x):
        g = [_grad(x[0], ax, DX) for ax in (-1, -2, -3)]
        out = [_lap(x[0], 2, DX) + x[0] * (q[0] + x[0] * (q[1] + x[0] * q[2]))]
        for n, (i, j) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            if x.shape[0] > 1:
                out.append(_lap(x[1 + n], 2, DX) + g[i] * g[j])
        return torch.stack(out)

    gw = state.shape[0] > 2
    x = torch.cat([state[:1], state[2:8]]) if gw else state[:1].clone()
    v = torch.cat([state[1:2], state[8:]]) if gw else state[1:2].clone()
    acc = accel(x)
    for _ in range(steps):
        v = v + 0.5 * dt * acc
        x = x + dt * v
        acc = accel(x)
        v = v + 0.5 * dt * acc
    return torch.cat([x[:1], v[:1], x[1:], v[1:]]) if gw else torch.cat([x, v])


def _exact_spectrum(state, P, projection, unbinned):
    # components of du in the order xx xy xz yy yz zz
    N = state.shape[-1]
    F = []
    for c in (8, 11, 12, 9, 13, 10):
        u = torch.zeros(P, P, P, device="cuda", dtype=torch.float64)
        u[:N, :N, :N] = state[c]
        F.append(torch.fft.rfftn(u))
    n = torch.arange(P, device="cuda", dtype=torch.float64)
    th = 2 * math.pi / P * torch.where(n - P > -P / 2 - 1, n - P, n)
    k1 = {1: torch.sin(th), 2: (8 * torch.sin(th) - torch.sin(2 * th)) / 6,
          3: (45 * torch.sin(th) - 9 * torch.sin(2 * th) + torch.sin(3 * th)) / 30}[projection]
    H = P // 2 + 1
    k = [k1[None, None, :H], k1[None, :, None], k1[:, None, None]]
    norm = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    norm[0, 0, 0] = 1.0
    k = [x / norm.sqrt() for x in k]
    m = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
    v = [sum(F[m[i][j]] * k[j] for j in range(3)) for i in range(3)]
    s = sum(k[i] * v[i] for i in range(3))
    val = torch.zeros_like(norm)
    tr = 0.0
    for i in range(3):
        for j in range(i, 3):
            w = F[m[i][j]] - k[i] * v[j] - v[i] * k[j] + k[i] * k[j] * s
            val += (1 if i == j else 2) * (w.real ** 2 + w.imag ** 2)
            tr = tr + w if i == j else tr
    val -= 0.5 * (tr.real ** 2 + tr.imag ** 2)
    val[0, 0, 0] = 0.0
    a = torch.arange(P, device="cuda")
    f = torch.where(a >= P // 2, a - P, a) ** 2
    val[:, :, 1:] *= 2.0
    if P % 2 == 0:
        val[:, :, P // 2] *= 0.5
    sq = (f[:, None, None] + f[None, :, None] + f[None, None, :H]).reshape(-1)
    if unbinned:
        # every k^2 that a P^3 grid holds
        one = torch.unique(torch.tensor([(x if x < (P + 1) // 2 else x - P) ** 2
                                         for x in range(P)], device="cuda"))
        two = torch.unique(one[:, None] + one[None, :])
        ks = torch.unique(two[:, None] + one[None, :])
        idx = torch.searchsorted(ks, sq)
    else:
        ks = torch.arange(int(math.sqrt(3) / 2 * P + 0.5) + 1, device="cuda") ** 2
        idx = (sq.double().sqrt() + 0.5).long()
    bins = torch.zeros(ks.numel(), device="cuda", dtype=torch.float64)
    bins.index_add_(0, idx, val.reshape(-1))
    return {"bins": (bins / float(P) ** 6).cpu().numpy(), "ks": ks.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "level":
        N = case["N"]
        if case["project"] == "FirstOrderPhaseTransition":
            return _exact_fopt(_fopt(N, N * DX, seed, case["gw"]), 0.2 * DX, case["steps"],
                               _lambda_bar_params(0.8))
        if case["integrator"] == "rkn5":
            return None
        c = 0.0 if case["project"].startswith("AxionStringsLap") else 0.56233
        return _exact_axion(_axion(N, N * DX, seed), ETA0, 0.25 * DX, case["steps"],
                            case["integrator"],
                            LAP_ORDER[case["project"]], 1.0, c, case["ko"])
    if kind == "ensemble":
        Ns = [int(n) for n in case["sizes"].split(",")]
        lam = _couplings(len(Ns), seed)
        out = []
        for r, n in enumerate(Ns):
            if case["family"] == "fopt":
                e = _exact_fopt(_fopt(n, n * DX, 1000 * seed + r, True), 0.2 * DX, case["steps"],
                                _lambda_bar_params(0.8))
            else:
                e = _exact_axion(_axion(n, n * DX, 1000 * seed + r), ETA0, 0.25 * DX,
                                 case["steps"], "rkn4", 1 if case["family"] == "lap1" else 2,
                                 float(lam[r]), 0.0, 0)
            out.append(e.cpu().numpy())
        return out
    if kind == "spectrum":
        N = case["N"]
        return _exact_spectrum(_fopt(N, N * DX, seed, True), N * case["pad"], case["projection"],
                               case["unbinned"])
    return None
