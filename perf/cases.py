"""The calls a program makes into this solver, as measurable cases.

Each case is one pass through the public entry points (steppers, tendency,
derivatives, ensembles, the host-state stepper) on a doubly periodic planar
hexagonal mesh.  `exact` evaluates the same discrete equations in plain torch
float64: mesh tables, tendencies, time stepping, and derivatives by torch's
own automatic differentiation.
"""
import functools
import math

import numpy as np
import torch

import omega_playground_gb300 as og
from omega_playground_gb300 import autograd as og_autograd

DC = 1e4           # cell spacing, m
GRAV = 9.81
F0 = 1e-4
H0 = 1000.0
DT = 0.2 * DC / math.sqrt(GRAV * H0)   # 0.2 gravity-wave CFL

# dissipation settings: none, velocity del2 only (the small RK4 workload and
# the ensembles), every term (the large LSRK workload)
DISS = {"none": (0.0, 0.0, 0.0, 0.0), "vel2": (1e3, 0.0, 0.0, 0.0),
        "tr2": (1e3, 0.0, 1e3, 0.0), "all": (1e3, 1e9, 1e3, 1e9)}


def _case(name, kind, nx, ny, K, T, diss, **more):
    c = {"kind": kind, "nx": nx, "ny": ny, "K": K, "T": T, "diss": diss}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # one do_step call on a test-sized mesh: launches and latency
        _case("rk4_12x10x3", "step", 12, 10, 3, 2, "all", stepper="rk4",
              steps=1, graph=False),
        # the plain RK4 workload: 10 steps replayed from a captured graph
        _case("rk4_64x64x64", "step", 64, 64, 64, 1, "vel2", stepper="rk4",
              steps=10, graph=True),
        # the reference benchmark's protocol: one tracer, every dissipation
        # term, step calls one by one
        _case("lsrk5_100x100x64", "step", 100, 100, 64, 1, "all",
              stepper="lsrk5", steps=4, graph=False),
        # the large workload: one step of a time loop
        _case("lsrk5_512x512x64x8", "step", 512, 512, 64, 8, "all",
              stepper="lsrk5", steps=1, graph=True),
        # a single-level model (the reference's convergence and double-vortex
        # programs have few levels), no tracers, no dissipation
        _case("rk4_200x230x1", "step", 200, 230, 1, 0, "none", stepper="rk4",
              steps=5, graph=True),
        # one evaluation for a caller's own stepper, ragged level count
        _case("tendency_75x62x33x3", "tendency", 75, 62, 33, 3, "tr2"),
        # forward-mode derivative of a short trajectory
        _case("tlm_96x80x32x2", "tlm", 96, 80, 32, 2, "vel2", steps=2),
        # a tendency inside a torch program: value and gradient
        _case("vjp_64x64x40x2", "vjp", 64, 64, 40, 2, "all"),
        # checkpointed adjoint of a trajectory (the 128x128x32 workload)
        _case("adjoint_128x128x32x2", "adjoint", 128, 128, 32, 2, "vel2",
              steps=16, snapshots=5),
        # members of uneven size advanced together
        _case("batch_12_members", "batch", 96, 96, 48, 2, "vel2", members=12,
              steps=2),
        # their checkpointed gradients
        _case("adjoint_ensemble_4", "adjoint_ensemble", 48, 48, 32, 2, "vel2",
              members=4, steps=8, snapshots=3),
        # a state that lives in host memory, copied in and out every call
        _case("host_lsrk5_192x192x64x8", "host", 192, 192, 64, 8, "all",
              steps=1),
    ]


def draw(rng):
    """One more case: cells x levels spread over its logarithm, aspect, level
    and tracer counts ragged."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "tendency", "tlm", "vjp",
                       "adjoint", "batch", "adjoint_ensemble", "host"])
    most = {"step": 6e6, "tendency": 6e6, "tlm": 1e6, "vjp": 1e6,
            "adjoint": 5e5, "batch": 5e5, "adjoint_ensemble": 1e5,
            "host": 3e6}[kind]
    K = rng.choice([1, 2, 5, 16, 31, 32, 33, 40, 60, 64, 64, 80, 96])
    cells = max(96, logint(400, most) // K)
    ny = max(8, 2 * int(round(math.sqrt(cells) * rng.uniform(0.35, 0.65))))
    nx = max(8, int(round(cells / ny)))
    diff = kind in ("tlm", "vjp", "adjoint", "adjoint_ensemble")
    T = rng.randint(0, 4 if diff or kind == "batch" else 10)
    c = _case(None, kind, nx, ny, K, T,
              rng.choice(["none", "vel2", "tr2", "all", "all"]))
    if kind == "step":
        c.update(stepper=rng.choice(["rk4", "lsrk5", "euler"]),
                 steps=rng.randint(1, 3), graph=rng.random() < 0.7)
    elif kind in ("tlm", "host"):
        c.update(steps=rng.randint(1, 2))
    elif kind == "adjoint":
        c.update(steps=rng.randint(3, 20), snapshots=rng.randint(2, 6))
    elif kind == "batch":
        c.update(members=rng.randint(2, 16), steps=rng.randint(1, 3))
    elif kind == "adjoint_ensemble":
        c.update(members=rng.randint(2, 6), steps=rng.randint(3, 8),
                 snapshots=rng.randint(2, 4))
    return c


def _members(case):
    """Sizes of an ensemble's members: uneven meshes, levels and tracers."""
    out = []
    for i in range(case.get("members", 1)):
        s = 1.0 - 0.6 * ((5 * i) % 7) / 7.0
        out.append({**case, "nx": max(8, int(case["nx"] * s)),
                    "ny": max(8, 2 * int(case["ny"] * s / 2)),
                    "K": max(1, case["K"] - (3 * i) % max(1, case["K"] // 2)),
                    "T": case["T"] if case["kind"] == "adjoint_ensemble"
                    else max(0, case["T"] - i % 2)})
    return out


# ---------------------------------------------------------------- inputs ---

@functools.lru_cache(maxsize=4)
def _hex(nx, ny):
    """Tables of the doubly periodic hexagonal mesh (even ny): row-major
    cells, cell c owning edges 3c..3c+2 (west, south-west, south-east) and
    vertices 2c, 2c+1; odd rows shifted half a cell east."""
    col, row = np.meshgrid(np.arange(nx), np.arange(ny))
    col, row = col.ravel(), row.ravel()
    odd = row % 2
    dcol = np.where(odd[:, None], [[-1, 0, 1, 1, 1, 0]], [[-1, -1, 0, 1, 0, -1]])
    nb = (row[:, None] + [[0, -1, -1, 0, 1, 1]]) % ny * nx + \
        (col[:, None] + dcol) % nx
    c = np.arange(nx * ny)
    ce = np.stack([3 * c, 3 * c + 1, 3 * c + 2, 3 * nb[:, 3], 3 * nb[:, 4] + 1,
                   3 * nb[:, 5] + 2], 1)
    cv = np.stack([2 * c, 2 * c + 1, 2 * nb[:, 2], 2 * nb[:, 3] + 1,
                   2 * nb[:, 3], 2 * nb[:, 4] + 1], 1)
    E, V = 3 * nx * ny, 2 * nx * ny
    coe, voe = np.zeros((E, 2), np.int64), np.zeros((E, 2), np.int64)
    eoe, woe = np.zeros((E, 10), np.int64), np.zeros((E, 10))
    third, sixth = 1 / 3, 1 / 6
    w = np.array([[third, sixth, 0, sixth, third],
                  [third, -sixth, 0, sixth, -third],
                  [-third, -sixth, 0, -sixth, -third]]) / math.sqrt(3.0)
    for j in range(3):
        coe[ce[:, j], 1] = c
        coe[ce[:, j + 3], 0] = c
        voe[ce[:, j], 0], voe[ce[:, j], 1] = cv[:, j + 1], cv[:, j]
        for s in range(5):
            eoe[ce[:, 3 + j], s] = ce[:, (j + 4 + s) % 6]
            eoe[ce[:, j], 5 + s] = ce[:, (j + 1 + s) % 6]
            woe[ce[:, 3 + j], s] = woe[ce[:, j], 5 + s] = w[j, s]
    cov, eov = np.zeros((V, 3), np.int64), np.zeros((V, 3), np.int64)
    for k, v in ((2, 1), (0, 3), (1, 5), (0, 0), (1, 2), (2, 4)):
        cov[cv[:, v], k] = c
    for k, v, e in ((0, 0, 0), (0, 1, 0), (2, 2, 1), (2, 1, 1), (1, 2, 2),
                    (1, 3, 2)):
        eov[cv[:, v], k] = ce[:, e]
    x = DC * col + np.where(odd, DC, DC / 2)
    y = DC * (row + 1) * math.sqrt(3.0) / 2
    t = dict(nb=nb, ce=ce, coe=coe, voe=voe, eoe=eoe, woe=woe, cov=cov,
             eov=eov, x=x, y=y,
             sc=np.where(coe[ce, 0] == c[:, None], 1.0, -1.0),
             sv=np.where(voe[eov, 0] == np.arange(V)[:, None], -1.0, 1.0))
    t = {k: torch.from_numpy(np.ascontiguousarray(a)).cuda()
         for k, a in t.items()}
    t["Lx"], t["Ly"] = nx * DC, ny * DC * math.sqrt(3.0) / 2
    t["dv"], t["area"] = DC / math.sqrt(3.0), DC * DC * math.sqrt(3.0) / 2
    return t


def _inputs(case, seed, what=0):
    """(h, vn, tr): 1000 m plus two 1 m bumps per level, divergence-free
    velocity noise of 0.05 m/s, tracers as thickness times four plane waves
    in [0, 1]."""
    m, K, T = _hex(case["nx"], case["ny"]), case["K"], case["T"]
    g = torch.Generator(device="cuda").manual_seed(1000003 * what + seed)
    C, dev = case["nx"] * case["ny"], "cuda"

    def rand(*n):
        return torch.rand(n, generator=g, device=dev, dtype=torch.float64)

    h = torch.full((C, K), H0, device=dev, dtype=torch.float64)
    u = rand(2, 2, K)
    for b in range(2):
        d2 = 0
        for a, L, ub in ((m["x"], m["Lx"], u[b, 0]), (m["y"], m["Ly"], u[b, 1])):
            d = a[:, None] - ub[None, :] * L
            d2 = d2 + (d - L * torch.round(d / L)) ** 2
        h += torch.exp(-d2 / (0.1 * m["Lx"]) ** 2)
    psi = rand(2 * C, K) - 0.5
    vn = (psi[m["voe"][:, 0]] - psi[m["voe"][:, 1]]) / m["dv"]
    vn *= 0.05 / vn.square().mean().sqrt()
    tr = torch.zeros((T, C, K), device=dev, dtype=torch.float64)
    for l in range(T):
        a = rand(4, 3).cpu()
        k = torch.randint(-2, 3, (4, 2), generator=g, device=dev).cpu()
        f = torch.zeros(C, device=dev, dtype=torch.float64)
        for w in range(4):
            kx, ky = int(k[w, 0]) or 1, int(k[w, 1])
            f += (0.5 + 0.5 * float(a[w, 0])) * torch.sin(
                2 * math.pi * (kx * m["x"] / m["Lx"] + ky * m["y"] / m["Ly"]
                               + float(a[w, 1])))
        f = (f - f.min()) / (f.max() - f.min())
        lev = 1 - 0.3 * torch.arange(K, device=dev, dtype=torch.float64) / K
        tr[l] = h * f[:, None] * lev[None, :]
    return h, vn, tr


def _cotangent(case, seed):
    """dL/dx of a loss on the state: each field's scale, smooth in space."""
    h, vn, tr = _inputs(case, seed, what=1)
    return h - H0, 1e2 * vn, 1e-3 * tr


def _state(mesh, T, fields):
    s = og.ShallowWaterState(mesh, T)
    for dst, src in zip(s.as_tensors(), fields):
        dst.copy_(src)
    return s


def _model(case):
    v2, v4, k2, k4 = DISS[case["diss"]]
    mesh = og.PlanarHexagonalMesh(case["nx"], case["ny"], DC, case["K"])
    params = og.ShallowWaterParams(
        m_f0=F0, m_grav=GRAV, m_visc_del2=v2, m_visc_del4=v4, m_eddy_diff2=k2,
        m_eddy_diff4=k4, m_ntracers=case["T"])
    return mesh, og.ShallowWaterModel(mesh, params)


def prepare(case, seed):
    kind, T = case["kind"], case["T"]
    if kind in ("batch", "adjoint_ensemble"):
        ms = [(c,) + _model(c) for c in _members(case)]
        st = [_state(mesh, c["T"], _inputs(c, seed, 2 + i))
              for i, (c, mesh, _) in enumerate(ms)]
        models = [md for _, _, md in ms]
        if kind == "batch":
            b = og.Batch(models, st, "rk4")
            # the shape the tuner prefers where it has been run: one launch
            # per pass, 256 threads, two elements a thread
            b.set_config(b.config_count() - 1)
            return dict(case=case, batch=b, states=st)
        adjs = [og.Adjoint(md, case["snapshots"]) for md in models]
        return dict(case=case, ens=og.AdjointEnsemble(adjs), states=st,
                    finals=[_state(mesh, c["T"], ()) for c, mesh, _ in ms],
                    lams=[_state(mesh, c["T"], ()) for c, mesh, _ in ms],
                    seeds=[_state(mesh, c["T"], _cotangent(c, seed + i))
                           for i, (c, mesh, _) in enumerate(ms)])
    mesh, model = _model(case)
    x = _inputs(case, seed)
    s = dict(case=case, model=model)
    if kind == "host":
        K = case["K"]
        s["stepper"] = og.HostStepper(model, "lsrk", 5,
                                      levels=og.HostStepper.edge_layout(K, 16, 4))
        s["arrays"] = s["stepper"].pinned_state()
        for dst, src in zip(s["arrays"], x):
            dst[...] = src.cpu().numpy()
        return s
    if kind == "vjp":
        s["adj"] = og.Adjoint(model, 1)
        s["x"] = [f.requires_grad_(True) for f in x]
        s["cot"] = _cotangent(case, seed)
        return s
    s["state"] = _state(mesh, T, x)
    if kind == "step":
        s["stepper"] = (og.RK4Stepper(model) if case["stepper"] == "rk4" else
                        og.LSRKStepper(model, 5 if case["stepper"] == "lsrk5"
                                       else 1))
    elif kind == "tendency":
        s["tend"] = _state(mesh, T, ())
    elif kind == "tlm":
        s["adj"] = og.Adjoint(model, 1)
        s["seed"] = _state(mesh, T, _cotangent(case, seed))
        s["dx"] = _state(mesh, T, ())
    elif kind == "adjoint":
        s["adj"] = og.Adjoint(model, case["snapshots"])
        s["seed"] = _state(mesh, T, _cotangent(case, seed))
        s["lam"], s["final"] = _state(mesh, T, ()), _state(mesh, T, ())
    return s


def _out(state):
    return [t for t in state.as_tensors() if t.numel()]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":  # the state moves on, as in a time loop
        dt = DT / 4 if case["stepper"] == "euler" else DT
        if case["graph"]:
            s["stepper"].step(s["state"], 0.0, dt, case["steps"])
        else:
            for _ in range(case["steps"]):
                s["stepper"].do_step(0.0, dt, s["state"])
        return _out(s["state"])
    if kind == "tendency":
        s["model"].compute_tendency(s["tend"], s["state"], 0.0)
        return _out(s["tend"])
    if kind == "host":
        s["stepper"].step(*s["arrays"], 0.0, DT, case["steps"])
        return [a for a in s["arrays"] if a.size]
    if kind == "tlm":
        s["dx"].copy_from(s["seed"])
        s["adj"].tlm_apply(s["state"], s["dx"], 0.0, DT, case["steps"])
        return _out(s["dx"])
    if kind == "vjp":
        out = og_autograd.tendency(s["adj"], *s["x"])
        grads = torch.autograd.grad(out, s["x"], s["cot"])
        return [t.detach() for t in (*out, *grads) if t.numel()]
    if kind == "adjoint":
        s["adj"].forward(s["state"], 0.0, DT, case["steps"], s["final"])
        s["lam"].copy_from(s["seed"])
        s["adj"].backward(s["lam"])
        return _out(s["final"]) + _out(s["lam"])
    if kind == "batch":
        s["batch"].step(0.0, DT, case["steps"], check_status=False)
        return [t for st in s["states"] for t in _out(st)]
    s["ens"].forward(s["states"], 0.0, DT, case["steps"], s["finals"])
    for lam, seed in zip(s["lams"], s["seeds"]):
        lam.copy_from(seed)
    s["ens"].backward(s["lams"])
    return [t for a, b in zip(s["finals"], s["lams"])
            for t in _out(a) + _out(b)]


# ----------------------------------------------------------------- floor ---

def _ops(case):
    """Float64 multiply-adds per cell and level of one evaluation: per edge
    two sums over eight edges, flux, kinetic energy and the gradients; per
    vertex vorticity and thickness; per cell the divergence; seven-point
    sums per tracer and dissipation term."""
    v2, v4, k2, k4 = DISS[case["diss"]]
    n = 24 + 6 + 3 * 27 + 6
    n += (6 + 3 * 4) if v2 or v4 else 0
    n += (12 + 3 * 3) if v4 else 0
    T = case["T"]
    if T:
        n += 6 + 5
        n += T * (1 + 7 + 2 + (14 if k4 else 0)) + \
            (6 + 12 if (k2 or k4) else 0)
    return n


def work(case):
    kind = case["kind"]
    ms = _members(case) if kind in ("batch", "adjoint_ensemble") else [case]
    nbytes = ops = 0.0
    for c in ms:
        cl = c["nx"] * c["ny"] * c["K"]
        state = 8.0 * cl * (4 + c["T"])
        if kind in ("tendency", "vjp"):
            stages = 1
        elif kind in ("step", "host"):
            stages = c["steps"] * {"rk4": 4, "lsrk5": 5, "euler": 1}[
                c.get("stepper", "lsrk5")]
        else:
            stages = 4 * c["steps"]
        # value, value + tangent, value + gradient (its transpose costs
        # about the value's work once more, and the value is needed)
        times = {"tlm": 3, "vjp": 2, "adjoint": 2, "adjoint_ensemble": 2}
        nbytes += state * {"vjp": 4, "tlm": 3, "adjoint": 4,
                           "adjoint_ensemble": 4}.get(kind, 2)
        ops += times.get(kind, 1) * stages * cl * _ops(c)
    return {"bytes": nbytes, "flops": 2.0 * ops}


# ----------------------------------------------------------------- exact ---

def _tendency64(case, x):
    """The discrete tendency in plain torch float64."""
    m = _hex(case["nx"], case["ny"])
    v2, v4, k2, k4 = DISS[case["diss"]]
    h, vn, tr = x
    dv, area = m["dv"], m["area"]
    at = area / 2
    c0, c1 = m["coe"][:, 0], m["coe"][:, 1]
    v0, v1 = m["voe"][:, 0], m["voe"][:, 1]

    def curl(u):
        return sum(m["sv"][:, j, None] * u[m["eov"][:, j]]
                   for j in range(3)) * (DC / at)

    def div(u):
        return sum(m["sc"][:, j, None] * u[m["ce"][:, j]]
                   for j in range(6)) * (dv / area)

    def lap_edge(d, z):
        return (d[c1] - d[c0]) / DC - (z[v1] - z[v0]) / dv

    zeta = curl(vn)
    q = (zeta + F0) / (sum(h[m["cov"][:, j]] for j in range(3)) / 3)
    mh = 0.5 * (h[c0] + h[c1])
    F = mh * vn
    Q = 0.5 * (q[v0] + q[v1])
    vt = 0
    for j in range(10):
        e = m["eoe"][:, j]
        vt = vt + m["woe"][:, j, None] * F[e] * (0.5 * (Q + Q[e]))
    ke = sum((vn * vn)[m["ce"][:, j]] for j in range(6)) * \
        (dv * DC * 0.25 / area)
    vt = vt - (ke[c1] - ke[c0]) / DC - GRAV * (h[c1] - h[c0]) / DC
    if v2 or v4:
        d2u = lap_edge(div(vn), zeta)
        if v2:
            vt = vt + v2 * d2u
        if v4:
            vt = vt - v4 * lap_edge(div(d2u), curl(d2u))
    ht = -div(F)
    tts = []
    for l in range(tr.shape[0]):
        n = tr[l] / h
        t, L = 0, 0
        for j in range(6):
            e, b = m["ce"][:, j], m["nb"][:, j]
            t = t - m["sc"][:, j, None] * F[e] * (0.5 * dv / area) * (n + n[b])
            if k2 or k4:
                L = L + mh[e] * (n[b] - n) * (dv / (area * DC))
        if k2:
            t = t + k2 * L
        if k4:
            t = t - k4 * sum((L[m["nb"][:, j]] - L) for j in range(6)) * \
                (dv / (area * DC))
        tts.append(t)
    return ht, vt, torch.stack(tts) if tts else torch.zeros_like(tr)


_LSRK5 = ([0., -567301805773. / 1357537059087.,
           -2404267990393. / 2016746695238., -3550918686646. / 2091501179385.,
           -1275806237668. / 842570457699.],
          [1432997174477. / 9575080441755., 5161836677717. / 13612068292357.,
           1720146321549. / 2090206949498., 3134564353537. / 4481467310338.,
           2277821191437. / 14882151754819.])


def _step64(case, x, stepper, dt):
    def ax(a, p, q):
        return tuple(a * u + v for u, v in zip(p, q))

    if stepper == "rk4":
        k1 = _tendency64(case, x)
        k2 = _tendency64(case, ax(dt / 2, k1, x))
        k3 = _tendency64(case, ax(dt / 2, k2, x))
        k4 = _tendency64(case, ax(dt, k3, x))
        return tuple(u + dt / 6 * (a + 2 * b + 2 * c + d)
                     for u, a, b, c, d in zip(x, k1, k2, k3, k4))
    A, B = _LSRK5 if stepper == "lsrk5" else ([0.0], [1.0])
    p = tuple(torch.zeros_like(u) for u in x)
    for a, b in zip(A, B):
        p = ax(a, p, _tendency64(case, x))
        x = ax(dt * b, p, x)
    return x


def _steps64(case, x, stepper, dt):
    for _ in range(case["steps"]):
        x = _step64(case, x, stepper, dt)
    return x


def _full(ts):
    return [t.detach() for t in ts if t.numel()]


def _adjoint64(case, x, lam):
    """(x_N, dL/dx_0), one step's graph at a time."""
    xs = [x]
    with torch.no_grad():
        for _ in range(case["steps"]):
            xs.append(_step64(case, xs[-1], "rk4", DT))
    for y in reversed(xs[:-1]):
        y = tuple(t.detach().requires_grad_(True) for t in y)
        lam = torch.autograd.grad(_step64(case, y, "rk4", DT), y, lam)
    return _full(xs[-1]) + _full(lam)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "adjoint_ensemble"):
        out = []
        for i, c in enumerate(_members(case)):
            x = _inputs(c, seed, 2 + i)
            if kind == "batch":
                with torch.no_grad():
                    out += _full(_steps64(c, x, "rk4", DT))
            else:
                out += _adjoint64(c, x, _cotangent(c, seed + i))
        return out
    x = _inputs(case, seed)
    if kind == "adjoint":
        return _adjoint64(case, x, _cotangent(case, seed))
    if kind == "vjp":
        x = tuple(t.requires_grad_(True) for t in x)
        y = _tendency64(case, x)
        return _full(y) + _full(torch.autograd.grad(
            y, x, _cotangent(case, seed), allow_unused=True,
            materialize_grads=True))
    if kind == "tlm":
        _, dy = torch.func.jvp(
            lambda *a: _steps64(case, a, "rk4", DT), x,
            _cotangent(case, seed))
        return _full(dy)
    with torch.no_grad():
        if kind == "tendency":
            return _full(_tendency64(case, x))
        if kind == "host":
            return _full(_steps64(case, x, "lsrk5", DT))
        return _full(_steps64(case, x, case["stepper"], DT / 4 if
                              case["stepper"] == "euler" else DT))
