"""The work users have this framework do, as timed cases.

A case is one segment of a cylinder-flow run through the public Python layer (`Simulation`, `Batch`): the
handle, its tuned launch shape and its pinned read-back buffers are made beforehand, a pass advances the
flow by `steps` time steps and hands back what the segment is run for (force history, fields, restart
state, surface records, gradient).  Sizes are the package's own configurations (config.py, the tests, the
benchmark) and ragged neighbours of them.

`exact` repeats a segment from its start in FP64 with plain torch operations: lattice, curved-wall
geometry and closures are written out here from the method, nothing of the package is used.
"""
import math

import numpy as np
import torch

# ---- the cases ------------------------------------------------------------------------------------

RUN = dict(kind="run", walls="freeslip", tuned=True)


def listed():
    return [
        # the smallest calls: a host program that keeps its own time loop, one step per call, on the
        # tests' 80 x 50 lattice with the reference's default (y-periodic) walls
        dict(RUN, name="host_loop_80x50_f64", kind="loop", nx=80, ny=50, D=10, Re=100.0, U=0.05, precision=64, steps=32,
             walls="periodic", tuned=False),
        # the validation case, as a driver runs it: default handle, the force history and final fields
        dict(RUN, name="small_400x100_f64", nx=400, ny=100, D=20, Re=100.0, U=0.05, precision=64, steps=400, tuned=False),
        # the same in the fast precision, tuned for a long run
        dict(RUN, name="small_400x100_f32", nx=400, ny=100, D=20, Re=100.0, U=0.05, precision=32, steps=400),
        # a ragged no-slip channel: odd sizes, reference walls
        dict(RUN, name="noslip_1003x251_f64", nx=1003, ny=251, D=40, Re=150.0, U=0.05, precision=64, steps=300, walls="noslip"),
        # the benchmark case in both precisions
        dict(RUN, name="mid_2048x512_f64", nx=2048, ny=512, D=80, Re=200.0, U=0.04, precision=64, steps=400),
        dict(RUN, name="mid_2048x512_f32", nx=2048, ny=512, D=80, Re=200.0, U=0.04, precision=32, steps=400),
        # field statistics over a window (mean and rms of u, v, p)
        dict(RUN, name="fields_2048x512_f32", kind="fields", nx=2048, ny=512, D=80, Re=200.0, U=0.04, precision=32, steps=300),
        # production-size states far above the L2
        dict(RUN, name="large_4099x1023_f64", nx=4099, ny=1023, D=128, Re=500.0, U=0.04, precision=64, steps=300),
        dict(RUN, name="large_8192x2048_f32", nx=8192, ny=2048, D=128, Re=500.0, U=0.04, precision=32, steps=400),
        # the 64-case parameter sweep as one batch
        dict(name="sweep_64_f32", kind="sweep", cases=64, nx_lo=256, nx_hi=1024, precision=32, steps=300),
        # gradient of mean drag (body force and inlet profile)
        dict(name="adjoint_512x128_f64", kind="adjoint", nx=512, ny=128, D=32, Re=100.0, U=0.05, precision=64, steps=400, walls="freeslip"),
        # restart segment with surface records: state up, steps with wall pressure and probes, state down
        dict(RUN, name="restart_surface_800x200_f64", kind="restart", nx=800, ny=200, D=40, Re=100.0, U=0.05, precision=64, steps=150),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "run", "run", "run", "run", "run", "run", "fields", "sweep", "adjoint", "restart"])
    prec = rng.choice([64, 32])
    if kind == "sweep":
        lo = 32 * rng.randint(8, 16)
        return dict(kind=kind, cases=_log(rng, 4, 64), nx_lo=lo, nx_hi=lo + 32 * rng.randint(0, 16), precision=prec,
                    steps=_log(rng, 100, 300))
    top = {"loop": 400, "run": 5800 if prec == 64 else 8192, "fields": 2048, "adjoint": 640, "restart": 2048}[kind]
    nx = _log(rng, 80, top)
    ny = max(50, int(nx * rng.uniform(0.2, 0.34)))
    D = 2 * max(5, int(ny / rng.uniform(8.0, 13.0)))
    steps = {"loop": rng.randint(16, 48), "run": _log(rng, 100, 500), "fields": _log(rng, 100, 300),
             "adjoint": _log(rng, 100, 400), "restart": _log(rng, 50, 300)}[kind]
    while nx * ny * steps > 4.0e9:
        steps //= 2
    return dict(kind=kind, nx=nx, ny=ny, D=D, Re=round(rng.uniform(40.0, 150.0), 2), U=round(rng.uniform(0.03, 0.06), 4),
                precision=prec, steps=steps, tuned=kind != "loop" and rng.random() < 0.7,
                walls="freeslip" if kind == "adjoint" else rng.choice(["freeslip", "freeslip", "noslip", "periodic"]))


# ---- one case's flow parameters --------------------------------------------------------------------


def _centre(case):
    """Cylinder centre: an integer column a fifth into the channel, a half-integer row at mid height."""
    return float(max(case["D"] + 12, round(case["nx"] / 5))), case["ny"] // 2 + 0.5


def _flows(case, seed):
    """(nx, ny, D, xc, yc, Re, U, walls, noise seed) of each lattice of a case."""
    if case["kind"] != "sweep":
        return [(case["nx"], case["ny"], float(case["D"]), *_centre(case), case["Re"], case["U"], case["walls"], seed)]
    rng, out = np.random.default_rng(4242), []                       # the lattices are the case's, the noise the seed's
    for c in range(case["cases"]):
        nx = int(rng.integers(case["nx_lo"] // 32, case["nx_hi"] // 32 + 1)) * 32
        ny = nx // 4
        out.append((nx, ny, ny / 5.0, nx / 5.0, ny / 2.0 + 0.5, float(rng.uniform(50.0, 200.0)), 0.05, "freeslip", seed * 1000 + c))
    return out


def _every(case):
    """Checkpoint interval of an adjoint case: about the square root of its steps, as a user picks it."""
    return max(5, int(math.sqrt(case["steps"])) * 2)


def _force(case, seed):
    """The body force an adjoint case is differentiated at: weak, another value at every node."""
    return 1e-7 * np.random.default_rng(seed).standard_normal((2, case["nx"], case["ny"]))


def _config(flow):
    from mrlbm_2d_b200 import config
    nx, ny, D, xc, yc, Re, U, walls, seed = flow
    c = config.cylinder_case(nx, ny, D, xc, yc, Re, U, seed=seed)
    if walls != "freeslip":
        c = c.replace(wall_mode=config.WALL_REFERENCE, y_periodic=1 if walls == "periodic" else 0)
    return c


# ---- prepare and run --------------------------------------------------------------------------------


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    import mrlbm_2d_b200 as m
    cfgs = [_config(f) for f in _flows(case, seed)]
    nodes = sum(c.nx * c.ny for c in cfgs)
    st = {"case": dict(case), "out": [_pinned(nodes) for _ in range(3)] if case["kind"] in ("loop", "run", "sweep") else None}
    if case["kind"] == "sweep":
        st["sim"] = m.Batch(cfgs, precision=case["precision"])
        st["sim"].autotune(trial_steps=50)
        at = np.cumsum([0] + [c.nx * c.ny for c in cfgs])
        st["views"] = [[o[a:b] for o in st["out"]] for a, b in zip(at[:-1], at[1:])]
        return st
    sim = st["sim"] = m.Simulation(cfgs[0], precision=case["precision"])
    if case["kind"] == "restart":
        f = sim.get_state()
        st["f"], st["f_out"] = _pinned(9 * nodes), _pinned(9 * nodes)
        st["f"][:] = f.transpose(2, 1, 0).ravel()
        sim.surface_enable()
    if case["kind"] == "fields":
        sim.field_stats_window(2, 1 << 30)
    if case["kind"] == "adjoint":
        sim.set_body_force(_force(case, seed))
    if case.get("tuned"):
        sim.autotune(trial_steps=20)
    return st


def run(state):
    case, sim = state["case"], state["sim"]
    kind, steps = case["kind"], case["steps"]
    if kind == "loop":
        for _ in range(steps - 1):
            sim.step(1)
        sim.step(1, macro=True)
        return [sim.forces(), sim.macro(out=state["out"])]
    if kind == "run":
        sim.step(steps, macro=True)
        return [sim.forces(), sim.macro(out=state["out"])]
    if kind == "fields":
        sim.field_stats_window(sim.iter + 1, sim.iter + steps)
        sim.step(steps)
        return [sim.forces(), sim.field_stats()]
    if kind == "restart":
        sim.load_state(state["f"], iter=1)
        sim.step(steps)
        return [sim.forces(), sim.surface(cap=steps), sim.get_state(out=state["f_out"])]
    if kind == "adjoint":
        return list(sim.adjoint_drag(steps, steps // 3, _every(case)))
    sim.step(steps, macro=True)
    for c, v in zip(sim.cases, state["views"]):
        c.macro(out=v)
    return [[np.stack(a) for a in zip(*(c.forces(cap=steps) for c in sim.cases))], state["out"]]


def work(case):
    """The state read and written once a pass, the outputs written once, and the arithmetic of every node's
    steps (about 150 operations: nine-population sums, collision, reconstruction); an adjoint adds
    one recomputed step and one reverse step of about twice that for each."""
    nodes = float(sum(f[0] * f[1] for f in _flows(case, 1)))
    size = case["precision"] // 8
    flops = 150.0 * nodes * case["steps"]
    outs = {"adjoint": 16, "fields": 48, "restart": 144}.get(case["kind"], 24) * nodes
    if case["kind"] == "adjoint":
        flops *= 4
    return {"bytes": 18.0 * size * nodes + outs + 32.0 * case["steps"], "flops": flops}


# ---- the same segments in plain FP64 ------------------------------------------------------------------
# Populations are flat, (9, M) over the M nodes of every lattice of a case; streaming is one gather.

EX, EY = [0, 1, 0, -1, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1]
MIRROR = [0, 1, 4, 3, 2, 8, 7, 6, 5]
W = [float(np.float32(a) / np.float32(36)) for a in (16, 4, 4, 4, 4, 1, 1, 1, 1)]       # single-precision weights
CS2 = 1.0 / 3.0
# incoming and outgoing populations by quadrant label
INCS = {1: "110010001", 2: "100110010", 3: "110110011", 4: "111001000", 5: "111011001", 7: "111111011", 8: "101100100",
        10: "101110110", 11: "111110111", 12: "111101100", 13: "111111101", 14: "111111110", 15: "111111111"}
OUTS = {1: "101100100", 2: "111001000", 3: "111101100", 4: "100110010", 5: "101110110", 7: "111111110", 8: "110010001",
        10: "111011001", 11: "111111101", 12: "110110011", 13: "111110111", 14: "111111011", 15: "111111111"}


def _lattice(flow):
    """Index tables of one lattice (0-based flat nodes j * nx + i) and its curved-wall tables."""
    nx, ny, D, xc, yc, Re, U, walls, _ = flow
    r, N = D / 2.0, nx * ny
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    src, stale = np.empty((9, N), np.int64), np.zeros((9, N), bool)
    for k in range(9):
        si, sj, sk = i - EX[k], j - EY[k], np.full_like(i, k)
        hit = (j == ny - 1) & (EY[k] < 0) | (j == 0) & (EY[k] > 0)
        if walls == "freeslip":
            sj, sk = np.where(hit, j, sj), np.where(hit, MIRROR[k], sk)
        elif walls == "periodic":
            si, sj = np.where(hit, i, si), np.where(hit, (ny - 1) - j, sj)
        out = (si < 0) | (si >= nx) | (sj < 0) | (sj >= ny)
        src[k] = np.where(out, k * N + j * nx + i, sk * N + sj * nx + si).ravel()
        stale[k] = out.ravel()
    # node classes: wall ring, solid core, and solid neighbours of fluid moved to the wall
    d = np.sqrt((i + 1 - xc) ** 2 + (j + 1 - yc) ** 2)
    cls = np.where(np.abs(d - r) <= 0.5, 2, np.where(d <= r, 1, 0))
    fluid = cls == 0
    near = np.zeros_like(fluid)
    inner = np.zeros_like(fluid)
    inner[1:-1, 1:-1] = fluid[1:-1, 1:-1]
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            near |= np.roll(inner, (a, b), (0, 1))
    cls[(cls == 1) & near] = 2
    bi, bj = (v + 1 for v in np.nonzero((cls == 2).T))                                   # column by column
    F = np.pad(fluid, 1)
    at = lambda a, b: F[bj + b, bi + a].astype(int)  # noqa: E731
    label = ((at(-1, 0) | at(-1, 1) | at(0, 1)) + 2 * (at(1, 0) | at(1, 1) | at(0, 1)) + 4 * (at(-1, 0) | at(-1, -1) | at(0, -1))
             + 8 * (at(1, 0) | at(1, -1) | at(0, -1)))
    bits = lambda t: np.array([[c == "1" for c in t[q]] for q in label]).T  # noqa: E731
    rr = np.sqrt((bi - xc) ** 2 + (bj - yc) ** 2)
    rcyl, dx = rr.max(), math.sqrt(2.0)
    n1, n2 = (bi - xc) / rr, (bj - yc) / rr
    xr, yr = [xc + (rcyl + q * dx) * n1 for q in range(4)], [yc + (rcyl + q * dx) * n2 for q in range(4)]
    delta = np.sqrt((bi - xr[0]) ** 2 + (bj - yr[0]) ** 2)
    theta = np.arctan2(yr[0] - yc, xr[0] - xc)
    theta = np.where(theta < 0, theta + 2 * math.pi, theta)

    def rot(a, b):
        q = np.sqrt((a - xc) ** 2 + (b - yc) ** 2)
        return (a - xc) / q, (b - yc) / q

    sten, sc, ss, xd, yd = [], [], [], [], []
    for q in (1, 2, 3):
        fx, fy = np.floor(xr[q]), np.floor(yr[q])
        xd.append(xr[q] - fx)
        yd.append(yr[q] - fy)
        for a, b in ((0, 0), (1, 0), (0, 1), (1, 1)):
            sten.append(((fy + b - 1) * nx + fx + a - 1).astype(np.int64))
            c, s = rot(fx + a, fy + b)
            sc.append(c)
            ss.append(s)
    c, s = rot(bi, bj)
    own = (bj - 1) * nx + bi - 1
    col = np.arange(ny) * nx
    probe = [(int(math.floor(yc)) * nx + int(math.floor(xc + (1.0 + 0.5 * k) * D + 0.5)) - 1) for k in range(4)]
    order = np.argsort(theta, kind="stable")
    return dict(N=N, nb=len(bi), ny=ny, omega=1.0 / (3.0 * (U * D / Re) + 0.5), U=U, src=src, stale=stale, own=own, Is=bits(INCS), Os=bits(OUTS),
                sten=np.array(sten), sc=np.array(sc), ss=np.array(ss), xd=np.array(xd), yd=np.array(yd), c=c, s=s,
                t2=delta * (delta - 2 * dx) / dx ** 2, t3=delta * (delta - dx) / (2 * dx ** 2), inlet=col, outlet=col + nx - 1,
                top=np.arange(nx) + (ny - 1) * nx if walls == "noslip" else np.zeros(0, np.int64),
                bottom=np.arange(nx) if walls == "noslip" else np.zeros(0, np.int64), probe=probe, order=order, theta=theta,
                rad=np.array([np.sqrt((xr[q] - xc) ** 2 + (yr[q] - yc) ** 2) for q in (1, 2, 3, 0)]))


def _join(lats, dev):
    """The lattices of a case side by side in one flat index space."""
    M = sum(q["N"] for q in lats)
    t = {}
    base = np.cumsum([0] + [q["N"] for q in lats])
    for key in ("own", "sten", "inlet", "outlet", "top", "bottom"):
        t[key] = np.concatenate([q[key] + b for q, b in zip(lats, base)], axis=-1)
    for key in ("Is", "Os", "sc", "ss", "xd", "yd", "c", "s", "t2", "t3", "stale"):
        t[key] = np.concatenate([q[key] for q in lats], axis=-1)
    t["src"] = np.concatenate([(q["src"] // q["N"]) * M + q["src"] % q["N"] + b for q, b in zip(lats, base)], axis=-1)
    t["omega"] = np.concatenate([np.full(q["N"], q["omega"]) for q in lats])
    t["U"] = np.concatenate([np.full(q["ny"], q["U"]) for q in lats])
    t["wall_of"] = np.repeat(np.arange(len(lats)), [q["nb"] for q in lats])
    t["row_of"] = np.repeat(np.arange(len(lats)), [q["ny"] for q in lats])
    t = {k: torch.as_tensor(np.ascontiguousarray(v), device=dev) for k, v in t.items()}
    for k in ("Is", "Os"):
        t[k] = t[k].double()
    t["n"] = len(lats)
    return t


def _noise(seed, n, dev):
    """Two standard normals per node: Box-Muller on SplitMix64 draws (int64 arithmetic wraps as uint64 does)."""
    def i64(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    def shr(z, b):
        return (z >> b) & ((1 << (64 - b)) - 1)

    def mix(z):
        z = z + i64(0x9E3779B97F4A7C15)
        z = (z ^ shr(z, 30)) * i64(0xBF58476D1CE4E5B9)
        z = (z ^ shr(z, 27)) * i64(0x94D049BB133111EB)
        return z ^ shr(z, 31)

    def unit(counter):
        return (shr(mix(mix(counter) ^ seed), 11).double() + 0.5) / 2.0 ** 53

    at = 4 * torch.arange(n, device=dev, dtype=torch.int64)
    return [torch.sqrt(-2.0 * torch.log(unit(at + 2 * c))) * torch.cos(2.0 * math.pi * unit(at + 2 * c + 1)) for c in (0, 1)]


def _equilibrium(u, v):
    return torch.stack([W[k] * (1.0 + 3.0 * (EX[k] * u + EY[k] * v) + 4.5 * u * u * (EX[k] ** 2 - CS2) + 4.5 * v * v * (EY[k] ** 2 - CS2)
                                + 9.0 * u * v * (EX[k] * EY[k])) for k in range(9)])


def _moments(f):
    rho = f.sum(0)
    inv = 1.0 / rho
    d = (f[5] + f[6]) + (f[7] + f[8])
    return (rho, (f[1] - f[3] + f[5] - f[6] - f[7] + f[8]) * inv, (f[2] - f[4] + f[5] + f[6] - f[7] - f[8]) * inv,
            (f[1] + f[3] + d) * inv - CS2, (f[2] + f[4] + d) * inv - CS2, (f[5] - f[6] + f[7] - f[8]) * inv)


def _incoming(f, ks):
    """Sums over the incoming populations: density, density times Hxx, Hyy and Hxy."""
    q = f[ks]
    w = lambda v: (torch.as_tensor(v, dtype=torch.float64, device=f.device)[:, None] * q).sum(0)  # noqa: E731
    return q.sum(0), w([EX[k] ** 2 - CS2 for k in ks]), w([EY[k] ** 2 - CS2 for k in ks]), w([float(EX[k] * EY[k]) for k in ks])


def _closed(t, f, uin):
    """Macroscopic values after the boundary conditions, of populations f."""
    m = _moments(f)
    rho, ux, uy, mxx, myy, mxy = m
    om = t["omega"]

    def put(at, vals):
        return [a if v is None else a.index_put((at,), v) for a, v in zip((rho, ux, uy, mxx, myy, mxy), vals)]

    # outlet: density and velocity of the neighbouring column, regularized moments
    at = t["outlet"]
    r, u, v = rho[at - 1], ux[at - 1], uy[at - 1]
    _, xx, yy, xy = _incoming(f[:, at], [0, 1, 2, 4, 5, 8])
    rows = put(at, (r, u, v, (r + 9 * xx - 3 * r * u) / (6 * r), 6 * yy / (5 * r), (6 * xy - r * v) / (3 * r)))
    rho, ux, uy, mxx, myy, mxy = rows
    at, u = t["inlet"], uin
    rI, xx, yy, xy = _incoming(f[:, at], [0, 2, 3, 4, 6, 7])
    r = (4 * rI + 3 * xx) / (3 - 3 * u)
    rho, ux, uy, mxx, myy, mxy = put(at, (r, u, torch.zeros_like(u), (r + 9 * xx + 3 * r * u) / (6 * r), 6 * yy / (5 * r), 2 * xy / r))
    for at, ks in ((t["top"], [0, 1, 2, 3, 5, 6]), (t["bottom"], [0, 1, 3, 4, 7, 8])):
        if len(at):
            rI, xx, yy, xy = _incoming(f[:, at], ks)
            r = 3 * (4 * rI + 3 * (1 - om[at]) * yy) / (9 + om[at])
            z = torch.zeros_like(r)
            rho, ux, uy, mxx, myy, mxy = put(at, (r, z, z, 6 * xx / (5 * r), (r + 9 * yy) / (6 * r), 2 * xy / r))
    # curved wall: velocity and rotated normal moments extrapolated from two points along the normal, then
    # the strong rotated closure for density and shear moment
    st = t["sten"][:8]
    _, u, v, xx, yy, xy = (q[st] for q in m)
    cc, ss, s2 = t["sc"][:8] ** 2, t["ss"][:8] ** 2, 2 * t["sc"][:8] * t["ss"][:8]

    def wall(q):
        p = []
        for a in (0, 1):
            x, y, b = t["xd"][a], t["yd"][a], 4 * a
            p.append((1 - y) * ((1 - x) * q[b] + x * q[b + 1]) + y * ((1 - x) * q[b + 2] + x * q[b + 3]))
        return t["t2"] * p[0] - t["t3"] * p[1]

    wu, wv, X, Y = wall(u), wall(v), wall(xx * cc + yy * ss + xy * s2), wall(xx * ss + yy * cc - xy * s2)
    c, s, o = t["c"], t["s"], om[t["own"]]
    s2, c2 = 2 * s * c, c * c - s * s
    up, vp = wu * c + wv * s, wv * c - wu * s
    fw = f[:, t["own"]]
    zero = torch.zeros_like(c)
    A, E, B11, B22, B12, rI, mI, Dxy, F11, F22, F12 = [zero] * 11
    for k in range(9):
        hx, hy, hz = EX[k] ** 2 - CS2, EY[k] ** 2 - CS2, float(EX[k] * EY[k])
        cx, cy = EX[k] * c + EY[k] * s, EY[k] * c - EX[k] * s
        hxx, hyy = hx * c * c + hy * s * s + hz * s2, hx * s * s + hy * c * c - hz * s2
        hxy = (hy - hx) * 0.5 * s2 + hz * c2
        a = W[k] * (1 + 3 * up * cx + 3 * vp * cy)
        e = a + W[k] * (4.5 * up * up * hxx + 4.5 * vp * vp * hyy + 9 * up * vp * hxy)
        I, O, b = t["Is"][k], t["Os"][k], 4.5 * W[k]
        A, E, B11, B22, B12 = A + O * a, E + O * e, B11 + O * b * hxx, B22 + O * b * hyy, B12 + O * b * hxy
        rI, mI, Dxy = rI + I * fw[k], mI + I * fw[k] * hxy, Dxy + I * a * hxy
        F11, F22, F12 = F11 + I * b * hxx * hxy, F22 + I * b * hyy * hxy, F12 + I * b * hxy * hxy
    mI, G = mI / rI, (1 - o) * A + o * E
    L11, L22, L12 = (1 - o) * B11 * mI - F11, (1 - o) * B22 * mI - F22, 2 * ((1 - o) * B12 * mI - F12)
    Z = (Dxy - G * mI - X * L11 - Y * L22) / L12
    r = rI / (G + (1 - o) * (X * B11 + Y * B22 + 2 * Z * B12))
    return put(t["own"], (r, wu, wv, X * c * c + Y * s * s - Z * s2, X * s * s + Y * c * c + Z * s2, (X - Y) * 0.5 * s2 + Z * c2))


def _step(t, f, uin, body=None):
    """One time step: (next populations, macroscopic values, drag, lift and inlet density sum per lattice)."""
    mac = _closed(t, f, uin)
    rho, ux, uy, mxx, myy, mxy = mac
    om = t["omega"]
    xx, yy, xy = (1 - om) * mxx + om * ux * ux, (1 - om) * myy + om * uy * uy, (1 - om) * mxy + om * ux * uy
    fo = torch.stack([W[k] * rho * (1 + 3 * (EX[k] * ux + EY[k] * uy) + 4.5 * xx * (EX[k] ** 2 - CS2) + 4.5 * yy * (EY[k] ** 2 - CS2)
                                    + 9 * xy * (EX[k] * EY[k])) for k in range(9)])
    fw, gw = f[:, t["own"]], fo[:, t["own"]]
    fx = sum(EX[k] * (t["Is"][k] * fw[k] - t["Os"][k] * gw[k]) for k in range(9))
    fy = sum(EY[k] * (t["Is"][k] * fw[k] - t["Os"][k] * gw[k]) for k in range(9))
    per = lambda v, of: torch.zeros(t["n"], dtype=torch.float64, device=f.device).index_add(0, of, v)  # noqa: E731
    rec = [per(fx, t["wall_of"]), per(fy, t["wall_of"]), per(rho[t["inlet"]], t["row_of"])]
    if body is not None:                                             # momentum source, not at curved-wall nodes
        b = body * t["bulk"]
        fo = fo + torch.stack([3 * W[k] * (EX[k] * b[0] + EY[k] * b[1]) for k in range(9)])
    return torch.where(t["stale"], f, fo.reshape(-1)[t["src"]]), mac, rec


def _surface(t, lat, f):
    """Wall pressure in angular order, its Gaussian smoothing, and the probes, from populations f."""
    rho, ux, uy, *_ = _moments(f)
    p, q = rho[t["sten"]] * CS2, []
    for a in range(3):
        x, y, b = t["xd"][a], t["yd"][a], 4 * a
        q.append((1 - y) * ((1 - x) * p[b] + x * p[b + 1]) + y * ((1 - x) * p[b + 2] + x * p[b + 3]))
    r1, r2, r3, rs = t["rad"]
    ps = (q[0] * (rs - r2) * (rs - r3) / ((r1 - r2) * (r1 - r3)) + q[1] * (rs - r1) * (rs - r3) / ((r2 - r1) * (r2 - r3))
          + q[2] * (rs - r1) * (rs - r2) / ((r3 - r1) * (r3 - r2)))[t["order"]]
    at = t["probe"]
    return ps, t["gauss"] @ ps, torch.cat([rho[at], ux[at], uy[at]]) / 3.0


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    flows = _flows(case, seed)
    lats = [_lattice(f) for f in flows]
    t = _join(lats, dev)
    start = []
    for flow, lat in zip(flows, lats):
        a, b = _noise(flow[8], lat["N"], dev)
        start.append(_equilibrium(flow[6] + 1e-4 * flow[6] * a, 1e-4 * flow[6] * b))
    f = torch.cat(start, 1)
    steps, kind = case["steps"], case["kind"]
    if kind == "adjoint":
        return _gradient(t, lats[0], case, f, _force(case, seed))
    if kind == "restart":
        th = torch.as_tensor(lats[0]["theta"][lats[0]["order"]], device=dev)
        g = torch.exp(-(th[:, None] - th[None, :]) ** 2 / (2 * 0.1 ** 2))
        t.update(rad=torch.as_tensor(lats[0]["rad"], device=dev), order=torch.as_tensor(lats[0]["order"], device=dev),
                 probe=torch.as_tensor(lats[0]["probe"], device=dev), gauss=g / g.sum(1, keepdim=True))
    recs, surf, sums = [], [], 0.0
    for _ in range(steps):
        if kind == "restart":
            surf.append(_surface(t, lats[0], f))
        f, mac, rec = _step(t, f, t["U"])
        recs.append(torch.stack(rec))
        if kind == "fields":
            q = torch.stack([mac[1], mac[2], mac[0] * CS2])
            sums = sums + torch.stack([q, q * q])
    iters = np.arange(2, steps + 2, dtype=np.int32)
    r = torch.stack(recs).cpu().numpy()                                # (steps, 3, lattices)
    forces = [iters, r[:, 0, 0], r[:, 1, 0], r[:, 2, 0]]
    if kind in ("loop", "run"):
        return [forces, [q.cpu().numpy() for q in mac[:3]]]
    if kind == "sweep":
        return [[np.stack([iters] * t["n"]), *(r[:, c].T.copy() for c in range(3))], [q.cpu().numpy() for q in mac[:3]]]
    if kind == "restart":
        return [forces, [iters, *(torch.stack([s[q] for s in surf]).cpu().numpy() for q in range(3))], f.cpu().numpy().ravel()]
    mean, sq = (sums / steps).cpu()
    rms = torch.sqrt(torch.clamp(sq - mean * mean, min=0.0))
    nx, ny = case["nx"], case["ny"]
    named = {a + b: v[c].reshape(ny, nx).T.numpy() for a, v in (("mean_", mean), ("rms_", rms)) for c, b in enumerate("uvp")}
    # the rms of a window whose fluctuations are far below its mean is a difference of nearly equal sums
    # with no digits to hold a value to
    return [forces, dict({k: None if k.startswith("rms") else v for k, v in named.items()}, n=steps)]


def _gradient(t, lat, case, f, force):
    """Mean drag over the last third of the steps and its gradient, by torch's autograd."""
    from torch.utils.checkpoint import checkpoint
    nx, ny, steps, window = case["nx"], case["ny"], case["steps"], case["steps"] // 3
    bulk = torch.ones(lat["N"], dtype=torch.float64, device=f.device)
    bulk[t["own"]] = 0.0
    t["bulk"] = bulk
    body = torch.as_tensor(force.transpose(0, 2, 1).reshape(2, -1).copy(), device=f.device).requires_grad_(True)
    uin = t["U"].clone().requires_grad_(True)

    def segment(f, body, uin, a, b):
        J = 0.0
        for n in range(a, b):
            f, _, rec = _step(t, f, uin, body)
            if n >= steps - window:
                J = J + rec[0][0] / window
        return f, J + 0.0 * uin[0]

    J = 0.0
    for a in range(0, steps, 20):
        f, part = checkpoint(segment, f, body, uin, a, min(a + 20, steps), use_reentrant=False)
        J = J + part
    gb, gu = torch.autograd.grad(J, (body, uin))
    return [float(J.detach()), gb.reshape(2, ny, nx).transpose(1, 2).cpu().numpy(), gu.cpu().numpy()]
