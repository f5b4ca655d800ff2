"""Performance cases of the step loop, its nudging, its ensemble and its adjoint.

Each case is work that a user of this package has it do, through the public
entry points: the Python binding (Run, Ensemble) for set-up, and the C-ABI
calls of include/lbrb.h that a program with its own buffers makes in its
loop (step, record drain, read-out of the moments).  Kinds:

  free     one run: nsteps steps, trajectory records drained, moments read;
           optionally stopped every `monitor` steps for the diagnostics
           (the evolution.dat line of the reference's loop)
  nudged   one run with bilinear temperature nudging toward a series of
           observations (a repeating series, a row per step)
  box      one run of the reference's nudging program: adiabatic walls, 7x7
           boxes around the observations, a file every `every` steps
  ensemble many runs of uneven size advanced together
  adjoint  an assimilation window: misfit and its gradient

exact() restates the model in 64-bit torch, from the lattice-Boltzmann
formulas alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import lagrangianrbnudging_b200 as lb

ST = (0.0, 0.1, 0.5, 1.0, 2.0)  # Stokes numbers of a mixed particle set (0: tracer)
OBS_ROWS = 100                  # rows of a repeating observation series


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest run in use: a test-sized domain watched closely (the
        # diagnostics every 20 steps), where launches and read-backs count
        dict(name="small_monitored_fp64", kind="free", nx=128, ny=64, ra=1e5, uff=0.1, precision="fp64",
             nprtcl=256, mixed=False, beta=0.0, full=False, every=20, nsteps=200, monitor=20),
        # the reference's CPU-runnable configuration: tracers recorded every
        # 10 steps; FP64 is what a user checks against the reference
        dict(name="plain_fp64", kind="free", nx=512, ny=256, ra=1e6, uff=0.1, precision="fp64",
             nprtcl=4096, mixed=False, beta=0.0, full=False, every=10, nsteps=500, monitor=0),
        # the same in the production precision
        dict(name="plain_fp32", kind="free", nx=512, ny=256, ra=1e6, uff=0.1, precision="fp32",
             nprtcl=4096, mixed=False, beta=0.0, full=False, every=10, nsteps=500, monitor=0),
        # production trajectories: 2^17 particles of five Stokes numbers,
        # recorded every 20 steps
        dict(name="production_fp32", kind="free", nx=4096, ny=2048, ra=1e8, uff=0.05, precision="fp32",
             nprtcl=1 << 17, mixed=True, beta=0.0, full=False, every=20, nsteps=400, monitor=0),
        # the same with the reference's own arithmetic
        dict(name="production_fp64", kind="free", nx=4096, ny=2048, ra=1e8, uff=0.05, precision="fp64",
             nprtcl=1 << 17, mixed=True, beta=0.0, full=False, every=20, nsteps=200, monitor=0),
        # a grid that fits no tile, inertial particles with the Maxey-Riley
        # terms and full records
        dict(name="ragged_inertial_fp32", kind="free", nx=1500, ny=701, ra=1e7, uff=0.1, precision="fp32",
             nprtcl=20000, mixed=True, beta=0.5, full=True, every=25, nsteps=301, monitor=0),
        # fields only, odd sizes, 64-bit: a spin-up run
        dict(name="ragged_field_fp64", kind="free", nx=1020, ny=333, ra=1e6, uff=0.1, precision="fp64",
             nprtcl=0, mixed=False, beta=0.0, full=False, every=0, nsteps=401, monitor=0),
        # nudging toward 2^14 recorded trajectories, one observation row a step
        dict(name="nudged_fp32", kind="nudged", nx=2048, ny=1024, ra=1e7, uff=0.1, precision="fp32",
             nobs=1 << 14, alpha=0.1, nsteps=300),
        # the reference's nudging program on its own grid: 1600 observations,
        # files every 20 steps
        dict(name="box_fp64", kind="box", nx=1680, ny=840, ra=1e7, uff=0.1, nobs=1600, alpha=1.0, every=20,
             nsteps=100),
        # a sweep: 64 members of three sizes, tracers in each, half nudged
        dict(name="ensemble_fp32", kind="ensemble", members=64, base=256, precision="fp32", nprtcl=1024,
             nsteps=300),
        # an assimilation window of the production precision
        dict(name="adjoint_fp32", kind="adjoint", nx=1024, ny=512, ra=1e6, uff=0.1, precision="fp32",
             nobs=4096, every=10, nsteps=400),
        # a small window in 64 bits, as a gradient check uses it
        dict(name="adjoint_small_fp64", kind="adjoint", nx=252, ny=130, ra=1e5, uff=0.1, precision="fp64",
             nobs=300, every=4, nsteps=101),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _grid(rng, a, b):
    """a grid of a..b nodes, about twice as wide as high (nx a multiple of 4)"""
    n = math.exp(rng.uniform(math.log(a), math.log(b)))
    aspect = rng.uniform(1.0, 3.0)
    ny = max(24, int(round(math.sqrt(n / aspect))))
    nx = max(32, 4 * int(round(aspect * ny / 4)))
    return nx, ny


def draw(rng):
    kind = rng.choice(["free", "free", "free", "free", "nudged", "box", "ensemble", "adjoint"])
    precision = rng.choice(["fp32", "fp64"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(8, 40), base=rng.choice([192, 224, 256]), precision=precision,
                    nprtcl=_log(rng, 64, 1024), nsteps=rng.randint(60, 240))
    nx, ny = _grid(rng, 8192, {"free": 6e6, "nudged": 3e6, "box": 2e6, "adjoint": 3e5}[kind])
    ra = 10 ** (5 + 2 * min(1.0, max(0.0, math.log10(nx * ny / 8192) / 2.5)))
    most = int(min(600, max(40, 6e8 / (nx * ny))))
    nsteps = rng.randint(max(20, most // 2), most)
    c = dict(kind=kind, nx=nx, ny=ny, ra=ra, uff=0.1)
    if kind == "free":
        n = 0 if rng.random() < 0.25 else _log(rng, 100, 1 << 17)
        full = n > 0 and rng.random() < 0.3
        c.update(precision=precision, nprtcl=n, mixed=rng.random() < 0.6, beta=rng.choice([0.0, 0.0, 0.5]),
                 full=full, every=0 if n == 0 else rng.choice([10, 20, 25, 50]), nsteps=nsteps,
                 monitor=rng.choice([0, 0, 0, 50]))
    elif kind == "nudged":
        c.update(precision=precision, nobs=min(_log(rng, 256, 1 << 14), nx * ny // 100 + 1), alpha=rng.choice([0.01, 0.1, 1.0]), nsteps=nsteps)
    elif kind == "box":
        every = rng.choice([5, 10, 20])
        c.update(nobs=_log(rng, 100, 1600), alpha=rng.choice([0.1, 1.0]), every=every,
                 nsteps=every * max(1, min(nsteps, 120) // every))
    else:
        c.update(precision=precision, nobs=_log(rng, 256, 4096), every=rng.choice([5, 10]),
                 nsteps=max(20, min(nsteps, 300)))
    return c


# ------------------------------------------------------------------ inputs
def _params(nx, ny, ra, uff):
    return lb.closure(nx, ny, Ra=ra, Pr=1.0, U=uff)


def _closure64(nx, ny, ra, uff):
    """relax, relaxg, gravity and the wall temperatures (Pr = 1): nu = kappa = U Ny / sqrt(Ra)"""
    nu = uff * ny / math.sqrt(ra)
    return 3.0 * nu + 0.5, 3.0 * nu + 0.5, -(uff * uff) / ny, -0.5, 0.5


W = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
CX = [0, 1, 0, -1, 0, 1, -1, -1, 1]
CY = [0, 0, 1, 0, -1, 1, 1, -1, -1]
OPP = [0, 3, 4, 1, 2, 7, 8, 5, 6]


def _equil(q, u, v):
    """w_k q (1 + 3 c.u + 9/2 (c.u)^2 - 3/2 u^2)"""
    usq = 1.5 * (u * u + v * v)
    out = []
    for k in range(9):
        cu = CX[k] * u + CY[k] * v
        out.append(W[k] * q * (1.0 + 3.0 * cu + 4.5 * cu * cu - usq))
    return torch.stack(out)


def _fields(nx, ny, uff, seed, noise=1e-3):
    """a convecting state: conduction profile with plume-scale waves and a
    little noise, rolls that vanish at the walls"""
    rng = np.random.default_rng(seed)
    X = (torch.arange(nx, device="cuda", dtype=torch.float64) / nx)[None, :]
    Y = ((torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5) / ny)[:, None]
    T = (0.5 - Y) + 0.0 * X
    u = torch.zeros(ny, nx, device="cuda", dtype=torch.float64)
    v = torch.zeros_like(u)
    for _ in range(4):
        m, ph, a = int(rng.integers(1, 7)), rng.uniform(0, 2 * math.pi), rng.uniform(0.03, 0.08)
        T = T + a * torch.sin(math.pi * Y) * torch.cos(2 * math.pi * m * X + ph)
        m, ph, a = int(rng.integers(1, 5)), rng.uniform(0, 2 * math.pi), rng.uniform(0.01, 0.02) * uff
        s = torch.sin(math.pi * Y)
        # stream function a ny sin^2(pi y) cos(2 pi m x + ph)
        u = u + a * 2 * math.pi * s * torch.cos(math.pi * Y) * torch.cos(2 * math.pi * m * X + ph)
        v = v + a * (ny / nx) * 2 * math.pi * m * s * s * torch.sin(2 * math.pi * m * X + ph)
    T = T + noise * torch.from_numpy(rng.uniform(-1, 1, (ny, nx))).to("cuda")
    return u, v, T


def _particles(nx, ny, uff, n, mixed, seed):
    rng = np.random.default_rng(seed + 17)
    x = rng.uniform(0.5, nx - 0.5, n)
    y = rng.uniform(1.0, ny, n)
    st = np.array(ST)[np.arange(n) * len(ST) // n] if mixed else np.zeros(n)
    ptype = (st > 0).astype(np.int32)
    invtau = np.where(st > 0, uff / (np.where(st > 0, st, 1.0) * ny), 0.0)
    return x, y, ptype, invtau


def _observations(nx, ny, nobs, rows, seed):
    """rows of positions along slow paths, and temperatures near the conduction profile"""
    rng = np.random.default_rng(seed + 29)
    x = rng.uniform(1.0, nx - 1.0, nobs)[None] + 0.02 * rng.uniform(-1, 1, nobs)[None] * np.arange(rows)[:, None]
    y = rng.uniform(2.0, ny - 1.0, nobs)[None] + 0.005 * rng.uniform(-1, 1, nobs)[None] * np.arange(rows)[:, None]
    x = np.where(x > nx, x - nx, np.where(x <= 0, x + nx, x))
    T = 0.5 - (y - 0.5) / ny + 0.05 * rng.standard_normal(nobs)[None] + 0.002 * rng.standard_normal((rows, nobs))
    return x, np.clip(y, 1.0, float(ny)), T


def _box_files(c, seed):
    """observation files, one every c['every'] steps: positions that stay
    inside the domain (between files they are interpolated in time)"""
    rng = np.random.default_rng(seed + 31)
    n, nf = c["nobs"], c["nsteps"] // c["every"] + 1
    p0 = np.stack([rng.uniform(2.0, c["nx"] - 2.0, n), rng.uniform(3.0, c["ny"] - 3.0, n)])
    p1 = p0 + rng.uniform(-0.9, 0.9, (2, n))
    files = []
    for q in range(nf):
        a = 0.5 - 0.5 * math.cos(math.pi * q / max(1, nf - 1))  # there; a repeated pass starts from p1 again
        x, y = (1 - a) * p0 + a * p1
        files.append((x, y, 0.4 - 0.8 * y / c["ny"] + 0.05 * np.sin(np.arange(n) + 0.3 * q)))
    return files


def _member_cases(c, seed):
    """the members of an ensemble: sizes base x base/2 times 1, 2 or 4, Ra
    log-uniform in [1e5, 1e7], half of them nudged (sizes from the member's
    index, so that every seed has the same work)"""
    rng = np.random.default_rng(seed + 41)
    pick = np.random.default_rng(c["members"])
    out = []
    for i in range(c["members"]):
        s = (1, 2, 4)[int(pick.integers(3))]
        out.append(dict(nx=c["base"] * s, ny=c["base"] * s // 2, ra=float(10 ** rng.uniform(5, 7)), uff=0.1,
                        alpha=0.1 if i % 2 else 0.0, seed=int(rng.integers(1 << 30))))
    return out


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _ip(a):
    return a.ctypes.data_as(C.POINTER(C.c_int))


def _pinned(*shape):
    """a program's own read-out buffer"""
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _set_state(r, nx, ny, uff, seed):
    u, v, T = _fields(nx, ny, uff, seed)
    one = torch.ones_like(u)
    f, g = _equil(one, u, v), _equil(T, u, v)
    r.set_populations(_host(f), _host(g))
    r.set_moments(_host(one), _host(u), _host(v), _host(T))
    return u, v, T


def _start_particles(r, nx, ny, uff, n, mixed, seed, u, v):
    x, y, ptype, invtau = _particles(nx, ny, uff, n, mixed, seed)
    up, vp = (_host(_bilinear(q[None], *_cells(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), nx, ny)))
              for q in (u, v))
    r.set_particles(np.arange(n, dtype=np.int32), x, y, up, vp, ptype, invtau)


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "ensemble":
        return _prepare_ensemble(c, seed)
    nx, ny = c["nx"], c["ny"]
    kw = dict(_params(nx, ny, c["ra"], c["uff"]))
    if kind == "free":
        n = c["nprtcl"]
        nrec = c["nsteps"] // c["every"] + 1 if n and c["every"] else 0
        r = lb.Run(**kw, precision=c["precision"], nprtcl=n, noutconfig=c["every"] if n else 0, record_full=c["full"],
                   record_slots=max(nrec, 1), beta=c["beta"])
        u, v, T = _set_state(r, nx, ny, c["uff"], seed)
        if n:
            _start_particles(r, nx, ny, c["uff"], n, c["mixed"], seed, u, v)
        return dict(kind=kind, run=r, nsteps=c["nsteps"], monitor=c["monitor"], n=n, fields=_pinned(4, ny, nx),
                    rec=_pinned(nrec, r.nrec, n) if nrec else None, rec_steps=np.zeros(max(nrec, 1), np.int32),
                    part=_pinned(4, n) if n else None)
    if kind == "nudged":
        r = lb.Run(**kw, precision=c["precision"], nudge="bilinear", alpha=c["alpha"], nobs=c["nobs"], obs_cycle=1)
        _set_state(r, nx, ny, c["uff"], seed)
        r.nudge_obs(1, *_observations(nx, ny, c["nobs"], OBS_ROWS, seed))
        return dict(kind=kind, run=r, nsteps=c["nsteps"], fields=_pinned(4, ny, nx))
    if kind == "box":
        r = lb.Run(**kw, precision="fp64", twall="adiabatic", nudge="refbox", alpha=c["alpha"], nobs=c["nobs"],
                   ntempread=c["every"])
        _set_state(r, nx, ny, c["uff"], seed)
        files = _box_files(c, seed)
        ids = np.arange(c["nobs"], dtype=np.int32)
        r.nudge_init(files[0][0], files[0][1], files[0][2], ids)
        return dict(kind=kind, run=r, files=files, ids=ids, every=c["every"], fields=_pinned(4, ny, nx))
    r = lb.Run(**kw, precision=c["precision"])
    steps, x, y, T, T0 = _window(c, seed)
    r.adjoint_set_obs(steps, x, y, T)
    return dict(kind=kind, run=r, T0=_host(T0), nsteps=c["nsteps"], grad=_pinned(ny, nx))


def _window(c, seed):
    _, _, T0 = _fields(c["nx"], c["ny"], c["uff"], seed, noise=1e-2)
    steps = np.arange(c["every"], c["nsteps"] + 1, c["every"], dtype=np.int32)
    x, y, T = _observations(c["nx"], c["ny"], c["nobs"], len(steps), seed)
    return steps, x, y, T, T0


def _prepare_ensemble(c, seed):
    members = []
    for m in _member_cases(c, seed):
        kw = dict(_params(m["nx"], m["ny"], m["ra"], m["uff"]), precision=c["precision"], nprtcl=c["nprtcl"])
        if m["alpha"]:
            kw.update(nudge="bilinear", alpha=m["alpha"], nobs=c["nprtcl"], obs_cycle=1)
        r = lb.Run(**kw)
        u, v, _ = _set_state(r, m["nx"], m["ny"], m["uff"], m["seed"])
        _start_particles(r, m["nx"], m["ny"], m["uff"], c["nprtcl"], False, m["seed"], u, v)
        if m["alpha"]:
            r.nudge_obs(1, *_observations(m["nx"], m["ny"], c["nprtcl"], OBS_ROWS, m["seed"]))
        members.append(r)
    ens = lb.Ensemble(members)
    return dict(kind="ensemble", ens=ens, members=members, nsteps=c["nsteps"], n=c["nprtcl"],
                fields=_pinned(4 * sum(r.nx * r.ny for r in members)), part=_pinned(len(members), 4, c["nprtcl"]))


# -------------------------------------------------------------------- pass
def _check(rc, r):
    if rc:
        raise lb.LbrbError(rc, (lb.lib().lbrb_last_error(r.h) or b"").decode())


def _moments(r, out):
    _check(lb.lib().lbrb_get_moments(r.h, _dp(out[0]), _dp(out[1]), _dp(out[2]), _dp(out[3]), lb.LAYOUT["soa"]), r)


def _positions(r, n, out):
    _check(lb.lib().lbrb_particles_get(r.h, n, None, _dp(out[0]), _dp(out[1]), _dp(out[2]), _dp(out[3]), None, None,
                                       None, None), r)


def run(state):
    s = state
    kind = s["kind"]
    if kind == "ensemble":
        s["ens"].step(s["nsteps"])
        s["ens"].sync()
        at = 0
        for i, r in enumerate(s["members"]):
            k = 4 * r.nx * r.ny
            _moments(r, s["fields"][at:at + k].reshape(4, -1))
            _positions(r, s["n"], s["part"][i])
            at += k
        return {"fields": s["fields"], "particles": s["part"]}
    r = s["run"]
    if kind == "adjoint":
        J = C.c_double()
        _check(lb.lib().lbrb_adjoint_window(r.h, _dp(s["T0"]), s["nsteps"], 100, C.byref(J), _dp(s["grad"])), r)
        return {"J": J.value, "gradient": s["grad"]}
    if kind == "box":
        for x, y, T in s["files"][1:]:
            r.nudge_load(x, y, s["ids"], T)
            r.step(s["every"])
        r.sync()
        _moments(r, s["fields"])
        return {"fields": s["fields"]}
    if kind == "nudged":
        r.step(s["nsteps"])
        r.sync()
        _moments(r, s["fields"])
        return {"fields": s["fields"]}
    out = {"fields": s["fields"]}
    if s["monitor"]:
        watch, done = [], 0
        while done < s["nsteps"]:
            k = min(s["monitor"], s["nsteps"] - done)
            r.step(k)
            done += k
            watch.append([*r.energy(), r.nusselt()])
        out["watch"] = np.array(watch)
    else:
        r.step(s["nsteps"])
    r.sync()
    if s["rec"] is not None:
        got = C.c_int()
        most = len(s["rec_steps"])
        _check(lb.lib().lbrb_record_drain(r.h, most, _ip(s["rec_steps"]), _dp(s["rec"]), None, C.byref(got)), r)
        out["records"] = s["rec"][: got.value]
        out["record_steps"] = s["rec_steps"][: got.value]
    if s["n"]:
        _positions(r, s["n"], s["part"])
        out["particles"] = s["part"]
    _moments(r, s["fields"])
    return out


# -------------------------------------------------------------------- work
FLOPS_NODE = 250        # one node update: moments, two equilibria, forcing, relaxation
FLOPS_ADJOINT = 400     # one node of the adjoint of a step


def work(case):
    """Of one pass: the state read once and written once, inputs and outputs
    once, and the arithmetic of every step."""
    c = case
    es = 4 if c.get("precision") == "fp32" else 8
    if c["kind"] == "ensemble":
        nodes = sum(m["nx"] * m["ny"] for m in _member_cases(c, 0))
        b = nodes * (2 * 19 * es + 4 * 8) + c["members"] * c["nprtcl"] * 8 * 12
        return {"bytes": b, "flops": nodes * c["nsteps"] * FLOPS_NODE}
    nodes = c["nx"] * c["ny"]
    flops = nodes * c["nsteps"] * FLOPS_NODE
    if c["kind"] == "adjoint":
        obs = c["nsteps"] // c["every"] * c["nobs"] * 24
        return {"bytes": nodes * 16 + obs, "flops": nodes * c["nsteps"] * (FLOPS_NODE + FLOPS_ADJOINT)}
    b = nodes * (2 * 19 * es + 4 * 8)
    if c["kind"] == "free" and c["nprtcl"]:
        b += c["nprtcl"] * 8 * (9 + 4 + c["nsteps"] // c["every"] * (17 if c["full"] else 9))
    elif c["kind"] == "nudged":
        b += min(c["nsteps"], OBS_ROWS) * c["nobs"] * 24
    elif c["kind"] == "box":
        b += (c["nsteps"] // c["every"] + 1) * c["nobs"] * 24
    return {"bytes": b, "flops": flops}


# ------------------------------------------------------------------- exact
def _cells(x, y, nx, ny):
    """a position's cell in the 1-based frame, corner indices wrapped, weights"""
    x1, y1 = torch.trunc(x), torch.trunc(y)
    i = [torch.remainder(x1.long() - 1 + d, nx) for d in (0, 1)]
    j = [torch.remainder(y1.long() - 1 + d, ny) for d in (0, 1)]
    wx, wy = [x1 + 1 - x, x - x1], [y1 + 1 - y, y - y1]
    return i, j, wx, wy


def _bilinear(q, i, j, wx, wy, m=None):
    """the field q[batch] at the cells (batch index m per point)"""
    b = 0 if m is None else m
    return sum(q[b, j[e], i[d]] * wx[d] * wy[e] for d in (0, 1) for e in (0, 1))


def _pull(a, k):
    """a_k streamed by one step, for the rows that have a source"""
    s = torch.roll(a[k], CX[k], -1)
    if CY[k] == 1:
        return s[..., :-1, :]
    if CY[k] == -1:
        return s[..., 1:, :]
    return s


def _with_rows(k, body, edge):
    """the streamed rows with the wall row's values put in their place"""
    return torch.cat([edge, body], -2) if CY[k] == 1 else torch.cat([body, edge], -2)


class _Model:
    """the step in 64 bits, on [9, batch, ny, nx] populations"""

    def __init__(self, nx, ny, cl, adiabatic=False):
        self.nx, self.ny, self.adiabatic = nx, ny, adiabatic
        relax, relaxg, self.gravity, self.Tup, self.Tdown = cl
        self.om, self.omg = 1.0 / relax, 1.0 / relaxg

    def stream(self, f, g):
        fs, gs = [], [None] * 9
        for k in range(9):
            b = _pull(f, k)
            if CY[k]:
                row = 0 if CY[k] == 1 else -1
                b = _with_rows(k, b, f[OPP[k]][..., row:, :][..., :1, :])
            fs.append(b)
        if self.adiabatic:
            # wall rows hold copies of the rows beside them and are not streamed into
            g = torch.cat([g[..., 1:2, :], g[..., 1:-1, :], g[..., -2:-1, :]], -2)
            for k in range(9):
                b = torch.roll(g[k], (CX[k], CY[k]), (-1, -2))
                gs[k] = torch.cat([g[k][..., :1, :], b[..., 1:-1, :], g[k][..., -1:, :]], -2)
            return fs, gs
        for k in range(9):
            gs[k] = _pull(g, k)
        full = [None] * 9
        for k in range(9):
            if not CY[k]:
                full[k] = gs[k]
                continue
            o, Tw = OPP[k], (self.Tdown if CY[k] == 1 else self.Tup)
            row = 0 if CY[k] == 1 else -1
            # the opposite population streaming into the wall row
            edge = -gs[o][..., row:, :][..., :1, :] + 2 * W[k] * Tw
            full[k] = _with_rows(k, gs[k], edge)
        return fs, full

    def step(self, f, g, F, box=None):
        """box: (mask, target, nud_term, alpha) of the box nudging"""
        fs, gs = self.stream(f, g)
        r, t = sum(fs), sum(gs)
        if box is not None:
            mask, target, nud, alpha = box
            t = t + torch.where(mask, 0.5 * nud, torch.zeros_like(nud))
        u = (fs[1] - fs[3] + fs[5] - fs[6] - fs[7] + fs[8]) / r
        v = (fs[2] - fs[4] + fs[5] + fs[6] - fs[7] - fs[8] + 0.5 * F) / r
        usq = 1.5 * (u * u + v * v)
        Q = None
        if box is not None:
            Q = torch.where(mask, alpha * (t - target), torch.zeros_like(t))
        fo, go = [], []
        for k in range(9):
            cu = CX[k] * u + CY[k] * v
            P = 1.0 + 3.0 * cu + 4.5 * cu * cu - usq
            S = (1 - 0.5 * self.om) * W[k] * F * (3.0 * (CY[k] - v) + 9.0 * cu * CY[k])
            fo.append(fs[k] + self.om * (W[k] * r * P - fs[k]) + S)
            q = gs[k] + self.omg * (W[k] * t * P - gs[k])
            if Q is not None:
                q = q - (1 - 0.5 * self.omg) * W[k] * Q
            go.append(q)
        if box is not None:
            nud = torch.where(mask, -Q, nud)
        return torch.stack(fo), torch.stack(go), -self.gravity * r * t, (r, u, v, t), (None if box is None else nud)


def _derivs(u, v, ub, vb):
    out = [u - ub, v - vb]
    for q in (u, v):
        out.append(0.5 * (torch.roll(q, -1, -1) - torch.roll(q, 1, -1)))
    for q in (u, v):
        d = 0.5 * (torch.roll(q, -1, -2) - torch.roll(q, 1, -2))
        d[..., 0, :] = q[..., 1, :] - q[..., 0, :]
        d[..., -1, :] = q[..., -1, :] - q[..., -2, :]
        out.append(d)
    return out


def _advance(p, mom, old, nx, ny, beta, m=None, need=False):
    """one step of the particles p (x, y, u, v, tracer, invtau); returns the new state and the record row"""
    r, u, v, t = mom
    x, y, pu, pv, tracer, invtau = p
    cell = _cells(x, y, nx, ny)
    fu, fv = (_bilinear(q, *cell, m) for q in (u, v))
    d = [torch.zeros_like(x)] * 6
    if need:
        d = [_bilinear(q, *cell, m) for q in _derivs(u, v, *old)]
    un = torch.where(tracer, fu, pu + beta * (d[0] + fu * d[2] + fv * d[4]) - invtau * (pu - fu))
    vn = torch.where(tracer, fv, pv + beta * (d[1] + fu * d[3] + fv * d[5]) - invtau * (pv - fv))
    xn = torch.where(tracer, x + 1.5 * fu - 0.5 * pu, x + un)
    yn = torch.where(tracer, y + 1.5 * fv - 0.5 * pv, y + vn)
    row = lambda: torch.stack([xn, yn, un, vn, x, y, pu, pv, _bilinear(t, *_cells(xn, yn, nx, ny), m),  # noqa: E731
                               *d, fu, fv])
    xw = torch.where(xn >= nx, xn - nx, torch.where(xn <= 0, xn + nx, xn))
    lo, hi = yn < 1.0, yn >= ny
    yw = torch.where(lo, 2.0 - yn, torch.where(hi, 2.0 * ny - yn, yn))
    return (xw, yw, un, torch.where(lo | hi, -vn, vn), tracer, invtau), row


def _nudge(g, t, row, alpha, nx, ny, m=None):
    """adds w_k alpha (T_obs - T) of each observation at its cell's corners"""
    x, y, T = row
    i, j, wx, wy = _cells(x, y, nx, ny)
    d = alpha * (T - _bilinear(t, i, j, wx, wy, m))
    S = torch.zeros_like(t)
    b = torch.zeros_like(i[0]) if m is None else m
    for a in (0, 1):
        for e in (0, 1):
            S.index_put_((b, j[e], i[a]), d * wx[a] * wy[e], accumulate=True)
    for k in range(9):
        g[k] += W[k] * S
    return g


def _cu(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _exact_free(c, seed):
    nx, ny, n = c["nx"], c["ny"], c["nprtcl"]
    M = _Model(nx, ny, _closure64(nx, ny, c["ra"], c["uff"]))
    u, v, T = _fields(nx, ny, c["uff"], seed)
    one = torch.ones_like(u)
    f, g = _equil(one, u, v)[:, None], _equil(T, u, v)[:, None]
    F = (-M.gravity * T)[None]
    old = (u[None], v[None])
    if n:
        px, py, ptype, invtau = _particles(nx, ny, c["uff"], n, c["mixed"], seed)
        px, py, ptype, invtau = _cu(px, py, ptype, invtau)
        cell = _cells(px, py, nx, ny)
        p = (px, py, _bilinear(old[0], *cell), _bilinear(old[1], *cell), ptype == 0, invtau)
    recs, watch = [], []
    for s in range(1, c["nsteps"] + 1):
        f, g, F, mom, _ = M.step(f, g, F)
        if n:
            rec = s % c["every"] == 0
            p, row = _advance(p, mom, old, nx, ny, c["beta"],
                              need=(c["mixed"] and c["beta"] != 0.0) or (rec and c["full"]))
            if rec:
                recs.append(row()[: 17 if c["full"] else 9].cpu())
        if c["monitor"] and (s % c["monitor"] == 0 or s == c["nsteps"]):
            r, uu, vv, t = mom
            kappa = (1.0 / M.omg - 0.5) / 3.0
            watch.append([float((0.5 * r * (uu * uu + vv * vv)).mean()), float(t.mean()),
                          1.0 + float((vv * t).mean()) * ny / (kappa * (M.Tdown - M.Tup))])
        old = mom[1:3]
    out = {"fields": torch.cat(mom).cpu()}
    if c["monitor"]:
        out["watch"] = np.array(watch)
    if n and c["every"]:
        out["records"] = torch.stack(recs) if recs else torch.zeros(0, 17 if c["full"] else 9, n)
        out["record_steps"] = None
    if n:
        out["particles"] = torch.stack(p[:4]).cpu()
    return out


def _exact_nudged(c, seed):
    nx, ny = c["nx"], c["ny"]
    M = _Model(nx, ny, _closure64(nx, ny, c["ra"], c["uff"]))
    u, v, T = _fields(nx, ny, c["uff"], seed)
    f, g = _equil(torch.ones_like(u), u, v)[:, None], _equil(T, u, v)[:, None]
    F = (-M.gravity * T)[None]
    x, y, To = _cu(*_observations(nx, ny, c["nobs"], OBS_ROWS, seed))
    for s in range(c["nsteps"]):
        f, g, F, mom, _ = M.step(f, g, F)
        q = s % OBS_ROWS
        g = _nudge(g, mom[3], (x[q], y[q], To[q]), c["alpha"], nx, ny)
    return {"fields": torch.cat(mom).cpu()}


def _exact_box(c, seed):
    nx, ny, nt, n = c["nx"], c["ny"], c["every"], c["nobs"]
    M = _Model(nx, ny, _closure64(nx, ny, c["ra"], c["uff"]), adiabatic=True)
    u, v, T = _fields(nx, ny, c["uff"], seed)
    f, g = _equil(torch.ones_like(u), u, v)[:, None], _equil(T, u, v)[:, None]
    F = (-M.gravity * T)[None]
    files = [torch.stack(_cu(*q)) for q in _box_files(c, seed)]
    nud = torch.zeros_like(F)
    d7 = torch.arange(-3, 4, device="cuda")
    d4 = torch.arange(0, 4, device="cuda")
    for s in range(1, c["nsteps"] + 1):
        q, ph = (s - 1) // nt, (s - 1) % nt + 1
        x, y, To = files[q] + (files[q + 1] - files[q]) * (ph / nt)
        xi = (torch.sign(x) * torch.floor(x.abs() + 0.5)).long()
        yi = (torch.sign(y) * torch.floor(y.abs() + 0.5)).long()
        num, cnt = torch.zeros(ny * nx, device="cuda", dtype=torch.float64), torch.zeros(ny * nx, device="cuda",
                                                                                      dtype=torch.float64)
        # the box, and its images over the periodic edge
        for cols, on in ((xi[:, None] + d7, None), (nx + xi[:, None] - d4, xi < 4), (xi[:, None] - nx + d4, xi > nx - 2)):
            i = cols[:, None, :].expand(-1, 7, -1)
            j = (yi[:, None] + d7)[:, :, None].expand(-1, -1, cols.shape[1])
            ok = (i >= 1) & (i <= nx) & (j >= 1) & (j <= ny)
            if on is not None:
                ok = ok & on[:, None, None]
            at = ((j - 1) * nx + i - 1)[ok]
            num.index_add_(0, at, To[:, None, None].expand_as(i)[ok])
            cnt.index_add_(0, at, torch.ones_like(at, dtype=torch.float64))
        mask = (cnt > 0).reshape(1, ny, nx)
        target = (num / cnt.clamp(min=1)).reshape(1, ny, nx)
        f, g, F, mom, nud = M.step(f, g, F, (mask, target, nud, c["alpha"]))
    return {"fields": torch.cat(mom).cpu()}


def _exact_ensemble(c, seed):
    cases = _member_cases(c, seed)
    fields, part = [None] * len(cases), [None] * len(cases)
    n = c["nprtcl"]
    for size in sorted({(m["nx"], m["ny"]) for m in cases}):
        ids = [i for i, m in enumerate(cases) if (m["nx"], m["ny"]) == size]
        nx, ny = size
        cl = np.array([_closure64(nx, ny, cases[i]["ra"], 0.1) for i in ids])
        M = _Model(nx, ny, tuple(torch.from_numpy(cl[:, a].copy()).cuda()[:, None, None] for a in range(2)) +
                   tuple(cl[0, 2:]))
        f, g, uu, vv, TT, P, m = [], [], [], [], [], [], []
        obs, om = [], []
        for b, i in enumerate(ids):
            u, v, T = _fields(nx, ny, 0.1, cases[i]["seed"])
            f.append(_equil(torch.ones_like(u), u, v))
            g.append(_equil(T, u, v))
            uu.append(u), vv.append(v), TT.append(T)
            px, py, ptype, invtau = _cu(*_particles(nx, ny, 0.1, n, False, cases[i]["seed"]))
            cell = _cells(px, py, nx, ny)
            P.append((px, py, _bilinear(u[None], *cell), _bilinear(v[None], *cell), ptype == 0, invtau))
            m.append(torch.full((n,), b, device="cuda"))
            if cases[i]["alpha"]:
                obs.append(_cu(*_observations(nx, ny, n, OBS_ROWS, cases[i]["seed"])))
                om.append(torch.full((n,), b, device="cuda"))
        f, g = torch.stack(f, 1), torch.stack(g, 1)
        old, F = (torch.stack(uu), torch.stack(vv)), -M.gravity * torch.stack(TT)
        p, m = tuple(torch.cat([q[a] for q in P]) for a in range(6)), torch.cat(m)
        if obs:
            obs, om = [torch.cat([o[a] for o in obs], 1) for a in range(3)], torch.cat(om)
        for s in range(c["nsteps"]):
            f, g, F, mom, _ = M.step(f, g, F)
            if len(obs):
                q = s % OBS_ROWS
                g = _nudge(g, mom[3], (obs[0][q], obs[1][q], obs[2][q]), 0.1, nx, ny, om)
            p, _ = _advance(p, mom, old, nx, ny, 0.0, m)
            old = mom[1:3]
        for b, i in enumerate(ids):
            fields[i] = torch.stack([q[b] for q in mom]).reshape(-1).cpu()
            part[i] = torch.stack([q[b * n:(b + 1) * n] for q in p[:4]]).cpu()
    return {"fields": torch.cat(fields), "particles": torch.stack(part)}


def _exact_adjoint(c, seed):
    from torch.utils.checkpoint import checkpoint

    nx, ny = c["nx"], c["ny"]
    M = _Model(nx, ny, _closure64(nx, ny, c["ra"], c["uff"]))
    steps, x, y, To, T0 = _window(c, seed)
    x, y, To = _cu(x, y, To)
    at = {int(s): q for q, s in enumerate(steps)}
    T0 = T0.clone().requires_grad_(True)

    def chunk(f, g, F, a, b):
        J = torch.zeros((), device="cuda", dtype=torch.float64)
        for s in range(a, b):
            f, g, F, mom, _ = M.step(f, g, F)
            q = at.get(s)
            if q is not None:
                J = J + (_bilinear(mom[3], *_cells(x[q], y[q], nx, ny)) - To[q]).square().sum()
        return f, g, F, J

    w = torch.tensor(W, device="cuda", dtype=torch.float64)[:, None, None, None]
    f = w * torch.ones(1, 1, ny, nx, device="cuda", dtype=torch.float64)
    g, F, J = w * T0[None, None], (-M.gravity * T0)[None], 0.0
    for a in range(1, c["nsteps"] + 1, 10):
        f, g, F, Jc = checkpoint(chunk, f, g, F, a, min(a + 10, c["nsteps"] + 1), use_reentrant=False)
        J = J + Jc
    grad, = torch.autograd.grad(J, T0)
    return {"J": float(J), "gradient": grad.cpu()}


def exact(case, seed):
    return {"free": _exact_free, "nudged": _exact_nudged, "box": _exact_box, "ensemble": _exact_ensemble,
            "adjoint": _exact_adjoint}[case["kind"]](case, seed)
