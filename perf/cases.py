"""Timed cases of the level-set transport path, through the package's public
entry points.

A pass takes an initial level set from host memory through a number of time
steps (wall ghost fill, CFL step, RK3 WENO5 convection, reinitialisation,
volume sums) and reads the result back, as a program does that transports a
level set between two outputs.  Every pass starts from the same initial
level set, so it can be repeated.  Grids are boxes with spheres carried by
Taylor-Green modes (the ensemble and serving workloads), or wave tanks.

kinds
  run     one LevelSet: upload, r3d_ls_run, download
  dropin  one step of REEF3D's time loop: the four fields come from host
          arrays in REEF3D's layout, one step, the level set goes back
  tank    a numerical wave tank: relaxation-zone targets and one step at a
          time, density and viscosity read back with the level set
  batch   an ensemble advanced together
`stretch` is the amplitude of the grid's stretching, 0 for uniform spacing;
`tune`: the program calls the autotuner once, as a long run does.
"""
import math

import numpy as np
import torch

import reef3d_b200 as r3d

BASE = dict(kind="run", form="f32", nx=64, ny=64, nz=64, steps=10, f44=2, f49=1, stretch=0.0, airy=False,
            period=0.0, fluid=False, tune=False, members=1)
DEPTH, AMP, WAVELENGTH = 0.5, 0.05, 2.0
WATER = (998.2, 1.004e-6, 1.205, 1.41e-5)


def _case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    return [
        # the smallest call: one step of a drop-in loop on a coarse box; copies and launches count
        _case("dropin_40_f64", kind="dropin", form="f64", nx=40, ny=36, nz=32, steps=1),
        # a drop-in step of an ordinary grid in the FP32 form
        _case("dropin_128_f32", kind="dropin", nx=128, ny=128, nz=128, steps=1),
        # a 2D verification run (the slotted disc's grid): kernels of a few microseconds
        _case("plane_128_f64", form="f64", nx=128, ny=1, nz=128, steps=60),
        # a 2D flume, REEF3D's everyday use: stretched in z, relaxation zones, fluid update
        _case("flume_2d_f64", kind="tank", form="f64", nx=600, ny=1, nz=75, steps=10, f44=3, stretch=0.3),
        # a small box, run between two outputs
        _case("box_64_f32", steps=50),
        # odd sizes, unequal spacings, the cells at the interface frozen (F49 0), the default F44 3
        _case("ragged_f32", nx=201, ny=97, nz=153, steps=20, f44=3, f49=0),
        # a stretched grid: node tables instead of uniform constants
        _case("stretched_f32", nx=160, ny=128, nz=96, steps=10, stretch=0.3),
        _case("stretched_f64", form="f64", nx=96, ny=80, nz=112, steps=5, stretch=0.3, fluid=True),
        # the benchmark grid in both forms, velocity reversing with the clock
        _case("vortex_256_f32", nx=256, ny=256, nz=256, steps=30, period=3.0, tune=True),
        _case("vortex_256_f64", form="f64", nx=256, ny=256, nz=256, steps=4, period=3.0),
        # the largest: the wave tank with its velocity regenerated before every step
        _case("airy_tank_f32", nx=1024, ny=128, nz=256, steps=20, f44=1, airy=True),
        # an ensemble of uneven 2D and 3D members
        _case("ensemble_f32", kind="batch", nx=160, ny=160, nz=160, steps=20, members=16),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "dropin", "tank", "batch"])
    c = dict(BASE, kind=kind, f44=rng.choice([1, 2, 2, 3]))
    if kind == "batch":
        c.update(nx=_edge(rng, 112, 160), ny=64, nz=64, members=rng.randint(4, 16), steps=rng.randint(5, 20))
        c["ny"] = c["nz"] = c["nx"]
        return c
    two_d = kind != "dropin" and rng.random() < 0.3
    c["form"] = "f64" if kind == "tank" else rng.choice(["f32", "f32", "f64"])
    c["stretch"] = 0.3 if kind == "tank" else rng.choice([0.0, 0.0, 0.3])
    hi = 900 if two_d else 224 if c["form"] == "f32" and not c["stretch"] else 112
    lo = 48 if kind == "run" else 24  # a coarser box does not resolve its spheres over many steps
    c["nx"], c["ny"], c["nz"] = _edge(rng, lo, hi), 1 if two_d else _edge(rng, lo, hi), _edge(rng, lo, hi)
    if kind == "tank":
        c.update(nx=max(c["nx"], 2 * c["nz"]), nz=min(c["nz"], 96), ny=1 if two_d else min(c["ny"], 24),
                 steps=rng.randint(3, 10))
    elif kind == "dropin":
        c.update(steps=1, f49=rng.choice([1, 1, 0]))
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
        most = 1.2e8 / cells if c["form"] == "f32" and not c["stretch"] else 3e7 / cells
        most = min(most, 50, 0.6 * min(c["nx"], c["nz"], c["nx"] if two_d else c["ny"]))
        c.update(steps=max(2, int(rng.uniform(0.3, 1.0) * most)), f49=rng.choice([1, 1, 0]),
                 airy=rng.random() < 0.15, fluid=rng.random() < 0.2, period=rng.choice([0.0, 0.0, 3.0]))
        if c["airy"]:
            c["period"] = 0.0
    return c


# ------------------------------------------------------------------ inputs
def _tank(c):
    return c["kind"] == "tank" or c["airy"]


def _box(c):
    """Lengths of the axes: the unit box, or a tank one metre high."""
    if not _tank(c):
        return 1.0, (1.0 / c["nx"] if c["ny"] == 1 else 1.0), 1.0
    h = 1.0 / c["nz"]
    return c["nx"] * h, c["ny"] * h, 1.0


def _nodes(c):
    out = []
    for n, length in zip((c["nx"], c["ny"], c["nz"]), _box(c)):
        x = r3d.uniform_nodes(n, length)
        if c["stretch"] and n > 1:
            t = x / length
            x = length * (t + c["stretch"] * np.sin(2 * np.pi * t) / (2 * np.pi))
        out.append(x)
    return out


def _member_nodes(m):
    """The nodes of an ensemble's member: the unit box."""
    return [r3d.uniform_nodes(m[0]), r3d.uniform_nodes(m[1], 1.0 / m[0] if m[1] == 1 else 1.0), r3d.uniform_nodes(m[2])]


def _members(c, seed):
    """(nx, ny, nz, spheres, modes) of each member: one, or an uneven
    ensemble of 2D and 3D grids."""
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"]])
    sizes = np.random.default_rng([c["nx"], c["members"]])  # the case's own, not the seed's
    out = []
    for q in range(c["members"]):
        dims = (c["nx"], c["ny"], c["nz"])
        if c["kind"] == "batch":
            e = [max(24, int(c["nx"] * f)) for f in sizes.uniform(0.4, 1.0, 3)]
            dims = (e[0], 1 if q % 2 else e[1], e[2])
        ns = int(rng.integers(1, 9))
        cs, rs = rng.uniform(0.2, 0.8, (ns, 3)), rng.uniform(0.05, 0.2, ns)
        sph = [(float(a[0]), float(a[1]), float(a[2]), float(r)) for a, r in zip(cs, rs)]
        modes = [(int(rng.integers(1, 4)), float(rng.normal(0.0, 0.5))) for _ in range(4)]
        out.append((*dims, sph, modes))
    return out


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())


def _centres(x):
    return 0.5 * (x[2:-3] + x[3:-2])


def _spheres(xc, yc, zc, sph, two_d):
    """Signed distance to the union, indexed [z, y, x]."""
    d = None
    for cx, cy, cz, r in sph:
        e = (xc - cx)[None, None, :] ** 2 + (zc - cz)[:, None, None] ** 2
        e = e + (0.0 * yc if two_d else (yc - cy) ** 2)[None, :, None]
        e = torch.sqrt(e) - r
        d = e if d is None else torch.minimum(d, e)
    return d


def _taylor_green(xn, yn, zn, modes, two_d):
    """Face velocities [z, y, x] at padded indices -3 .. n+2."""
    cen = [_t(_centres(a)) for a in (xn, yn, zn)]
    fac = [_t(a[3:-2]) for a in (xn, yn, zn)]
    out = []
    for comp in range(3):
        x, y, z = (fac[a] if a == comp else cen[a] for a in range(3))
        f = torch.zeros((len(z), len(y), len(x)), dtype=torch.float64, device=x.device)
        for k, a in modes:
            p = k * math.pi
            fx = torch.sin(p * x) if comp == 0 else torch.cos(p * x)
            if two_d:
                if comp != 1:
                    fz = torch.cos(p * z) if comp == 0 else torch.sin(p * z)
                    f += (a if comp == 0 else -a) * fz[:, None, None] * fx[None, None, :]
            elif comp < 2:
                fy = torch.cos(p * y) if comp == 0 else torch.sin(p * y)
                f += (a if comp == 0 else -a) * torch.cos(p * z)[:, None, None] * fy[None, :, None] * fx
        out.append(f)
    return out


def _wave(seed):
    """(amplitude, phase) of a tank's wave."""
    rng = np.random.default_rng(seed)
    return AMP * float(rng.uniform(0.6, 1.0)), float(rng.uniform(0.0, 2 * math.pi))


def _omega():
    k = 2 * math.pi / WAVELENGTH
    return k, math.sqrt(9.81 * k * math.tanh(k * DEPTH))


def _elevation(x, t, amp, phase):
    k, om = _omega()
    return DEPTH + amp * np.cos(k * x - om * t + phase)


def _airy(xn, yn, zn, t, amp, phase=0.0):
    """Face velocities of the linear wave, constant above the still water."""
    k, om = _omega()
    a = amp * om / math.sinh(k * DEPTH)
    xc, yc, zc = (_t(_centres(q)) for q in (xn, yn, zn))
    xf, zf = _t(xn[3:-2]), _t(zn[3:-2])
    one = torch.ones_like(yc)[None, :, None]
    u = a * torch.cosh(k * zc.clamp(max=DEPTH))[:, None, None] * one * torch.cos(k * xf - om * t + phase)
    w = a * torch.sinh(k * zf.clamp(max=DEPTH))[:, None, None] * one * torch.sin(k * xc - om * t + phase)
    return u, torch.zeros_like(u), w


def _tank_zones(c, xn):
    """Weights of the generation zone (the first fifth of the tank) and the
    beach (the last), per column; negative outside."""
    x = _centres(xn)[3:-3] / xn[c["nx"] + 5]
    s = np.clip(x / 0.2, 0.0, 1.0)
    b = np.clip((x - 0.8) / 0.2, 0.0, 1.0)
    gen = np.where(x < 0.2, s * s * (3.0 - 2.0 * s), -1.0)
    beach = np.where(x > 0.8, 1.0 - b * b * (3.0 - 2.0 * b), -1.0)
    return (np.ascontiguousarray(np.repeat(a[:, None], c["ny"], axis=1)) for a in (gen, beach))


def _tank_target(c, xn, zn, t, amp, phase, cols):
    xc, zc = _centres(xn)[3:-3], _centres(zn)[3:-3]
    eta = np.repeat(_elevation(xc[:cols], t, amp, phase), c["ny"])
    return np.ascontiguousarray(eta[:, None] - zc[None, :])


def _initial(c, nodes, member, seed):
    """phi [z, y, x] at padded indices -3 .. n+2 and the face velocities."""
    xn, yn, zn = nodes
    two_d = member[1] == 1
    if _tank(c):
        amp, phase = _wave(seed)
        xc, zc = _centres(xn), _centres(zn)
        phi = _t(_elevation(xc, 0.0, amp, phase))[None, None, :] - _t(zc)[:, None, None]
        phi = phi.expand(-1, c["ny"] + 6, -1).contiguous()
        return phi, _airy(xn, yn, zn, 0.0, amp, 0.0 if c["airy"] else phase)
    xc, yc, zc = (_t(_centres(a)) for a in nodes)
    return _spheres(xc, yc, zc, member[3], two_d), _taylor_green(xn, yn, zn, member[4], two_d)


def _host(f, two_d):
    """REEF3D's layout [x, y, z] on the host, y ghost planes of 2D zero."""
    a = f.permute(2, 1, 0).contiguous()
    if two_d:
        a[:, :3] = 0.0
        a[:, 4:] = 0.0
    return a.cpu().numpy()


def _dense(f, dims):
    """The interior [z, y, x]."""
    nx, ny, nz = dims
    return f[3:3 + nz, 3:3 + ny, 3:3 + nx].contiguous()


def _walls(f):
    """The interior with its wall ghosts (a Neumann copy, three layers)."""
    return torch.nn.functional.pad(f[None, None], (3,) * 6, mode="replicate")[0, 0]


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _instance(c, dims, nodes):
    return r3d.LevelSet(*dims, *nodes, f43=0.5, f44=c["f44"], f45=2.1, f49=c["f49"], n47=0.125,
                        precision=r3d.FP64 if c["form"] == "f64" else r3d.FP32)


class State:
    pass


def _put(s):
    s.ls.upload_ptr(r3d.PHI, s.phi0.data_ptr(), r3d.LAYOUT_DENSE)
    s.ls.ghost_fill(r3d.PHI)
    s.ls.set_time(0.0)


def _member_state(c, member, nodes, seed):
    """An instance with its velocities on the device, its initial level set
    in pinned host memory, and pinned room for the result."""
    s = State()
    s.dims, s.c = member[:3], c
    s.ls = _instance(c, s.dims, nodes)
    shape = (s.dims[2], s.dims[1], s.dims[0])
    if _tank(c):
        phi, vel = _initial(c, nodes, member, seed)
        if not c["airy"]:
            for f, a in zip((r3d.U, r3d.V, r3d.W), vel):
                s.ls.upload(f, _host(a, False))
        phi = _dense(phi, s.dims)
    else:
        s.ls.init_spheres_tg(member[3], member[4])
        xc, yc, zc = (_t(_centres(a)) for a in nodes)
        phi = _dense(_spheres(xc, yc, zc, member[3], s.dims[1] == 1), s.dims)
    s.phi0 = _pinned(shape)
    s.phi0.copy_(phi)
    _put(s)
    s.out = [_pinned(shape) for _ in range(3 if c["fluid"] or c["kind"] == "tank" else 1)]
    if c["fluid"] or c["kind"] == "tank":
        s.ls.set_fluid(*WATER)
    return s


def prepare(case, seed):
    c = dict(BASE, **case)
    s = State()
    s.c = c
    members = _members(c, seed)
    if c["kind"] == "batch":
        s.members, s.batch = [], r3d.Batch()
        for m in members:
            s.members.append(_member_state(c, m, _member_nodes(m), seed))
            s.batch.add(s.members[-1].ls)
        return s
    nodes = _nodes(c)
    if c["kind"] == "dropin":
        dims = (c["nx"], c["ny"], c["nz"])
        s.ls = _instance(c, dims, nodes)
        phi, vel = _initial(c, nodes, members[0], seed)
        phi = _walls(_dense(phi, dims))
        s.fields = [_host(f, False) for f in (phi, *vel)]
        s.out = np.zeros_like(s.fields[0])
        return s
    s = _member_state(c, members[0], nodes, seed)
    if c["airy"]:
        s.ls.set_velocity_airy(_wave(seed)[0], WAVELENGTH, DEPTH, 9.81)
    if c["period"]:
        s.ls.set_velocity_period(c["period"])
    if c["kind"] == "tank":
        amp, phase = _wave(seed)
        gen, beach = _tank_zones(c, nodes[0])
        cols = int(np.sum(gen[:, 0] >= 0.0))
        s.ls.set_ioflow(waves=True, f50=2, b77=1)
        s.ls.set_relaxation(gen, beach, DEPTH)
        s.dt = s.ls.cfl_dt()
        # the wave theory's targets, as REEF3D's wave generator hands them over
        s.targets = [_tank_target(c, nodes[0], nodes[2], (n + 1) * s.dt, amp, phase, cols) for n in range(c["steps"])]
    if c["tune"]:
        s.ls.autotune()
    return s


def _get(s):
    for f, o in zip((r3d.PHI, r3d.RO, r3d.VISC), s.out):
        s.ls.download_ptr(f, o.data_ptr(), r3d.LAYOUT_DENSE)
    return list(s.out) + list(s.ls.last_volume())


def run(s):
    c = s.c
    if c["kind"] == "dropin":
        for f, a in zip((r3d.PHI, r3d.U, r3d.V, r3d.W), s.fields):
            s.ls.upload(f, a)
        dt = s.ls.cfl_dt()
        s.ls.step(dt)
        s.ls.download(r3d.PHI, out=s.out)
        return [s.out[3:-3, 3:-3, 3:-3], dt, *s.ls.last_volume()]
    if c["kind"] == "batch":
        for m in s.members:
            _put(m)
        s.batch.step(c["steps"])
        return [_get(m) for m in s.members]
    _put(s)
    if c["kind"] == "tank":
        for t in s.targets:
            s.ls.set_relaxation_target(t, 1.0)
            s.ls.step(s.dt)
    else:
        s.ls.run(c["steps"], adaptive=True)
    return _get(s)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: each stage reads its input, the step's start value and (in the
    convection) the face velocities once and writes its output, the CFL step
    reads the velocities; the host copies of a pass.  Flops: 85 a WENO5
    evaluation of an axis and 20 for the rest of a stage."""
    c = dict(BASE, **case)
    total = flops = 0.0
    for m in _members(c, 1):
        cells, dim = float(m[0]) * m[1] * m[2], 2 if m[1] == 1 else 3
        vel = dim
        stages = (2 + vel) + 2 * (3 + vel) + 8 * c["f44"]
        fields = 1 + (2 if c["fluid"] or c["kind"] == "tank" else 0)
        elem = 8 if c["form"] == "f64" else 4
        words = c["steps"] * (stages + (0 if c["kind"] == "tank" else vel) + (2 * fields - 1 if fields > 1 else 0))
        up = 4 if c["kind"] == "dropin" else 1
        total += cells * (words * elem + (up + fields) * (elem + 8))
        flops += cells * c["steps"] * 3 * (1 + c["f44"]) * (85 * dim + 20)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """FP64: the sums' order and nothing else (6e-16 is measured against
    exact()).  FP32: four times what the runs are off exact() by (5e-7 over
    10 steps, up to 2.7e-6 over 50), and a single cell four times what the
    tiled and the one-cell-per-thread kernels differ by (4e-4 with F49 0,
    where rounding decides which cells are frozen)."""
    c = dict(BASE, **case)
    if c["form"] == "f64":
        return {"rel": 1e-13, "max": 1e-11}
    return {"rel": 1e-5, "max": 4e-3}


# ------------------------------------------------------------------- exact
class _Side:
    """WENO5 upwind from the lower side on the nodes X[-2] .. X[3] (the cell
    between X[0] and X[1], the value at X[1]): REEF3D's reconstruction
    weights, ideal weights and smoothness indicators."""

    def __init__(self, X, shape):
        a, b, x0, x1, x2, x3 = (X[m] for m in range(-2, 4))
        h = x1 - x0
        q = [(x2 - x1) / (x3 - x0) * ((x3 - x1) / (x2 - x0)), (x2 - x1) / (x3 - x0) * (h / (x3 - x1)),
             h / (x2 - b) * ((x1 - b) / (x2 - x0)), h / (x2 - b) * ((x2 - x1) / (x1 - b)),
             h / (x0 - a) * ((x1 - b) / (x1 - a)), 1.0 + h / (x1 - b) + h / (x1 - a)]
        c = [(x1 - a) / (x3 - a) * ((x1 - b) / (x3 - b)),
             (x1 - a) / (x3 - a) * ((x3 - x1) / (x3 - b)) * ((x3 - b) / (x2 - a) + 1.0),
             (x2 - x1) / (x3 - a) * ((x3 - x1) / (x2 - a))]
        f = [4 * (h / (x3 - x0)) ** 2, 4 * (h / (x2 - b)) ** 2, 4 * (h / (x1 - a)) ** 2]
        t = 10 * h ** 2
        s = [f[0] * (t + (x2 - x0) * (x2 - x1)) / (x3 - x1) ** 2,
             f[0] * (2 * t + 2 * (x2 - x0) * (x2 - x1) + (x3 - x0) * (2 * x2 - x1 - x0)) / ((x3 - x1) * (x2 - x0)),
             f[0] * (t + (x3 + x2 - 2 * x0) * (x3 + x2 - x1 - x0)) / (x2 - x0) ** 2,
             f[1] * (t + (x2 - x0) * (x2 - x1)) / (x1 - b) ** 2,
             f[1] * (2 * t - (x2 - x1) * (x0 - b) - (x2 - x0) * (x1 - b)) / ((x2 - x0) * (x1 - b)),
             f[1] * (t + (x0 - b) * (x1 - b)) / (x2 - x0) ** 2,
             f[2] * (t + (x1 - b) * (x0 - b)) / (x0 - a) ** 2,
             f[2] * (2 * t + 2 * (x1 - b) * (x0 - b) + (x1 - a) * (x1 + x0 - 2 * b)) / ((x1 - b) * (x0 - a)),
             f[2] * (t + (2 * x1 - a - b) * (x1 + x0 - a - b)) / (x1 - b) ** 2]
        self.q, self.c, self.s = ([_t(v).reshape(shape) for v in g] for g in (q, c, s))

    def __call__(self, q1, q2, q3, q4, q5):
        Q, C, S = self.q, self.c, self.s
        i1 = S[0] * (q5 - q4) ** 2 + S[1] * (q5 - q4) * (q3 - q4) + S[2] * (q3 - q4) ** 2 + 1e-6
        i2 = S[3] * (q2 - q3) ** 2 + S[4] * (q4 - q3) * (q2 - q3) + S[5] * (q4 - q3) ** 2 + 1e-6
        i3 = S[6] * (q1 - q2) ** 2 + S[7] * (q3 - q2) * (q1 - q2) + S[8] * (q3 - q2) ** 2 + 1e-6
        a1, a2, a3 = C[0] / i1 ** 2, C[1] / i2 ** 2, C[2] / i3 ** 2
        p1 = q4 + Q[0] * (q3 - q4) - Q[1] * (q5 - q4)
        p2 = q3 + Q[2] * (q4 - q3) - Q[3] * (q2 - q3)
        p3 = q2 + Q[4] * (q1 - q2) + Q[5] * (q3 - q2)
        return (a1 * p1 + a2 * p2 + a3 * p3) / (a1 + a2 + a3)


class _Axis:
    """One axis of n cells along dimension `dim` of fields [z, y, x]."""

    def __init__(self, x, n, dim):
        shape = [1, 1, 1]
        shape[dim] = -1
        self.n, self.dim = n, dim
        xp = 0.5 * (x[:-1] + x[1:])
        self.dxp = _t(np.diff(xp)[2:n + 7]).reshape(shape)  # between the cells -3 .. n+2
        self.dxp_cell = _t(np.diff(xp)[5:5 + n]).reshape(shape)
        self.dxn = _t(np.diff(x)[5:5 + n]).reshape(shape)
        self.dxp_mean_sum = float(np.sum(np.diff(xp)[5:5 + n]))
        self.first, self.least = float(x[6] - x[5]), float(np.min(np.diff(x)[5:5 + n]))
        X = {m: x[5 + m:5 + m + n] for m in range(-2, 5)}
        self.minus = _Side(X, shape)
        self.plus = _Side({m: -X[2 - m] for m in range(-2, 4)}, shape)  # the mirrored axis

    def faces(self, f):
        d, n = self.dim, self.n
        lo, hi = f.narrow(d, 0, 1), f.narrow(d, n - 1, 1)
        p = torch.cat([lo, lo, lo, f, hi, hi, hi], d)
        q = (p.narrow(d, 1, n + 5) - p.narrow(d, 0, n + 5)) / self.dxp
        return [q.narrow(d, m, n) for m in range(6)]

    def derivative(self, q, plus):
        return torch.where(plus, self.plus(q[5], q[4], q[3], q[2], q[1]), self.minus(*q[:5]))


class _Exact:
    """The transport in 64 bits: fields [z, y, x] over the interior, walls on
    every face (a Neumann copy)."""

    def __init__(self, c, nodes, dims):
        self.c, self.two_d = c, dims[1] == 1
        ax = [_Axis(nodes[a], dims[a], 2 - a) for a in range(3)]
        self.axes = [ax[0], ax[2]] if self.two_d else ax
        mean = sum(a.dxp_mean_sum for a in self.axes) / sum(a.n for a in self.axes)
        self.psi = 2.1 * (0.5 * (mean + ax[2].first) if self.two_d else (mean + ax[1].first + ax[2].first) / 3.0)
        self.least = min(a.least for a in ax)
        self.cell = ax[0].dxn * ax[1].dxn * ax[2].dxn
        self.delta = sum(a.dxn for a in self.axes) / len(self.axes)
        step = self.axes[0].dxp_cell
        for a in self.axes[1:]:
            step = torch.minimum(step, a.dxp_cell)
        self.dtau = 0.5 * step

    def velocity(self, vel):
        """Cell values, and the largest face values, of padded faces."""
        self.vel, self.vmax = [], 0.0
        for a, f in zip((0, 1, 2), vel):
            if self.two_d and a == 1:
                continue
            d = 2 - a
            n = [f.shape[q] - 6 for q in range(3)]
            for q in range(3):
                f = f.narrow(q, 2, n[q] + 1) if q == d else f.narrow(q, 3, n[q])
            self.vel.append(0.5 * (f.narrow(d, 1, n[d]) + f.narrow(d, 0, n[d])))
            inner = f.narrow(d, 1, n[d] - 1)
            self.vmax += float(inner.abs().max()) ** 2 if inner.numel() else 0.0
        self.vmax = math.sqrt(self.vmax)

    def dt(self, scale):
        return 0.125 * min(1e10, 2.0 / (abs(scale) * self.vmax / self.least))

    def convection(self, f, scale):
        out = torch.zeros_like(f)
        for a, v in zip(self.axes, self.vel):
            v = scale * v
            out -= v * a.derivative(a.faces(f), v < 0)
        return out

    def frozen(self, f):
        """F49 0: cells whose neighbours change sign keep their value; the y
        neighbours of a 2D cell count as zero."""
        pos, neg = f >= 0, f < 0
        for a in self.axes:
            d, n = a.dim, a.n
            p = torch.cat([f.narrow(d, 0, 1), f, f.narrow(d, n - 1, 1)], d)
            for m in (0, 2):
                pos &= p.narrow(d, m, n) >= 0
                neg &= p.narrow(d, m, n) < 0
        return ~pos if self.two_d else ~(pos | neg)

    def reini(self, f):
        sg = torch.where(f > 0, 1.0, -1.0).double()
        sg = torch.where(f.abs() < 1e-8, torch.ones_like(sg), sg)
        g = torch.zeros_like(f)
        for a in self.axes:
            q = a.faces(f)
            m, p = q[2] * sg, q[3] * sg
            c1, c2 = (m > 0) & (p > -m), (p < 0) & (m < -p)
            g += torch.where(c1 | c2, a.derivative(q, c2), torch.zeros_like(f)) ** 2
        n = torch.sqrt(g)
        s = f / torch.sqrt(f * f + g * self.delta ** 2)
        s = torch.where(torch.isnan(s), torch.ones_like(s), s)
        out = s - s * n
        return torch.where(self.frozen(f), torch.zeros_like(out), out) if self.c["f49"] == 0 else out

    @staticmethod
    def rk3(f, step, after=lambda f: f):
        a = after(f + step(f))
        b = after(0.75 * f + 0.25 * (a + step(a)))
        return after(f / 3.0 + 2.0 / 3.0 * (b + step(b)))

    def step(self, f, dt, scale=1.0, after=lambda f: f):
        f = self.rk3(f, lambda p: dt * self.convection(p, scale), after)
        for _ in range(self.c["f44"]):
            f = self.rk3(f, lambda p: self.dtau * self.reini(p))
        return f

    def heaviside(self, f):
        h = 0.5 * (1.0 + f / self.psi + torch.sin(3.14159265359 * f / self.psi) / 3.14159265359)
        return torch.where(f > self.psi, torch.ones_like(f), torch.where(f < -self.psi, torch.zeros_like(f), h))

    def volumes(self, f):
        h = self.heaviside(f)
        return [float((self.cell * h).sum()), float((self.cell * (1.0 - h)).sum())]

    def fluid(self, f):
        h = self.heaviside(f)
        return [WATER[0] * h + WATER[2] * (1.0 - h), WATER[1] * h + WATER[3] * (1.0 - h)]


def _exact_member(c, member, nodes, seed):
    dims = member[:3]
    e = _Exact(c, nodes, dims)
    f, vel = _initial(c, nodes, member, seed)
    f = _dense(f, dims)
    e.velocity(vel)
    if c["kind"] == "dropin":
        dt = e.dt(1.0)
        f = e.step(f, dt)
        return [f.permute(2, 1, 0).contiguous(), dt, *e.volumes(f)]
    t = 0.0
    amp, phase = _wave(seed)
    if c["kind"] == "tank":
        gen, beach = (_t(a.T[None, :, :]) for a in _tank_zones(c, nodes[0]))
        zc = _t(_centres(nodes[2])[3:-3])[:, None, None]
        xc = _centres(nodes[0])[3:-3]
        dt = e.dt(1.0)
        for n in range(c["steps"]):
            target = _t(_elevation(xc, (n + 1) * dt, amp, phase))[None, None, :] - zc

            def relax(p):
                p = torch.where(gen >= 0, (1.0 - gen) * target + gen * p, p)
                return torch.where(beach >= 0, (1.0 - beach) * (DEPTH - zc) + beach * p, p)
            f = e.step(f, dt, after=relax)
    else:
        for _ in range(c["steps"]):
            if c["airy"]:
                e.velocity(_airy(*nodes, t, amp))
            scale = math.cos(math.pi * t / c["period"]) if c["period"] else 1.0
            dt = e.dt(scale)
            f = e.step(f, dt, scale)
            t += dt
    more = e.fluid(f) if c["fluid"] or c["kind"] == "tank" else []
    return [f, *more, *e.volumes(f)]


def exact(case, seed):
    c = dict(BASE, **case)
    members = _members(c, seed)
    if c["kind"] == "batch":
        return [_exact_member(c, m, _member_nodes(m), seed) for m in members]
    return _exact_member(c, members[0], _nodes(c), seed)
