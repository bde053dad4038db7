"""The work a user of this library has it do, as measurable cases.

Five kinds, each through the public entry points:

  engine   a device-resident simulation (Engine): `steps` Runge-Kutta steps, then the state
           is read back into the caller's pinned buffer, as a program that writes a snapshot
           every few steps does;
  dropin   one step of a host-driven solver that keeps its blocks in device arrays: time-step
           size, then per stage halo update, right-hand side and Runge-Kutta stage;
  fluxes   the ConvectiveTermSolver call alone, on the blocks a solver hands over at once
           (one node at a time in the smallest integration);
  levels   a multi-level hierarchy (alp_levels_*): `steps` macro steps with local time
           stepping, then the leaves are read back;
  serve    a batch of independent requests through alp_serve, results kept.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from alpaca_b200 import api
from alpaca_b200 import cases as K
from alpaca_b200 import native as N
from alpaca_b200 import serving as S

IC, HS = 16, 4
GAS, WATER = (1.4, 0.0), (6.12, 3430.0)  # (gamma, B); water in units of 1e5 Pa
CFL = 0.6
NEVER = 1e300
# operations of one face flux (the reference algorithm's add, mul, div, sqrt), by dimension
FACE_FLOPS = {"fvchar": (0, 750, 1200, 1631), "fvprim": (0, 480, 770, 1048),
              "fsroe": (0, 1050, 1700, 2333)}
SERVE_BUDGET = 4 << 30


def listed():
    eng = {"kind": "engine", "precision": "fp64", "fluid": "gas", "tune": True}
    return [
        # the smallest simulation: the Sod tube's 128 cells, where launches count
        dict(eng, name="sod_1d_8", dim=1, bx=8, by=1, bz=1, scheme="fvchar", edge="open",
             steps=50, tune=False),
        # a large plane problem, odd block counts
        dict(eng, name="plane_2d_2025", dim=2, bx=45, by=45, bz=1, scheme="fvchar",
             edge="periodic", steps=20),
        # a small 3D water problem with open faces, engine as created (no autotuning)
        dict(eng, name="water_3d_60", dim=3, bx=5, by=4, bz=3, scheme="fvprim", edge="open",
             fluid="water", steps=10, tune=False),
        # the benchmark's workload: 128^3 cells, periodic, characteristic WENO5 + HLLC
        dict(eng, name="box_3d_512", dim=3, bx=8, by=8, bz=8, scheme="fvchar",
             edge="periodic", steps=20),
        # the same in the precision form
        dict(eng, name="box_3d_512_fp32flux", dim=3, bx=8, by=8, bz=8, scheme="fvchar",
             edge="periodic", steps=20, precision="fp32_flux"),
        # Roe flux splitting between walls, a middling uneven box
        dict(eng, name="walls_3d_210_fsroe", dim=3, bx=7, by=6, bz=5, scheme="fsroe",
             edge="wall", steps=10),
        # the largest: 256 x 256 x 128 cells
        dict(eng, name="box_3d_2048", dim=3, bx=16, by=16, bz=8, scheme="fvchar",
             edge="periodic", steps=10),
        # a run-time selected scheme
        dict(eng, name="weno5z_3d_64", dim=3, bx=4, by=4, bz=4, scheme="fvchar_weno5z",
             edge="periodic", steps=10),
        # the smallest integration: a solver that hands over one node's block
        {"name": "fluxes_3d_1", "kind": "fluxes", "dim": 3, "bx": 1, "by": 1, "bz": 1,
         "scheme": "fvchar", "precision": "fp64", "fluid": "gas", "edge": "periodic"},
        # a host-driven solver's step over all leaves of a level
        {"name": "dropin_3d_125", "kind": "dropin", "dim": 3, "bx": 5, "by": 5, "bz": 5,
         "scheme": "fvchar", "precision": "fp64", "fluid": "gas", "edge": "periodic"},
        # static hierarchy of three levels (two occupied) around a spherical front
        {"name": "levels_3d", "kind": "levels", "dim": 3, "n0": 2, "lmax": 2,
         "scheme": "fvchar", "precision": "fp64", "steps": 8},
        # a batch of plane quadrant problems and blasts, gas and water
        {"name": "serve_8", "kind": "serve", "count": 8, "min_blocks": 4, "max_blocks": 48,
         "scheme": "fvchar", "precision": "fp64", "steps": 48},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, dim, lo, hi):
    """Block counts per dimension with a product near a log-uniform draw from lo..hi."""
    target = _log(rng, lo, hi)
    n = [1, 1, 1]
    side = max(1.0, target ** (1.0 / dim))
    for d in range(dim - 1):
        n[d] = max(1, int(round(side * rng.uniform(0.7, 1.4))))
    n[dim - 1] = max(1, target // (n[0] * (n[1] if dim > 2 else 1)))
    while n[0] * n[1] * n[2] > hi:
        n[n.index(max(n))] -= 1
    return n


def draw(rng):
    kind = rng.choices(("engine3", "engine2", "engine1", "fluxes", "dropin", "levels", "serve"),
                       (8, 3, 2, 2, 2, 2, 2))[0]
    precision = rng.choice(("fp64", "fp64", "fp32_flux"))
    if kind.startswith("engine"):
        dim = int(kind[-1])
        bx, by, bz = _box(rng, dim, 4, (0, 64, 2025, 2048)[dim])
        scheme = rng.choice(("fvchar", "fvchar", "fvprim", "fsroe", "fvchar_weno5z", "fs_llf"))
        if "_" in scheme:
            precision = "fp64"
        cells = bx * by * bz * IC ** dim
        steps = max(2, min(rng.randint(5, 40), (8 << 20) * 10 // (2 * cells)))
        # WENO5-Z's epsilon lies far below the rounding of water's pressure
        fluid = "gas" if scheme == "fvchar_weno5z" else rng.choice(("gas", "gas", "water"))
        return {"kind": "engine", "dim": dim, "bx": bx, "by": by, "bz": bz, "scheme": scheme,
                "precision": precision, "fluid": fluid,
                "edge": rng.choice(("periodic", "open", "wall")), "steps": steps,
                "tune": rng.random() < 0.6}
    if kind in ("fluxes", "dropin"):
        dim = rng.choice((2, 3, 3))
        bx, by, bz = _box(rng, dim, 1, 512)
        return {"kind": kind, "dim": dim, "bx": bx, "by": by, "bz": bz,
                "scheme": rng.choice(("fvchar", "fvprim", "fsroe")), "precision": precision,
                "fluid": rng.choice(("gas", "gas", "water")), "edge": "periodic"}
    if kind == "levels":
        dim = rng.choice((2, 3, 3))
        return {"kind": "levels", "dim": dim, "n0": rng.choice((2, 3) if dim == 3 else (4, 6, 8)),
                "lmax": rng.choice((1, 2)), "scheme": rng.choice(("fvchar", "fsroe")),
                "precision": precision, "steps": rng.randint(1, 8)}
    return {"kind": "serve", "count": rng.randint(3, 8), "min_blocks": rng.randint(2, 6),
            "max_blocks": rng.randint(12, 64), "scheme": rng.choice(("fvchar", "fvprim")),
            "precision": precision, "steps": rng.randint(24, 56)}


# ---- inputs -------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _blocks_of(case):
    return (case["bx"], case["by"], case["bz"])


def _cell_size(case):
    return 1.0 / (IC * max(_blocks_of(case)))


def _precision(case):
    return N.FP32_FLUX if case["precision"] == "fp32_flux" else N.FP64


def _modes(rng, x, dim):
    """A sum of eight seeded Fourier modes over the box, largest value 1."""
    m = 0.0
    for _ in range(8):
        k = rng.integers(-4, 5, size=3)
        k[dim:] = 0
        if not k.any():
            k[0] = 1
        arg = 2.0 * math.pi * sum(float(k[d]) * x[d] for d in range(dim))
        m = m + float(rng.uniform(0.0, 1.0)) * torch.sin(arg + float(rng.uniform(0.0, 2.0 * math.pi)))
    return m / m.abs().max()


def _conservatives(rho, p, vel, gamma, B):
    e = (p + gamma * B) / (gamma - 1.0) + 0.5 * rho * sum(v * v for v in vel)
    return torch.stack([rho, e] + [rho * v for v in vel])


def _initial(case, seed):
    """Conserved fields [NE, X, Y, Z] of the whole box: gas with a Mach-2 front in a smooth
    field, or water at rest with spheres of higher pressure."""
    dim, n = case["dim"], _blocks_of(case)
    rng = np.random.default_rng(1000 + seed)
    dev = _device()
    ax = [(torch.arange(IC * n[d], device=dev, dtype=torch.float64) + 0.5) / (IC * n[d])
          if d < dim else torch.zeros(1, device=dev, dtype=torch.float64) for d in range(3)]
    x = torch.meshgrid(*ax, indexing="ij")
    if case["fluid"] == "water":
        gamma, B = WATER
        rho = 1.0 + 0.01 * _modes(rng, x, dim)
        p = torch.ones_like(rho)
        for _ in range(6):
            c, r = rng.uniform(0.0, 1.0, 3), rng.uniform(0.05, 0.2)
            v = 10.0 ** rng.uniform(0.0, 2.0)
            near = sum((x[d] - float(c[d])) ** 2 for d in range(dim)) < r * r
            p = torch.where(near, torch.full_like(p, v), p)
        vel = [torch.zeros_like(rho) for _ in range(dim)]
        return _conservatives(rho, p, vel, gamma, B)
    gamma, B = GAS
    rho = 1.0 + 0.1 * _modes(rng, x, dim)
    p = 1.0 + 0.1 * _modes(rng, x, dim)
    vel = [0.2 * _modes(rng, x, dim) for _ in range(dim)]
    mach2 = 4.0
    ratio = (gamma + 1.0) * mach2 / ((gamma - 1.0) * mach2 + 2.0)
    front = vel[0] + 2.0 * torch.sqrt(gamma * p / rho)
    behind = x[0] < 0.25
    u2 = front - (front - vel[0]) / ratio
    vel[0] = torch.where(behind, u2, vel[0])
    p = torch.where(behind, p * (2.0 * gamma * mach2 - (gamma - 1.0)) / (gamma + 1.0), p)
    rho = torch.where(behind, rho * ratio, rho)
    return _conservatives(rho, p, vel, gamma, B)


def _cut(u, dim, width, halo):
    """Global fields [NE, ...], padded by `halo` in the active dimensions, as blocks
    [nb, NE, width, ...] whose origins are 16 cells apart."""
    for d in range(dim):
        u = u.unfold(1 + d, width, IC)  # block index stays in place, cells go last
    for d in range(dim, 3):
        u = u.unsqueeze(-1)
    return u.permute(1, 2, 3, 0, 4, 5, 6).reshape((-1, u.shape[0]) + tuple(u.shape[4:])).contiguous()


def _pad(u, dim, width, edge):
    """Global fields with `width` more cells beyond every face of the active dimensions."""
    for d in range(dim):
        n = u.shape[1 + d]
        i = torch.arange(-width, n + width, device=u.device)
        out = (i < 0) | (i >= n)
        if edge == "periodic":
            j = i % n
        elif edge == "open":
            j = i.clamp(0, n - 1)
        else:
            j = torch.where(i < 0, -1 - i, torch.where(i >= n, 2 * n - 1 - i, i))
        u = u.index_select(1 + d, j)
        if edge == "wall":
            shape = [1, 1, 1]
            shape[d] = -1
            u[2 + d] = torch.where(out.view(shape), -u[2 + d], u[2 + d])
    return u


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _grid(case):
    per = {"periodic": True, "open": False, "wall": K.SYMMETRY}[case["edge"]]
    dim = case["dim"]
    return K.BlockGrid(dim, _blocks_of(case)[:dim], (per,) * dim, _cell_size(case))


def _level_case(case, seed):
    """Leaves around a sphere with a seeded mild front (the hierarchy is static, so the front
    may leave the finest level)."""
    rng = np.random.default_rng(2000 + seed)
    c = K.spherical_shock_levels(case["n0"], case["dim"], case["lmax"], seed=1)
    dim = case["dim"]
    rho_in, p_in = rng.uniform(1.2, 1.6), rng.uniform(1.3, 1.8)
    phase = rng.uniform(0.0, 2.0 * math.pi, 3)
    inside = K.interior(dim)
    for b in range(c.nleaf):
        x = c.cell_centres(b)
        r = np.sqrt(sum((x[d] - 0.5) ** 2 for d in range(dim)))
        f = 0.5 * (1.0 - np.tanh((r - 0.3) / 0.02))
        rho = 1.0 + (rho_in - 1.0) * f
        p = 1.0 + (p_in - 1.0) * f
        vel = [0.1 * np.sin(2.0 * math.pi * x[d] + phase[d]) for d in range(dim)]
        c.u[(b, slice(None)) + inside[1:]] = K.primes_to_conservatives(dim, rho, p, vel, 1.4)
    return c


def _requests(case, seed):
    """Independent requests: sizes and step counts are the case's, the states the seed's."""
    rng, sizes = np.random.default_rng(3000 + seed), np.random.default_rng(case["count"])
    out = []
    for i in range(case["count"]):
        nb = int(round(math.exp(sizes.uniform(math.log(case["min_blocks"]),
                                              math.log(case["max_blocks"])))))
        steps = int(sizes.integers(max(1, case["steps"] // 2), case["steps"] + 1))
        if i % 2 == 0:
            shape = S.grid_shape(nb, 2)
            h = 1.0 / (IC * max(shape[:2]))
            params = [0.5 * shape[0] * IC * h, 0.5 * shape[1] * IC * h]
            for _ in range(4):
                rho, p = rng.uniform(0.3, 2.0, 2)
                u, v = rng.uniform(-0.5, 0.5, 2)
                params += [rho, u, v, p]
            out.append(S.Request(2, shape, h, 1.4, 0.0, N.IC_QUADRANTS, params, steps))
        else:
            shape = S.grid_shape(nb, 3)
            h = 1.0 / (IC * max(shape))
            gamma, B = WATER if i % 4 == 3 else GAS
            params = [0.5 * n * IC * h for n in shape] + [0.2, 1.0, rng.uniform(10.0, 200.0), 1.0, 1.0]
            out.append(S.Request(3, shape, h, gamma, B, N.IC_BLAST, params, steps))
    return out


class _Levels:
    """A LevelEngine and the pinned buffer its leaves are read into (alp_levels_get)."""

    def __init__(self, engine):
        self.engine, self.out = engine, _pinned(engine.shape)

    def get(self):
        t, m = C.c_double(), C.c_int()
        N.check(N.lib().alp_levels_get(self.engine.h, self.out.ctypes.data_as(C.POINTER(C.c_double)),
                                       C.byref(t), C.byref(m)))
        return self.out[K.interior(self.engine.dim)], t.value, m.value


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return {"kind": kind, "requests": _requests(case, seed), "scheme": case["scheme"],
                "precision": _precision(case)}
    if kind == "levels":
        eng = api.LevelEngine(_level_case(case, seed), case["scheme"], _precision(case))
        return {"kind": kind, "levels": _Levels(eng), "steps": case["steps"]}
    dim, u = case["dim"], _initial(case, seed)
    gamma, B = WATER if case["fluid"] == "water" else GAS
    if kind == "engine":
        grid = _grid(case)
        interior = _pinned((grid.nb, dim + 2) + tuple(IC if d < dim else 1 for d in range(3)))
        interior[...] = _cut(u, dim, IC, 0).cpu().numpy()
        scheme = N.Scheme.make(case["scheme"], _precision(case))
        eng = api.Engine(dim, scheme, capacity_blocks=grid.nb, max_cases=1)
        cid = eng.add_case(K.Case("box", grid, None, gamma, B, CFL, NEVER, 0), interior=interior)
        if case["tune"]:
            eng.autotune(trial_steps=3)
        return {"kind": kind, "engine": eng, "cid": cid, "out": interior, "steps": case["steps"]}
    blocks = _cut(_pad(u, dim, HS, case["edge"]), dim, IC + 2 * HS, HS)
    state = {"kind": kind, "dim": dim, "scheme": case["scheme"], "precision": _precision(case),
             "material": N.Material.make(gamma, B), "h": _cell_size(case), "u": blocks}
    if kind == "dropin":
        nb = blocks.shape[0]
        words = max(1, N.lib().alp_space_rhs_workspace_size(dim, nb) // 8)
        state["work"] = torch.empty(words, dtype=torch.float64, device=blocks.device)
        state["u0"] = torch.zeros_like(blocks)
        state["nbr"] = torch.from_numpy(_grid(case).nbr26).to(blocks.device)
    return state


# ---- one pass -----------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "engine":
        eng = state["engine"]
        eng.step(state["steps"])
        out, t, steps = eng.get_interior(state["cid"], out=state["out"])
        return {"state": out, "t": t, "steps": steps}
    if kind == "levels":
        state["levels"].engine.step(state["steps"])
        out, t, macro = state["levels"].get()
        return {"state": out, "t": t, "macro": macro}
    if kind == "serve":
        results, _, states = api.serve(state["requests"], SERVE_BUDGET, state["scheme"],
                                       state["precision"], keep_results=True)
        return {"states": states, "t": [r["t"] for r in results],
                "steps": [r["steps"] for r in results]}
    dim, mat, h, u = state["dim"], state["material"], state["h"], state["u"]
    if kind == "fluxes":
        return [f for f in api.convective_fluxes(u, dim, state["scheme"], mat, h, state["precision"])
                if f is not None]
    dt = api.timestep_size(u, dim, mat, h, CFL)
    for stage in range(3):
        api.halo_update(u, dim, state["nbr"])
        rhs = api.space_rhs(u, dim, state["scheme"], mat, h, state["precision"],
                            workspace=state["work"])
        api.rk3_stage(u, state["u0"], rhs, dim, stage, dt)
    return {"u": u, "rhs": rhs, "dt": dt}


# ---- what a pass cannot do without --------------------------------------------------------

def _base(scheme):
    return "fsroe" if scheme.startswith("fs") else scheme.split("_")[0]


def _step_work(cells, dim, scheme, steps):
    """`steps` three-stage steps: stage 1 reads and writes the state, stages 2 and 3 read it
    and the step's initial state and write it."""
    faces = 3 * dim * (IC + 1) / IC
    return (8.0 * 8 * (dim + 2) * cells * steps,
            cells * steps * (faces * FACE_FLOPS[_base(scheme)][dim] + 30.0 * (dim + 2)))


def work(case):
    kind = case["kind"]
    if kind == "levels":
        c = _level_shape(case)
        b, f = _step_work(c, case["dim"], case["scheme"], case["steps"])
    elif kind == "serve":
        b = f = 0.0
        for r in _requests(case, 0):
            rb, rf = _step_work(r.blocks * IC ** r.dim, r.dim, case["scheme"], r.max_steps)
            b, f = b + rb, f + rf
    else:
        dim = case["dim"]
        nb = case["bx"] * case["by"] * case["bz"]
        cells, ne = nb * IC ** dim, dim + 2
        if kind == "engine":
            b, f = _step_work(cells, dim, case["scheme"], case["steps"])
        elif kind == "dropin":
            b, f = _step_work(cells, dim, case["scheme"], 1)
        else:  # the blocks with their halos in, the fluxes of every direction out
            faces = nb * dim * (IC + 1) * IC ** (dim - 1)
            b = 8.0 * ne * (nb * (IC + 2 * HS) ** dim + faces)
            f = faces * FACE_FLOPS[_base(case["scheme"])][dim]
    return {"bytes": b, "flops": f}


def _level_shape(case):
    c = K.spherical_shock_levels(case["n0"], case["dim"], case["lmax"], seed=1)
    return c.cell_updates_per_macro_step()


def tolerance(case):
    """About four times the difference seen from exact() (and, for levels, between the
    library's two builds, which round in different places)."""
    if case["precision"] == "fp32_flux":
        return {"rel": 4e-7, "max": 8e-6}
    if case.get("fluid") == "water":
        # pressure recovered from an energy of which gamma B is the larger part
        return {"rel": 2.5e-10, "max": 3e-9}
    return {"rel": 2e-14, "max": 1e-12}


# ---- the same in plain 64-bit torch -------------------------------------------------------

class _Plain:
    """The scheme on global fields [NE, X, Y, Z], textbook form."""

    def __init__(self, dim, scheme, gamma, B, h, edge):
        self.dim, self.gamma, self.B, self.h, self.edge = dim, gamma, B, h, edge
        self.splitting = scheme.startswith("fs")
        self.primitive = scheme.startswith("fvprim")
        self.llf = scheme == "fs_llf"
        self.z = scheme.endswith("weno5z")

    def pressure(self, c):
        q = sum(c[2 + d] * c[2 + d] for d in range(self.dim))
        return (self.gamma - 1.0) * (c[1] - 0.5 * q / c[0]) - self.gamma * self.B

    def sound(self, rho, p):
        return torch.sqrt(self.gamma * (p + self.B) / rho)

    def weno(self, a, b, c, d, e):
        s1 = 13.0 / 12.0 * (a - 2.0 * b + c) ** 2 + 0.25 * (a - 4.0 * b + 3.0 * c) ** 2
        s2 = 13.0 / 12.0 * (b - 2.0 * c + d) ** 2 + 0.25 * (b - d) ** 2
        s3 = 13.0 / 12.0 * (c - 2.0 * d + e) ** 2 + 0.25 * (3.0 * c - 4.0 * d + e) ** 2
        if self.z:
            tau, eps = (s1 - s3).abs(), 2.0 ** -52
            w1, w2, w3 = (g * (1.0 + tau / (s + eps)) for g, s in ((0.1, s1), (0.6, s2), (0.3, s3)))
        else:
            w1, w2, w3 = (g / (s + 1e-6) ** 2 for g, s in ((0.1, s1), (0.6, s2), (0.3, s3)))
        q1 = (2.0 * a - 7.0 * b + 11.0 * c) / 6.0
        q2 = (-b + 5.0 * c + 2.0 * d) / 6.0
        q3 = (2.0 * c + 5.0 * d - e) / 6.0
        return (w1 * q1 + w2 * q2 + w3 * q3) / (w1 + w2 + w3)

    def roe(self, l, r, d):
        """Roe averages at the faces between states l and r; momenta `d` first."""
        g, B = self.gamma, self.B
        pl, pr = self.pressure(l), self.pressure(r)
        wl, wr = torch.sqrt(l[0]), torch.sqrt(r[0])
        one = 1.0 / (wl + wr)

        def mean(x, y):
            return (x * wl + y * wr) * one
        u = [mean(l[2 + k] / l[0], r[2 + k] / r[0]) for k in range(self.dim)]
        jump = sum((l[2 + k] / l[0] - r[2 + k] / r[0]) ** 2 for k in range(self.dim))
        H = mean((l[1] + pl) / l[0], (r[1] + pr) / r[0])
        rho = wl * wr
        cc = mean((pl + g * B) / l[0], (pr + g * B) / r[0]) + (g - 1.0) * (
            mean(pl / l[0], pr / r[0]) + 0.5 * rho * one * one * jump)
        return {"u": u, "H": H, "rho": rho, "cc": cc, "c": torch.sqrt(cc),
                "q2": sum(x * x for x in u), "d": d}

    def project(self, R, c, minors):
        """Characteristic values of the state or flux vector c."""
        g1, d = self.gamma - 1.0, R["d"]
        um = sum(R["u"][k] * c[2 + k] for k in range(self.dim))
        # pressure-like part g1 ((q2 - H) c0 - u.m + E) + cc c0, velocity-like part m - u c0
        a = g1 * ((R["q2"] - R["H"]) * c[0] - um + c[1]) + R["cc"] * c[0]
        b = R["c"] * (c[2 + d] - R["u"][d] * c[0])
        half = 0.5 / R["cc"]
        out = [half * (a - b), half * (a + b), ((R["H"] - R["q2"]) * c[0] + um - c[1]) / R["cc"]]
        for k in minors:
            out.append((R["u"][k] * c[0] - c[2 + k]) / R["rho"])
        return out

    def restore(self, R, ch, minors):
        g1, d = self.gamma - 1.0, R["d"]
        rho = g1 * ch[2] + ch[0] + ch[1]
        dif = R["c"] * (ch[1] - ch[0])
        m = [None] * self.dim
        m[d] = R["u"][d] * rho + dif
        E = R["H"] * rho + R["u"][d] * dif - R["cc"] * ch[2]
        for i, k in enumerate(minors):
            m[k] = R["u"][k] * rho - R["rho"] * ch[3 + i]
            E = E - R["u"][k] * R["rho"] * ch[3 + i]
        return [rho, E] + m

    def hllc(self, l, r, pl, pr, d):
        ul, ur = l[2 + d] / l[0], r[2 + d] / r[0]
        cl, cr = self.sound(l[0], pl), self.sound(r[0], pr)
        wl, wr = torch.sqrt(l[0]), torch.sqrt(r[0])
        one = 1.0 / (wl + wr)
        u = (ul * wl + ur * wr) * one
        c = torch.sqrt((cl * cl * wl + cr * cr * wr) * one + 0.5 * wl * wr * one * one * (ur - ul) ** 2)
        sl, sr = torch.minimum(u - c, ul - cl), torch.maximum(u + c, ur + cr)
        s = ((pr - pl) + (l[2 + d] * (sl - ul) - r[2 + d] * (sr - ur))) / (
            l[0] * (sl - ul) - r[0] * (sr - ur))

        def side(c, p, v, sk, sc):
            chi = (sk - v) / (sk - s)
            star = [c[0] * chi, c[0] * chi * (c[1] / c[0] + (s - v) * (s + p / (c[0] * (sc - v))))]
            f = [c[2 + d], v * (c[1] + p)]
            for k in range(self.dim):
                star.append(c[0] * chi * s if k == d else chi * c[2 + k])
                f.append(v * c[2 + k] + (p if k == d else 0.0))
            return [a + sc * (b - q) for a, b, q in zip(f, star, c)]
        left = side(l, pl, ul, sl, sl.clamp(max=0.0))
        right = side(r, pr, ur, sr, sr.clamp(min=0.0))
        sg = torch.sign(s)
        return [0.5 * (1.0 + sg) * a + 0.5 * (1.0 - sg) * b for a, b in zip(left, right)]

    def face_fluxes(self, pad, d):
        """Fluxes at the faces along d of fields padded by three cells along d."""
        n = pad.shape[1 + d] - 6
        cell = [[f.narrow(d, m, n + 1) for f in pad] for m in range(6)]
        minors = [k for k in range(self.dim) if k != d]
        if self.primitive:
            prim = [pad[0], self.pressure(pad)] + [pad[2 + k] / pad[0] for k in range(self.dim)]
            v = [[f.narrow(d, m, n + 1) for m in range(6)] for f in prim]
            sides = []
            for o in ((0, 1, 2, 3, 4), (5, 4, 3, 2, 1)):
                q = [self.weno(*(x[m] for m in o)) for x in v]
                E = (q[1] + self.gamma * self.B) / (self.gamma - 1.0) + 0.5 * q[0] * sum(x * x for x in q[2:])
                sides.append(([q[0], E] + [q[0] * x for x in q[2:]], q[1]))
            return self.hllc(sides[0][0], sides[1][0], sides[0][1], sides[1][1], d)
        R = self.roe(cell[2], cell[3], d)
        if not self.splitting:
            ch = [self.project(R, c, minors) for c in cell]
            l, r = ([self.weno(*(ch[m][k] for m in o)) for k in range(self.dim + 2)]
                    for o in ((0, 1, 2, 3, 4), (5, 4, 3, 2, 1)))
            l, r = self.restore(R, l, minors), self.restore(R, r, minors)
            return self.hllc(l, r, self.pressure(l), self.pressure(r), d)
        p = self.pressure(pad)
        vel = pad[2 + d] / pad[0]
        phys = [pad[2 + d], (pad[1] + p) * vel]
        phys += [pad[2 + k] * vel + (p if k == d else 0.0) for k in range(self.dim)]
        if self.llf:
            vs = [cell[m][2 + d] / cell[m][0] for m in (2, 3)]
            cs = [self.sound(cell[m][0], self.pressure(cell[m])) for m in (2, 3)]
            al = [torch.maximum((vs[0] + k * cs[0]).abs(), (vs[1] + k * cs[1]).abs()) for k in (-1, 1, 0)]
        else:
            al = [(R["u"][d] + k * R["c"]).abs() for k in (-1, 1, 0)]
        al += [al[2]] * len(minors)
        U = [self.project(R, c, minors) for c in cell]
        F = [self.project(R, [f.narrow(d, m, n + 1) for f in phys], minors) for m in range(6)]
        out = []
        for k in range(self.dim + 2):
            pos = self.weno(*(F[m][k] + al[k] * U[m][k] for m in (0, 1, 2, 3, 4)))
            neg = self.weno(*(F[m][k] - al[k] * U[m][k] for m in (5, 4, 3, 2, 1)))
            out.append(0.5 * (pos + neg))
        return self.restore(R, out, minors)

    def along(self, u, d):
        """u padded by three cells along d alone."""
        pad = _pad(u, self.dim, 3, self.edge)
        for k in range(self.dim):
            if k != d:
                pad = pad.narrow(1 + k, 3, u.shape[1 + k])
        return pad

    def rhs(self, u):
        out = torch.zeros_like(u)
        for d in range(self.dim):
            f = torch.stack(self.face_fluxes(self.along(u, d), d))
            n = u.shape[1 + d]
            out += (f.narrow(1 + d, 0, n) - f.narrow(1 + d, 1, n)) / self.h
        return out

    def dt(self, u):
        c = self.sound(u[0], self.pressure(u))
        s = sum((u[2 + d] / u[0]).abs() + c for d in range(self.dim))
        return CFL * self.h / float(s.max())

    def step(self, u):
        """One SSP-RK3 step: (new state, dt, the state and right-hand side of its last stage)."""
        dt = self.dt(u)
        a = u + dt * self.rhs(u)
        b = 0.25 * a + 0.75 * u + 0.25 * dt * self.rhs(a)
        last = self.rhs(b)
        return 2.0 / 3.0 * b + 1.0 / 3.0 * u + 2.0 / 3.0 * dt * last, dt, b, last


def _exact_request(r, scheme):
    dev, dim = _device(), r.dim
    ax = [(torch.arange(IC * r.nblocks[d], device=dev, dtype=torch.float64) + 0.5) * r.cell_size
          if d < dim else torch.zeros(1, device=dev, dtype=torch.float64) for d in range(3)]
    x = torch.meshgrid(*ax, indexing="ij")
    q = r.params
    if r.ic_type == N.IC_QUADRANTS:
        at = (x[0] >= q[0]).long() + 2 * (x[1] >= q[1]).long()
        v = torch.tensor(q[2:18], device=dev, dtype=torch.float64).view(4, 4)[at]
        rho, vel, p = v[..., 0], [v[..., 1], v[..., 2]], v[..., 3]
    else:
        near = sum((x[d] - q[d]) ** 2 for d in range(3)) < q[3] * q[3]
        zero = torch.zeros_like(x[0])
        rho = torch.where(near, zero + q[4], zero + q[6])
        p = torch.where(near, zero + q[5], zero + q[7])
        vel = [zero] * 3
    u = _conservatives(rho, p, vel, r.gamma, r.B)
    plain, t = _Plain(dim, scheme, r.gamma, r.B, r.cell_size, "open"), 0.0
    for _ in range(r.max_steps):
        u, dt, _, _ = plain.step(u)
        t += dt
    return _cut(_pad(u, dim, HS, "open"), dim, IC + 2 * HS, HS), t


def exact(case, seed):
    kind = case["kind"]
    if kind == "levels":
        return None  # local time stepping over the tree in plain torch takes minutes
    if kind == "serve":
        reqs = _requests(case, seed)
        done = [_exact_request(r, case["scheme"]) for r in reqs]
        return {"states": [u.cpu().numpy() for u, _ in done], "t": [t for _, t in done],
                "steps": [None for _ in reqs]}
    dim, u = case["dim"], _initial(case, seed)
    gamma, B = WATER if case["fluid"] == "water" else GAS
    plain = _Plain(dim, case["scheme"], gamma, B, _cell_size(case), case["edge"])
    if kind == "engine":
        t = 0.0
        for _ in range(case["steps"]):
            u, dt, _, _ = plain.step(u)
            t += dt
        return {"state": _cut(u, dim, IC, 0).cpu().numpy(), "t": t, "steps": None}
    if kind == "fluxes":
        nb, out = case["bx"] * case["by"] * case["bz"], []
        for d in range(dim):
            f = torch.stack(plain.face_fluxes(plain.along(u, d), d))
            full = torch.zeros((nb, dim + 2) + tuple(IC + 1 if k < dim else 2 for k in range(3)),
                               dtype=torch.float64, device=u.device)
            # faces 0..16 along d of each block, its own cells across
            for k in range(dim):
                f = f.unfold(1 + k, IC + 1 if k == d else IC, IC)
            for k in range(dim, 3):
                f = f.unsqueeze(-1)
            f = f.permute(1, 2, 3, 0, 4, 5, 6).reshape((nb, dim + 2) + tuple(f.shape[4:]))
            full[(slice(None), slice(None)) + tuple(
                slice(0, IC + 1) if k == d else slice(1, IC + 1) if k < dim else slice(1, 2)
                for k in range(3))] = f
            out.append(full)
        return out
    u, dt, last, rhs = plain.step(u)
    blocks = _cut(_pad(last, dim, HS, case["edge"]), dim, IC + 2 * HS, HS)  # halos: the last update's
    sums = torch.zeros_like(blocks)
    inside = K.interior(dim)
    blocks[inside] = _cut(u, dim, IC, 0)
    sums[inside] = _cut(rhs, dim, IC, 0)
    return {"u": blocks, "rhs": sums, "dt": dt}
