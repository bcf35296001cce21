"""The work this framework is measured on: right-hand sides, Runge-Kutta
steps, host-buffer evaluations and batches of cases through the public
operators (theseus_b200) and the batch engine (theseus_b200.serving).

listed() are the fixed cases and draw() gives more of the same ranges:
periodic boxes, cavities and channels in 2-D and 3-D, orders 2 to 5, Euler
and Navier-Stokes, FP64 and FP32-mixed, with and without subcell blending,
the ideal and the LTE gas.  exact() evaluates the ideal-gas cases with plain
torch in 64 bits, written from the scheme's definition (DGSEM with
flux-differencing volume terms on LGL nodes, BR1 viscous terms, SSP-RK3)."""
import functools
import math
import random

import numpy as np
import torch

import theseus_b200 as T
from theseus_b200 import cases as ic
from theseus_b200.serving import BatchEngine, Case

GAMMA = 1.4
PR = 0.72
LTE_PR = 0.71
ALPHA_MAX, ALPHA_MIN, SHARPNESS = 0.5, 0.001, 9.21024
CFL = 0.4
MOST_NODES = 4_100_000   # nodes of the largest listed mesh
MOST_WORK = 12_300_000   # nodes times right-hand sides of the largest listed pass


def listed():
    return [
        # The smallest call: one right-hand side of a coarse 2-D mesh, as a
        # host-driven time integrator asks for it; all latency and launches.
        dict(name="euler2d_p2_8_mult", call="mult", setup="vortex", gas="ideal", ns=False, order=2,
             nx=8, ny=8, nz=0, volume="chandrashekar", surface="roe", precision="fp64", blend=False, steps=1),
        # The 2-D isentropic vortex run: 100 steps of a mesh that fills a
        # fraction of the chip.
        dict(name="vortex2d_p3_32_rk3", call="rk3", setup="vortex", gas="ideal", ns=False, order=3,
             nx=32, ny=32, nz=0, volume="chandrashekar", surface="roe", precision="fp64", blend=False, steps=100),
        # The lid-driven cavity: small viscous run between no-slip walls.
        dict(name="cavity2d_p3_16_rk3", call="rk3", setup="cavity", gas="ideal", ns=True, order=3,
             nx=16, ny=16, nz=0, volume="chandrashekar", surface="chandrashekar", precision="fp64", blend=False,
             steps=50),
        # A supersonic channel with a shock (inflow, outflow, slip walls,
        # subcell blending) and the step from the CFL number on the device.
        dict(name="channel2d_p3_121x41_cfl", call="rk3_cfl", setup="channel", gas="ideal", ns=False, order=3,
             nx=121, ny=41, nz=0, volume="chandrashekar", surface="chandrashekar", precision="fp64", blend=True,
             steps=10),
        # The headline benchmark: one Navier-Stokes right-hand side of the
        # Taylor-Green vortex, 4.1 M nodes, in both precisions.
        dict(name="tgv3d_p4_32_mult", call="mult", setup="tgv", gas="ideal", ns=True, order=4,
             nx=32, ny=32, nz=32, volume="ranocha", surface="hll", precision="fp64", blend=False, steps=1),
        dict(name="tgv3d_p4_32_mult_mixed", call="mult", setup="tgv", gas="ideal", ns=True, order=4,
             nx=32, ny=32, nz=32, volume="ranocha", surface="hll", precision="fp32", blend=False, steps=1),
        # A compressible viscous run on a ragged box, FP32-mixed.
        dict(name="wave3d_p5_17x10x7_rk3_mixed", call="rk3", setup="wave", gas="ideal", ns=True, order=5,
             nx=17, ny=10, nz=7, volume="chandrashekar", surface="llf", precision="fp32", blend=False, steps=5),
        # The Sedov blast with subcell blending, a step of 4.1 M nodes, in
        # both precisions (FP32-mixed evaluates the blended blocks in FP64).
        dict(name="sedov3d_p3_40_rk3", call="rk3", setup="sedov", gas="ideal", ns=False, order=3,
             nx=40, ny=40, nz=40, volume="chandrashekar", surface="llf", precision="fp64", blend=True, steps=1),
        dict(name="sedov3d_p3_40_rk3_mixed", call="rk3", setup="sedov", gas="ideal", ns=False, order=3,
             nx=40, ny=40, nz=40, volume="chandrashekar", surface="llf", precision="fp32", blend=True, steps=1),
        # A reacting-gas (LTE table) Navier-Stokes right-hand side.
        dict(name="lte3d_p4_24_mult", call="mult", setup="tgv", gas="lte", ns=True, order=4,
             nx=24, ny=24, nz=24, volume="lteec", surface="lteec", precision="fp64", blend=False, steps=1),
        # Right-hand sides of states in host memory (a host solver's vectors),
        # three in flight.
        dict(name="host3d_p2_27x22x13_mult", call="host", setup="wave", gas="ideal", ns=True, order=2,
             nx=27, ny=22, nz=13, volume="pirozzoli", surface="hll", precision="fp64", blend=False, steps=3),
        # A batch of independent small 2-D cases of mixed size, order and flow
        # through the batch engine: admitted, advanced together, fetched.
        dict(name="engine2d_48_mixed", call="engine", setup="vortex", gas="ideal", ns=True, order=0,
             nx=64, ny=64, nz=0, volume="chandrashekar", surface="roe", precision="fp32", blend=False, steps=20,
             count=48),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges: kind, then order, mesh,
    fluxes and precision."""
    kind = rng.choice(["mult2d", "mult3d", "rk3_2d", "rk3_3d", "blend3d", "cavity", "channel", "lte", "host", "engine"])
    order = rng.choice([2, 3, 4, 5])
    pair = rng.choice([("chandrashekar", "roe"), ("chandrashekar", "llf"), ("ranocha", "hll"),
                       ("pirozzoli", "hll"), ("chandrashekar", "chandrashekar")])
    c = dict(call="mult", setup="wave", gas="ideal", ns=rng.random() < 0.5, order=order, nx=0, ny=0, nz=0,
             volume=pair[0], surface=pair[1], precision=rng.choice(["fp64", "fp32"]), blend=False, steps=1)
    dim = 2
    lo, hi, steps = 300, MOST_NODES, 1
    if kind == "mult2d":
        c["setup"] = "vortex"
    elif kind == "mult3d":
        dim, c["setup"], lo = 3, rng.choice(["tgv", "wave"]), 3000
    elif kind == "rk3_2d":
        steps = _spread(rng, 5, 100)
        c.update(call="rk3", setup="vortex", steps=steps)
        hi = MOST_WORK // (3 * steps)
    elif kind == "rk3_3d":
        steps = _spread(rng, 1, 8)
        dim, lo = 3, 3000
        c.update(call="rk3", steps=steps)
        hi = MOST_WORK // (3 * steps)
    elif kind == "blend3d":
        # up to 40 cells a side: the blast stays resolved and the step positive
        dim, lo, hi = 3, 8 ** 3 * (order + 1) ** 3, min(MOST_NODES, 40 ** 3 * (order + 1) ** 3)
        c.update(call="rk3", setup="sedov", ns=False, volume="chandrashekar", surface="llf", blend=True)
    elif kind == "cavity":
        steps = _spread(rng, 5, 50)
        c.update(call="rk3", setup="cavity", ns=True, precision="fp64", steps=steps)
        hi = MOST_WORK // (30 * steps)
    elif kind == "channel":
        steps = _spread(rng, 2, 10)
        c.update(call="rk3_cfl", setup="channel", ns=False, precision="fp64", steps=steps, blend=True,
                 volume="chandrashekar", surface=rng.choice(["chandrashekar", "llf"]))
        lo, hi = 2000, MOST_WORK // (12 * steps)
    elif kind == "lte":
        dim, lo, hi = 3, 3000, 24 ** 3 * 125
        c.update(setup="tgv", gas="lte", ns=True, precision="fp64", volume="lteec", surface="lteec")
    elif kind == "host":
        dim, lo, hi = 3, 3000, 250_000
        c.update(call="host", ns=True, precision="fp64", steps=3)
    else:
        c.update(call="engine", setup="vortex", order=0, ns=True, precision="fp32", volume="chandrashekar",
                 surface="roe", steps=rng.choice([10, 15, 20]), count=rng.randint(8, 48),
                 nx=rng.randint(16, 64))
        c["ny"] = c["nx"]
        return c
    cells = max(2 ** dim, _spread(rng, lo, hi) / (order + 1) ** dim)
    stretch = [math.exp(rng.uniform(-0.4, 0.4)) for _ in range(dim)]
    scale = (cells / math.prod(stretch)) ** (1.0 / dim)
    n = [max(3, int(s * scale)) for s in stretch]
    if kind == "channel":
        n = [2 * n[0] + 1, max(3, n[1] // 2)]
    c["nx"], c["ny"], c["nz"] = n + [0] * (3 - dim)
    return c


# ---- inputs ----------------------------------------------------------------
def _dims(c):
    return [c["nx"], c["ny"]] + ([c["nz"]] if c["nz"] else [])


def _bounds(c):
    n = _dims(c)
    if c["setup"] == "tgv" or c["setup"] == "wave":
        return [0.0] * len(n), [2 * math.pi] * len(n)
    if c["setup"] == "sedov":
        return [-1.0] * len(n), [1.0] * len(n)
    if c["setup"] == "cavity":
        return [0.0] * len(n), [2.0] * len(n)
    if c["setup"] == "channel":
        return [0.0, 0.0], [3.0, 1.0]
    return [-5.0] * len(n), [5.0] * len(n)


CHANNEL_STATE = (1.4, 1.4 * 3.0, 0.0, 1.0 / (GAMMA - 1.0) + 0.5 * 1.4 * 9.0)  # Mach 3
WALL = ("no-slip-adiabatic", 0.0, 0.0, 0.0)
LID = ("no-slip-adiabatic", 1.0, 0.0, 0.0)


@functools.lru_cache(maxsize=4)
def _mesh(setup, order, n, lo, hi):
    if setup == "cavity":
        return T.box(2, order, n, lo, hi, periodic=(False, False),
                     boundary={"x-": WALL, "x+": WALL, "y-": WALL, "y+": LID})
    if setup == "channel":
        return T.box(2, order, n, lo, hi, periodic=(False, False),
                     boundary={"x-": ("supersonic-inflow",) + CHANNEL_STATE, "x+": "supersonic-outflow",
                               "y-": "slip", "y+": "slip"})
    return T.periodic_box(len(n), order, n, lo, hi)


def _mesh_of(c):
    lo, hi = _bounds(c)
    return _mesh(c["setup"], c["order"], tuple(_dims(c)), tuple(lo), tuple(hi))


@functools.lru_cache(maxsize=1)
def _table():
    return T.HelmholtzTable.ideal_dissociating_gas(256, 512, (-6.0, 1.0), (2.3, 4.3), mu0=1.9e-5, T0=273.15,
                                                   Pr=LTE_PR, **ic.IDG_O2)


def _mu(c):
    return {"tgv": 1.0 / 1600, "wave": 0.01, "vortex": 0.01, "cavity": 0.02}.get(c["setup"], 0.0) if c["ns"] else 0.0


def _initial(c, coords, seed):
    """Conserved state (numpy, [eq][element][node]) on the given node coordinates."""
    rng = np.random.default_rng(seed)
    x = coords
    if c["setup"] == "tgv":
        shift = rng.uniform(0, 2 * np.pi, (3, 1, 1))
        if c["gas"] == "lte":
            return ic.lte_taylor_green(x + shift, T0=3000.0 + rng.uniform(-50, 50))
        return ic.taylor_green(x + shift, mach=0.1, noise=1e-6, seed=seed)
    if c["setup"] == "vortex":
        v = 0.5 * math.sqrt(GAMMA) * rng.uniform(0.5, 2.0) / math.sqrt(2.0)
        return ic.isentropic_vortex(x, strength=rng.uniform(2.0, 5.0), center=tuple(rng.uniform(-1, 1, 2)),
                                    u_inf=(v, v))
    if c["setup"] == "sedov":
        return ic.sedov(x + rng.uniform(-0.02, 0.02, (len(x), 1, 1)), p0=1e-5, width=0.05 + 1.0 / max(_dims(c)))
    if c["setup"] == "cavity":
        one = np.ones_like(x[0])
        v = [0.05 * np.sin(np.pi * x[0]) * np.sin(np.pi * x[1]) * rng.uniform(-1, 1) for _ in range(2)]
        return ic.conserved(one, v, one / (0.01 * GAMMA), GAMMA)
    if c["setup"] == "channel":
        r2 = ((x[0] - rng.uniform(1.0, 1.4)) ** 2 + (x[1] - rng.uniform(0.3, 0.7)) ** 2) / 0.12 ** 2
        one = np.ones_like(x[0])
        return ic.conserved(1.4 * one, [3.0 * one, 0.0 * one], one + 4.0 * (r2 < 1.0), GAMMA)
    # a smooth compressible field, two waves a side
    ph = rng.uniform(0, 2 * np.pi, 8)
    s = sum((k + 1) * x[k] for k in range(len(x)))
    rho = 1.0 + 0.2 * np.sin(s + ph[0])
    v = [0.3 * np.cos(x[k] * (1 + k % 2) + ph[1 + k]) + 0.3 for k in range(len(x))]
    return ic.conserved(rho, v, 1.0 + 0.2 * np.cos(s + ph[5]), GAMMA)


def _speed(c):
    """A bound of |u| + sound speed (ideal gas) over the case's states."""
    return {"tgv": 11.0, "wave": 2.5, "vortex": 4.0, "cavity": 11.0, "channel": 6.0}.get(c["setup"], 0.0)


def _step(c):
    """A fixed step below the stability limit of the case."""
    lo, hi = _bounds(c)
    n, p = _dims(c), c["order"]
    h = min((b - a) / k for a, b, k in zip(lo, hi, n))
    if c["setup"] == "sedov":
        width = 0.05 + 1.0 / max(n)
        speed = math.sqrt(GAMMA * (GAMMA - 1.0) / ((2 * math.pi) ** (len(n) / 2) * width ** len(n)))
    else:
        speed = _speed(c)
    dt = CFL * h / ((2 * p + 1) * len(n) * speed)
    if c["ns"]:
        dt = min(dt, CFL * h * h / ((p + 1) ** 4 * len(n) * 2.0 * _mu(c)))
    return dt


def _operator(c, mesh):
    cls = T.NSOperator if c["ns"] else T.EulerOperator
    if c["gas"] == "lte":
        return cls(mesh, numerical_flux="lteec", surface_flux="lteec", gas=_table(), Pr=LTE_PR)
    kw = dict(numerical_flux=c["volume"], surface_flux=c["surface"], precision=c["precision"])
    if c["ns"]:
        kw.update(mu=_mu(c), Pr=PR)
    if c["blend"]:
        kw.update(blending=True, fv_flux=c["surface"], alpha_max=ALPHA_MAX, alpha_min=ALPHA_MIN)
    if c["precision"] == "fp32" and c["setup"] in ("tgv", "wave", "vortex"):
        # the constant state the FP32 working copy is carried relative to
        dim = len(_dims(c))
        kw["state_offset"] = [1.0] + [0.0] * dim + [(1.0 / (0.01 * GAMMA) if c["setup"] == "tgv" else 1.0)
                                                    / (GAMMA - 1.0)]
    return cls(mesh, **kw)


def _batch(c, seed):
    """The engine's cases: sides 8 .. nx, orders 2..5, half of them viscous."""
    rng = random.Random(1000 + c["count"])      # sizes: the same for every seed
    out = []
    for i in range(c["count"]):
        side, order, ns = rng.randint(8, c["nx"]), rng.choice([2, 3, 4, 5]), rng.random() < 0.5
        one = dict(c, order=order, nx=side, ny=side, nz=0, ns=ns)
        mesh = _small_mesh(order, side)
        u0 = _initial(one, mesh.coords, seed * 1000 + i)
        off = (1.0, 0.5, 0.5, 1.0 / (GAMMA - 1.0) + 0.25, 0.0)
        out.append((one, Case(mesh=mesh, u0=u0, nsteps=c["steps"], dt=_step(one), viscous=ns, mu=_mu(one), Pr=PR,
                              state_offset=off, geometry_key=1 + 16 * side + order)))
    return out


@functools.lru_cache(maxsize=256)
def _small_mesh(order, side):
    return T.periodic_box(2, order, (side, side), (-5.0, -5.0), (5.0, 5.0))


# ---- a pass ----------------------------------------------------------------
def prepare(case, seed):
    c = case
    if c["call"] == "engine":
        # the engine and the requests: a server keeps the one and receives the others
        return dict(call="engine", engine=BatchEngine(numerical_flux=c["volume"], surface_flux=c["surface"],
                                                      precision=c["precision"], hbm_budget=1 << 33),
                    requests=[k for _, k in _batch(c, seed)])
    mesh = _mesh_of(c)
    s = dict(call=c["call"], op=_operator(c, mesh), steps=c["steps"])
    if c["call"] == "host":
        s["states"] = [torch.from_numpy(_initial(c, mesh.coords, seed * 10 + i)).contiguous().pin_memory()
                       for i in range(c["steps"])]
        s["rates"] = [torch.empty_like(t).pin_memory() for t in s["states"]]
        return s
    s["u0"] = torch.as_tensor(_initial(c, mesh.coords, seed), device="cuda").contiguous()
    s["out"] = torch.empty_like(s["u0"])
    if c["call"] == "rk3":
        s["dt"] = _step(c)
    return s


def run(state):
    s = state
    if s["call"] == "mult":
        return s["op"].Mult(s["u0"], s["out"])
    if s["call"] == "host":
        s["op"].mult_host(s["states"], s["rates"])
        torch.cuda.current_stream().synchronize()   # the rates are the caller's only then
        return s["rates"]
    if s["call"] == "engine":
        eng, reqs = s["engine"], s["requests"]
        ids = [eng.admit(r) for r in reqs]
        left = set(ids)
        while left:
            eng.advance()
            left.difference_update(eng.poll())
        return [eng.fetch(i, r.u0.shape) for i, r in zip(ids, reqs)]
    # a run starts from its own copy of the initial state
    u = s["out"].copy_(s["u0"])
    if s["call"] == "rk3":
        return s["op"].rk3_steps(u, s["dt"], s["steps"])
    return {"dt": s["op"].rk3_steps_cfl(u, CFL, s["steps"]), "u": u}


def _units(c):
    """(nodes, nodes per element, dim, right-hand sides) of a pass, per part."""
    if c["call"] == "engine":
        rng = random.Random(1000 + c["count"])
        out = []
        for _ in range(c["count"]):
            side, order, ns = rng.randint(8, c["nx"]), rng.choice([2, 3, 4, 5]), rng.random() < 0.5
            out.append((side * side, order, 2, ns, 3 * c["steps"]))
        return out
    n = _dims(c)
    rhs = {"mult": 1, "host": c["steps"]}.get(c["call"], 3 * c["steps"])
    return [(math.prod(n), c["order"], len(n), c["ns"], rhs)]


# operations of one two-point flux (3-D; +, -, *, /, sqrt, log one each)
PAIR_FLOPS = {"chandrashekar": 78, "ranocha": 82, "pirozzoli": 46, "lteec": 700}


def work(case):
    """bytes: each right-hand side reads the state and writes the rate (a
    fused stage reads and writes the state).  flops: the two-point fluxes,
    their accumulation and the viscous derivatives."""
    b = f = 0
    for ne, p, dim, ns, rhs in _units(case):
        N, neq = p + 1, dim + 2
        nodes = ne * N ** dim
        pairs = ne * dim * N ** (dim - 1) * N * (N - 1) // 2
        b += rhs * 2 * 8 * neq * nodes
        f += rhs * pairs * (PAIR_FLOPS[case["volume"]] + 4 * neq)
        if ns:
            f += rhs * nodes * (2 * dim * N * neq + 2 * dim * dim * neq + 2 * dim * N * (neq - 1)
                                + 2 * dim * dim * (neq - 1))
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the largest error against exact() seen over orders 2
    and 5, four flux pairs and coarse to full-size meshes (LTE: between two
    roundings of the CPU restatement, contracted and separate).  Right-hand
    sides cancel: a flow of Mach 0.1 carries the pressure 71 beside velocities
    of 1, and the rates of a smooth vortex or its viscous terms shrink as the
    mesh is refined while the rounding of the fluxes grows."""
    c = case
    if c["call"] in ("mult", "host"):
        if c["gas"] == "lte":
            return {"rel": 2.5e-9, "max": 1e-7}
        rel, most = {"fp64": {"tgv": (2.4e-10, 2.4e-9), "vortex": (3e-11, 5e-10), "wave": (5e-13, 8e-12)},
                     "fp32": {"tgv": (2.5e-2, 1.0), "vortex": (7e-3, 0.15), "wave": (2e-4, 5e-3)}}[
                         c["precision"]][c["setup"]]
        return {"rel": rel, "max": most}
    if c["precision"] == "fp32":
        return {"rel": 1e-7, "max": 1e-5}
    return {"rel": 4e-15, "max": 4e-13}


# ---- 64 bits, plain torch ----------------------------------------------------
def _lgl(N):
    """LGL nodes and weights on [0, 1]."""
    P = np.polynomial.legendre.Legendre.basis(N - 1)
    x = np.concatenate([[-1.0], np.sort(np.real(P.deriv().roots())), [1.0]])
    for _ in range(3):   # polish the inner nodes
        x[1:-1] -= P.deriv()(x[1:-1]) / P.deriv(2)(x[1:-1])
    w = 2.0 / (N * (N - 1) * P(x) ** 2)
    return 0.5 * (x + 1.0), 0.5 * w


def _log_mean(a, b):
    """(b - a) / log(b / a), without cancellation for near arguments."""
    s, d = a + b, b - a
    f = d / s
    u = f * f
    series = 1 + u * (1 / 3 + u * (1 / 5 + u * (1 / 7 + u * (1 / 9 + u * (1 / 11 + u * (1 / 13 + u / 15))))))
    far = u > 0.01
    return torch.where(far, d / torch.where(far, 2 * torch.atanh(f), torch.ones_like(f)), 0.5 * s / series)


class _Exact:
    """DGSEM on a Cartesian box: state [eq, (nz,) ny, nx, (k,) j, i]."""

    def __init__(self, c):
        self.c, self.n, self.N = c, _dims(c), c["order"] + 1
        self.dim = len(self.n)
        lo, hi = _bounds(c)
        self.h = [(b - a) / k for a, b, k in zip(lo, hi, self.n)]
        x, w = _lgl(self.N)
        N = self.N
        bw = np.array([1.0 / np.prod([x[i] - x[j] for j in range(N) if j != i]) for i in range(N)])
        D = np.array([[bw[j] / bw[i] / (x[i] - x[j]) if i != j else 0.0 for j in range(N)] for i in range(N)])
        D -= np.diag(D.sum(1))
        self.D, self.w, self.x = D, w, x
        self.mu = _mu(c)
        self.walls = c["setup"] in ("cavity", "channel")

    def ax(self, d):
        """Element and node axis of direction d in an [eq, ...] array."""
        return 1 + self.dim - 1 - d, 1 + 2 * self.dim - 1 - d

    def prims(self, u):
        v = [u[1 + d] / u[0] for d in range(self.dim)]
        p = (GAMMA - 1) * (u[-1] - 0.5 * u[0] * sum(k * k for k in v))
        return u[0], v, p

    def two_point(self, a, b, d):
        (r1, v1, p1), (r2, v2, p2) = a, b
        vb = [0.5 * (x + y) for x, y in zip(v1, v2)]
        kind = self.c["volume"]
        if kind == "pirozzoli":
            r = 0.5 * (r1 + r2)
            hh = sum(0.5 * (g * p / ((g - 1) * q) + 0.5 * sum(k * k for k in v))
                     for g, q, v, p in ((GAMMA, r1, v1, p1), (GAMMA, r2, v2, p2)))
            pm = 0.5 * (p1 + p2)
            fe = r * vb[d] * hh
        elif kind == "ranocha":
            r, pm = _log_mean(r1, r2), 0.5 * (p1 + p2)
            ie = p1 * p2 / _log_mean(r1 * p2, r2 * p1) / (GAMMA - 1)
            fe = 0.5 * (p1 * v2[d] + p2 * v1[d]) + r * vb[d] * (ie + 0.5 * sum(x * y for x, y in zip(v1, v2)))
        else:
            r = _log_mean(r1, r2)
            b1, b2 = 0.5 * r1 / p1, 0.5 * r2 / p2
            pm = 0.5 * (r1 + r2) / (b1 + b2)
            hh = 0.5 / _log_mean(b1, b2) / (GAMMA - 1) + pm / r
            hh = hh + sum(x * x for x in vb) - 0.25 * sum(x * x + y * y for x, y in zip(v1, v2))
            fe = r * vb[d] * hh
        f = [r * vb[d]] + [r * vb[d] * x for x in vb] + [fe]
        f[1 + d] = f[1 + d] + pm
        return torch.stack(f)

    def riemann(self, kind, ul, ur, d, sgn=1.0):
        """F*(ul, ur) along sgn * e_d."""
        (r1, v1, p1), (r2, v2, p2) = self.prims(ul), self.prims(ur)
        n1, n2 = sgn * v1[d], sgn * v2[d]
        c1, c2 = torch.sqrt(GAMMA * p1 / r1), torch.sqrt(GAMMA * p2 / r2)

        def flux(u, vn, p):
            f = u * vn
            f[1 + d] += sgn * p
            f[-1] += p * vn
            return f
        f1, f2, du = flux(ul, n1, p1), flux(ur, n2, p2), ur - ul
        if kind == "llf":
            return 0.5 * (f1 + f2) - 0.5 * torch.maximum(n1.abs() + c1, n2.abs() + c2) * du
        if kind == "hll":
            sl, sr = torch.minimum(n1 - c1, n2 - c2), torch.maximum(n1 + c1, n2 + c2)
            mid = (sr * f1 - sl * f2 + sl * sr * du) / (sr - sl)
            return torch.where(sl >= 0, f1, torch.where(sr <= 0, f2, mid))
        if kind == "roe":
            a, b = torch.sqrt(r1), torch.sqrt(r2)
            h1, h2 = (ul[-1] + p1) / r1, (ur[-1] + p2) / r2
            H = (a * h1 + b * h2) / (a + b)
            v = [(a * x + b * y) / (a + b) for x, y in zip(v1, v2)]
            vn, dvn, rr = sgn * v[d], n2 - n1, a * b
            v2_ = sum(x * x for x in v)
            cc = torch.sqrt((GAMMA - 1) * (H - 0.5 * v2_))
            dp, dr = p2 - p1, r2 - r1
            am, ap = (dp - rr * cc * dvn) / (2 * cc * cc), (dp + rr * cc * dvn) / (2 * cc * cc)
            az = dr - dp / (cc * cc)
            lm, lz, lp = (vn - cc).abs(), vn.abs(), (vn + cc).abs()
            e = [sgn if k == d else 0.0 for k in range(self.dim)]
            dvt = [(y - x) - dvn * e[k] for k, (x, y) in enumerate(zip(v1, v2))]
            diss = [lm * am + lz * az + lp * ap]
            for k in range(self.dim):
                diss.append(lm * am * (v[k] - cc * e[k]) + lz * (az * v[k] + rr * dvt[k]) + lp * ap * (v[k] + cc * e[k]))
            diss.append(lm * am * (H - cc * vn) + lz * (0.5 * az * v2_ + rr * sum(x * y for x, y in zip(v, dvt)))
                        + lp * ap * (H + cc * vn))
            return 0.5 * (f1 + f2) - 0.5 * torch.stack(diss)
        # entropy-conservative mean with scalar dissipation
        f = self.two_point((r1, v1, p1), (r2, v2, p2), d) * sgn   # only paired with the Chandrashekar mean
        lam = torch.maximum(n1.abs() + c1, n2.abs() + c2)
        dr, rm = r2 - r1, 0.5 * (r1 + r2)
        b1, b2 = 0.5 * r1 / p1, 0.5 * r2 / p2
        de = sum(0.5 * dr * x * y + rm * (y - x) * 0.5 * (x + y) for x, y in zip(v1, v2))
        de = de + 0.5 * dr / (GAMMA - 1) / _log_mean(b1, b2) + 0.5 * rm / (GAMMA - 1) * (1 / b2 - 1 / b1)
        diss = torch.cat([du[:-1], de[None]])
        return f - 0.5 * lam * diss

    def wall_pressure(self, u, d, sgn):
        r, v, p = self.prims(u)
        vn, c = sgn * v[d], torch.sqrt(GAMMA * p / r)
        g1, gm = GAMMA + 1, GAMMA - 1
        comp = p + 0.25 * vn * g1 * r * (vn + torch.sqrt(vn * vn + 8 / g1 * p * (gm / g1 + 1) / r))
        rare = p * torch.clamp(1 + 0.5 * gm * vn / c, min=1e-4) ** (2 * GAMMA / gm)
        return torch.where(vn > 0, comp, rare)

    def entropy(self, u):
        r, v, p = self.prims(u)
        b = r / p
        s = torch.log(p) - GAMMA * torch.log(r)
        return torch.stack([(GAMMA - s) / (GAMMA - 1) - 0.5 * b * sum(x * x for x in v)] + [b * x for x in v] + [-b])

    def lid(self, d, sgn):
        """Wall velocity of the cavity's side."""
        return [1.0 if (d == 1 and sgn > 0 and k == 0) else 0.0 for k in range(self.dim)]

    def boundary_flux(self, u, d, sgn, gp):
        """Flux out of a boundary side from its trace u (gp: primitive gradients)."""
        if self.c["setup"] == "cavity":
            r, v, p = self.prims(u)
            div = sum(gp[k][1 + k] for k in range(2))
            tr = [sgn * self.mu * ((gp[d][1 + k] + gp[k][1 + d]) - (2.0 / 3.0 * div if k == d else 0.0)) for k in range(2)]
            vw = self.lid(d, sgn)
            f = [torch.zeros_like(r)] + [-t for t in tr] + [-sum(a * t for a, t in zip(vw, tr))]
            f[1 + d] = f[1 + d] + sgn * self.wall_pressure(u, d, sgn)
            return torch.stack(f)
        if d == 1:
            f = torch.zeros_like(u)
            f[2] = sgn * self.wall_pressure(u, d, sgn)
            return f
        if sgn > 0:
            return self.riemann(self.c["surface"], u, u, d, sgn)
        q = torch.tensor(CHANNEL_STATE, dtype=u.dtype, device=u.device).reshape(-1, *[1] * (u.dim() - 1)).expand_as(u)
        return self.riemann(self.c["surface"], u, q, d, sgn)

    def faces(self, q, d):
        """Traces at every +d face: the element's own and its neighbour's."""
        ea, na = self.ax(d)
        return q.select(na, self.N - 1), torch.roll(q.select(na, 0), -1, ea)

    def viscous_flux(self, u, g):
        """Primitive gradients g[d][eq] -> viscous flux [d][eq]."""
        r, v, p = self.prims(u)
        div = sum(g[k][1 + k] for k in range(self.dim))
        out = []
        for d in range(self.dim):
            tau = [self.mu * (g[d][1 + k] + g[k][1 + d]) for k in range(self.dim)]
            tau[d] = tau[d] - 2.0 / 3.0 * self.mu * div
            q = self.mu * GAMMA / (PR * (GAMMA - 1)) / r * (g[d][-1] - p / r * g[d][0])
            out.append(torch.stack([torch.zeros_like(r)] + tau + [q + sum(a * t for a, t in zip(v, tau))]))
        return out

    def derive(self, M, q, d):
        na = self.ax(d)[1]
        m = torch.as_tensor(M, dtype=q.dtype, device=q.device)
        return torch.movedim(torch.tensordot(q, m, dims=([na], [1])), -1, na) / self.h[d]

    def gradients(self, u):
        """BR1 gradient of the entropy variables, as primitive gradients."""
        s = self.entropy(u)
        r, v, p = self.prims(u)
        out = []
        for d in range(self.dim):
            ea, na = self.ax(d)
            g = self.derive(self.D, s, d)
            sm, sp = self.faces(s, d)
            jump = 0.5 * (sp - sm)
            hi, lo = jump.clone(), torch.roll(jump, 1, ea)
            if self.walls:
                for sgn, side in ((1.0, hi), (-1.0, lo)):
                    k = self.n[d] - 1 if sgn > 0 else 0
                    w = s.select(na, self.N - 1 if sgn > 0 else 0).select(ea, k)
                    e = torch.stack([w[0]] + [-w[-1] * a for a in self.lid(d, sgn)] + [w[-1]])
                    side.select(ea, k).copy_(sgn * (e - w))
            scale = 1.0 / (self.w[0] * self.h[d])
            g.select(na, self.N - 1).add_(hi * scale)
            g.select(na, 0).add_(lo * scale)
            # entropy -> primitive gradient
            t = p / r
            dv = [t * (g[1 + k] + v[k] * g[-1]) for k in range(self.dim)]
            ke, ie = 0.5 * r * sum(x * x for x in v), p / (GAMMA - 1)
            dr = r * g[0] - g[-1] * (ke - ie) + r * r / p * sum(x * y for x, y in zip(v, dv))
            out.append(torch.stack([dr] + dv + [t * (dr + p * g[-1])]))
        return out

    def alpha(self, u):
        """Blending coefficient of every element (modal energy of p rho)."""
        r, _, p = self.prims(u)
        q = (p * r)[None]
        N = self.N
        V = np.array([[np.polynomial.legendre.Legendre.basis(k)(2 * x - 1) for k in range(N)] for x in self.x])
        for d in range(self.dim):
            q = self.derive(np.linalg.inv(V), q, d) * self.h[d]
        q = q[0] ** 2
        axes = list(range(q.dim() - self.dim, q.dim()))

        def upto(k):
            t = q
            for a in axes:
                t = t.narrow(a, 0, k)
            return t.sum(axes)
        mm, m1, m2 = upto(N), upto(N - 1), upto(N - 2)
        eta = torch.clamp(torch.maximum(1 - m1 / mm, 1 - m2 / m1), 0, 1)
        thr = 0.5 * 10 ** (-1.8 * (N - 1) ** 0.25)
        al = 1 / (1 + torch.exp(-SHARPNESS * (eta - thr) / thr))
        al = torch.where(al < ALPHA_MIN, torch.zeros_like(al), al)
        return torch.clamp(torch.where(al > 1 - ALPHA_MIN, torch.ones_like(al), al), max=ALPHA_MAX)

    def rhs(self, u):
        N, c = self.N, self.c
        r, v, p = self.prims(u)
        du = torch.zeros_like(u)
        for d in range(self.dim):
            na = self.ax(d)[1]
            at = [(r.select(na - 1, i), [x.select(na - 1, i) for x in v], p.select(na - 1, i)) for i in range(N)]
            for i in range(N):
                for j in range(i + 1, N):
                    f = self.two_point(at[i], at[j], d)
                    du.select(na, i).sub_(2 * self.D[i, j] / self.h[d] * f)
                    du.select(na, j).sub_(2 * self.D[j, i] / self.h[d] * f)
        if c["blend"]:
            fv = torch.zeros_like(u)
            for d in range(self.dim):
                na = self.ax(d)[1]
                for i in range(N - 1):
                    f = self.riemann(c["surface"], u.select(na, i), u.select(na, i + 1), d)
                    fv.select(na, i).sub_(f / (self.h[d] * self.w[i]))
                    fv.select(na, i + 1).add_(f / (self.h[d] * self.w[i + 1]))
            al = self.alpha(u)
            al = al.reshape(1, *al.shape, *[1] * self.dim)
            du = torch.where(al > 1e-16, (1 - al) * du + al * fv, du)
        gp = fv_ = None
        if c["ns"]:
            gp = self.gradients(u)
            fv_ = self.viscous_flux(u, gp)
            weak = -(self.w[None, :] / self.w[:, None]) * self.D.T
            for d in range(self.dim):
                du += self.derive(weak, fv_[d], d)
        for d in range(self.dim):
            ea, na = self.ax(d)
            f = self.riemann(c["surface"], *self.faces(u, d), d)
            if c["ns"]:
                a, b = self.faces(fv_[d], d)
                f = f - 0.5 * (a + b)
            lo = torch.roll(f, 1, ea)
            if self.walls:
                for sgn, side in ((1.0, f), (-1.0, lo)):
                    k, m = (self.n[d] - 1, N - 1) if sgn > 0 else (0, 0)
                    g = [x.select(na, m).select(ea, k) for x in gp] if gp else None
                    side.select(ea, k).copy_(sgn * self.boundary_flux(u.select(na, m).select(ea, k), d, sgn, g))
            scale = 1.0 / (self.w[0] * self.h[d])
            du.select(na, N - 1).sub_(f * scale)
            du.select(na, 0).add_(lo * scale)
        return du

    def cfl_step(self, u):
        """CFL / rate (Euler): the wave speeds over the order's calibrated length."""
        cal = {2: 5.41995189335, 3: 9.64849524786, 4: 14.7297419321, 5: 20.5984751391}[self.c["order"]]
        r, v, p = self.prims(u)
        snd = torch.sqrt(GAMMA * p / r)
        return CFL / (1.05 * cal * sum((v[d].abs() + snd) / self.h[d] for d in range(self.dim)).max())

    def steps(self, u, dt, steps):
        taken = []
        for _ in range(steps):
            t = self.cfl_step(u) if dt is None else dt
            taken.append(t)
            y = u + t * self.rhs(u)
            y = 0.75 * u + 0.25 * (y + t * self.rhs(y))
            u = u / 3 + 2.0 / 3.0 * (y + t * self.rhs(y))
        return u, taken


def exact(case, seed):
    """What run() returns, in 64 bits with plain torch.  None for the LTE gas:
    its thermodynamics are those of the table's own interpolant."""
    c = case
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def one(k, u0, fn):
        E = _Exact(k)
        u = torch.as_tensor(u0, dtype=torch.float64, device=dev)
        return fn(E, u.reshape(u.shape[0], *E.n[::-1], *[E.N] * E.dim).clone(), u.shape)
    if c["gas"] == "lte":
        return None
    if c["call"] == "engine":
        return [one(k, q.u0, lambda E, u, s: E.steps(u, q.dt, q.nsteps)[0].reshape(s).cpu()) for k, q in _batch(c, seed)]
    coords = _mesh_of(c).coords
    if c["call"] == "host":
        return [one(c, _initial(c, coords, seed * 10 + i), lambda E, u, s: E.rhs(u).reshape(s)) for i in range(c["steps"])]
    u0 = _initial(c, coords, seed)
    if c["call"] == "mult":
        return one(c, u0, lambda E, u, s: E.rhs(u).reshape(s))
    if c["call"] == "rk3":
        return one(c, u0, lambda E, u, s: E.steps(u, _step(c), c["steps"])[0].reshape(s))
    u, dt = one(c, u0, lambda E, u, s: (lambda r: (r[0].reshape(s), r[1]))(E.steps(u, None, c["steps"])))
    return {"dt": torch.stack(dt), "u": u}
