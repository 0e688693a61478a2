"""What this framework's time is spent on, as cases that can be measured.

A case is one pass of a user's program: simulations advance some time steps
and their conserved moments are read, a batch of simulations does the same, or
the closure network takes some training steps.  ``listed()`` names twelve,
``draw(rng)`` gives others of the same ranges, ``prepare`` makes what the
program has in hand before the pass, ``run`` is the pass, ``work`` what the
pass cannot do without and ``exact`` its result in 64 bits, from a restatement
of the schemes in this file alone.

The flows (a case's ``flow``):

* ``cavity``    D2Q9 MRT lid-driven cavity, bounce-back walls.
* ``shear``     D2Q9 MRT periodic double shear layer.
* ``learned``   the same at Re 30 000 with the trained collision closure.
* ``tgv``       D3Q19 MRT periodic Taylor-Green vortex.
* ``cube``      D3Q19 MRT lid-driven cube, bounce-back walls.
* ``disc``      D2Q9 MRT flow past a disc: anti-bounce-back inflow, Neumann
                outflow, periodic in y, bounce-back on the disc.
* ``karman``    D2Q9 Geier (relative velocity) flow past a disc: Bouzidi walls,
                inflow and disc, Neumann outflow.
* ``ensemble``  independent shear layers of uneven sizes and viscosities.
* ``training``  Adam steps of the closure network.

``read`` says how the program steps and reads: ``fields`` is ``run(steps)``
and ``fields(out=page-locked array)``; ``moments`` is a loop of
``one_time_step()`` and ``m[...]``, as pylbm's demos are written; ``restart``
is ``fields`` after new initial moments from page-locked host memory.
"""
import math
import os

import numpy as np
import torch

import pylbm_gb300
from pylbm_gb300 import Simulation, closure, pinned_empty, runtime
from pylbm_gb300 import workloads as W
from pylbm_gb300.ensemble import Ensemble
from pylbm_gb300.simulation import to_storage

BYTES = {"float64": 8, "float32": 4, "float16": 2, "bfloat16": 2}
MODEL = os.path.join(os.path.dirname(pylbm_gb300.__file__), "data", "closure_d2q9_shear_re30000.npz")
U0 = 0.05           # lid, inflow and shear-layer velocity
TGV_U0 = 0.04
RATES_2D = [0.0, 0.0, 0.0, 1.5, 1.5, 1.2, 1.2]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # pylbm's classic demo as written: a loop of single steps on a small
        # grid, one call at a time, and the moments read by name
        {"name": "shear_96_f32_steps", "flow": "shear", "n": 96, "dtype": "float32", "steps": 200, "read": "moments"},
        # a validation run: the FP64 path that reproduces pylbm's Cython
        {"name": "cavity_256_f64", "flow": "cavity", "n": 256, "dtype": "float64", "steps": 200, "read": "fields"},
        # an ordinary 2D run, all of it in the caches
        {"name": "shear_256_f32", "flow": "shear", "n": 256, "dtype": "float32", "steps": 500, "read": "fields"},
        # the learned closure at the size it was trained for, on new initial states
        {"name": "learned_256_f32", "flow": "learned", "n": 256, "dtype": "float32", "steps": 300, "read": "restart"},
        # obstacle flow with every boundary method but Bouzidi's
        {"name": "disc_2048x512_f32", "flow": "disc", "nx": 2048, "ny": 512, "radius": 32, "dtype": "float32",
         "steps": 300, "read": "fields"},
        # relative velocity, curved walls; the largest 2D grid
        {"name": "karman_2048x1024_f32", "flow": "karman", "ny": 1024, "dtype": "float32", "steps": 150,
         "read": "fields"},
        # the headline flow, end to end: host moments in, steps, host moments out
        {"name": "tgv_256_f32_restart", "flow": "tgv", "n": 256, "dtype": "float32", "steps": 100, "read": "restart"},
        # the same flow in 16 bits
        {"name": "tgv_192_f16", "flow": "tgv", "n": 192, "dtype": "float16", "steps": 200, "read": "fields"},
        # and in the FP64 form
        {"name": "tgv_64_f64", "flow": "tgv", "n": 64, "dtype": "float64", "steps": 20, "read": "fields"},
        # walls in 3D, a size that is a multiple of nothing
        {"name": "cube_131_f32", "flow": "cube", "n": 131, "dtype": "float32", "steps": 150, "read": "fields"},
        # a parameter study: many simulations advanced together
        {"name": "ensemble_48_f16", "flow": "ensemble", "count": 48, "dtype": "float16", "steps": 2000},
        # training the closure: forward, backward and update
        {"name": "training_32768", "flow": "training", "batch": 32768, "steps": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any flow, its size over the whole range (odd ones
    among them), any type that its users store it in."""
    flow = rng.choice(["cavity", "shear", "shear", "learned", "tgv", "tgv", "cube", "disc", "karman", "ensemble",
                       "training"])
    if flow == "cavity":
        case = {"n": _log_int(rng, 32, 1024), "dtype": rng.choice(["float64", "float32", "float16"]),
                "steps": rng.randint(50, 200), "read": "fields"}
        if case["dtype"] == "float64":
            case["n"] = min(case["n"], 512)
    elif flow == "shear":
        case = {"n": _log_int(rng, 48, 1536), "dtype": rng.choice(["float32", "float32", "float16", "bfloat16"]),
                "steps": rng.randint(50, 400), "read": rng.choice(["fields", "fields", "moments"])}
    elif flow == "learned":
        case = {"n": _log_int(rng, 128, 1100), "dtype": "float32", "steps": rng.randint(50, 300), "read": "restart"}
    elif flow == "tgv":
        case = {"n": _log_int(rng, 24, 224), "dtype": rng.choice(["float32", "float16", "bfloat16", "float64"]),
                "steps": rng.randint(20, 100), "read": rng.choice(["fields", "restart"])}
        if case["dtype"] == "float64":
            case["n"] = min(case["n"], 96)
            case["steps"] = min(case["steps"], 40)
    elif flow == "cube":
        case = {"n": _log_int(rng, 24, 144), "dtype": rng.choice(["float32", "float16"]),
                "steps": rng.randint(20, 150), "read": "fields"}
    elif flow == "disc":
        ny = _log_int(rng, 96, 700)
        case = {"nx": rng.randint(2 * ny, 4 * ny), "ny": ny, "radius": ny // 16, "dtype": "float32",
                "steps": rng.randint(50, 300), "read": "fields"}
    elif flow == "karman":
        case = {"ny": _log_int(rng, 96, 1024), "dtype": "float32", "steps": rng.randint(50, 150), "read": "fields"}
    elif flow == "ensemble":
        case = {"count": _log_int(rng, 8, 48), "dtype": rng.choice(["float16", "float32"]),
                "steps": rng.randint(200, 1000)}
    else:
        case = {"batch": _log_int(rng, 1024, 131072), "steps": rng.randint(20, 100)}
    return {"flow": flow, **case}


# ------------------------------------------------- inputs: flows and their starts
def _modes(seed, dim, count=3):
    """Seeded low modes (wave numbers, phase, amplitude) of a box-periodic perturbation."""
    rng = np.random.default_rng(seed)
    return [(rng.integers(1, 4, size=dim), rng.uniform(0.0, 2.0 * np.pi), rng.uniform(0.3, 1.0)) for _ in range(count)]


def _perturbed(base, modes, length, amplitude):
    """The function base(x, ...) + amplitude * sum of modes on a box of sides ``length``."""
    def value(*x):
        out = base(*x)
        for k, phase, a in modes:
            arg = phase + sum(2.0 * np.pi * int(kd) * xd / ld for kd, xd, ld in zip(k, x, length))
            out = out + amplitude * a * np.sin(arg)
        return out
    return value


def _constant(v):
    return lambda *x: v + 0.0 * sum(x)


def _start(case, seed):
    """Functions of the initial conserved moments, and the box sides."""
    flow = case["flow"]
    if flow in ("tgv", "cube"):
        side = 2.0 * np.pi if flow == "tgv" else 1.0
        length = (side,) * 3
        if flow == "tgv":
            base = W.tgv3d(n=case["n"], u0=TGV_U0)["init"]
            base = [base[s] for s in (W.RHO, W.QX, W.QY, W.QZ)]
        else:
            base = [_constant(1.0)] + [_constant(0.0)] * 3
        amplitude = 0.05 * TGV_U0
    else:
        length = {"disc": (case.get("nx", 1) / case.get("ny", 1), 1.0), "karman": (2.0, 1.0)}.get(flow, (1.0, 1.0))
        if flow == "shear":
            d = W.shear_layer(n=case["n"], u0=U0)["init"]
            base = [_constant(1.0), d[W.QX], d[W.QY]]
        elif flow == "learned":
            d = closure.study_dicos(seed, case["n"])["init"]
            base = [_constant(1.0), d[W.QX], d[W.QY]]
        elif flow == "cavity":
            base = [_constant(1.0), _constant(0.0), _constant(0.0)]
        else:
            base = [_constant(1.0), _constant(U0), _constant(0.0)]
        amplitude = 0.02 * U0
    dim = len(length)
    return [base[0]] + [_perturbed(b, _modes(1000 * seed + i, dim), length, amplitude)
                        for i, b in enumerate(base[1:])], length


def _disc_re(case):
    return 200.0 * case["radius"] / 32.0   # one viscosity at every size


def _disc_center(case):
    return (round(case["nx"] * 400 / 2048), case["ny"] // 2 + 1)


def _dico(case, seed):
    flow = case["flow"]
    if flow == "cavity":
        d = W.cavity(n=case["n"], lid=U0)
    elif flow == "shear":
        d = W.shear_layer(n=case["n"], u0=U0)
    elif flow == "learned":
        d = closure.study_dicos(seed, case["n"])
    elif flow == "tgv":
        d = W.tgv3d(n=case["n"], u0=TGV_U0)
    elif flow == "cube":
        d = W.cavity3d(n=case["n"], lid=U0)
    elif flow == "disc":
        d = W.cylinder(nx=case["nx"], ny=case["ny"], radius=case["radius"], center=_disc_center(case), u_in=U0,
                       re=_disc_re(case))
    else:
        d = W.karman(dx=1.0 / case["ny"], u_o=U0)
    symbols = (W.RHO, W.QX, W.QY, W.QZ)
    d["init"] = dict(zip(symbols, _start(case, seed)[0]))
    return d


def _reference_state(case):
    """Reference state of the stored deviations: rest, or the inflow."""
    nc = 4 if case["flow"] in ("tgv", "cube") else 3
    c0 = [1.0] + [0.0] * (nc - 1)
    if case["flow"] in ("disc", "karman"):
        c0[1] = U0
    return c0


def _members(case, seed):
    """Sides, viscosities and perturbation seeds of an ensemble: the sides
    belong to the case, the rest to the seed."""
    count = case["count"]
    sides = 64 + 32 * np.random.default_rng(count).integers(0, 15, size=count)
    rng = np.random.default_rng(seed)
    nu = np.exp(rng.uniform(np.log(5e-4), np.log(5e-2), size=count))
    return [int(s) for s in sides], nu, [int(seed * 1009 + i) for i in range(count)]


def _samples(case, seed):
    """Training inputs (normalised moments), targets and initial parameters."""
    rng = np.random.default_rng(seed)
    x = np.zeros((case["batch"], closure.IN))
    x[:, :9] = rng.normal(size=(case["batch"], 9))
    mix = rng.normal(size=(9, closure.OUT)) / 3.0
    t = np.tanh(x[:, :9] @ mix)
    return x, t, closure.init_params(seed)


def prepare(case, seed):
    flow = case["flow"]
    if flow == "training":
        x, t, params = _samples(case, seed)
        mlp = closure.Mlp(params=params)
        bits = to_storage(x, "bfloat16")
        dx, dt = runtime.DeviceBuffer(bits.nbytes), runtime.DeviceBuffer(4 * t.size)
        dx.upload(bits)
        dt.upload(t.astype(np.float32))
        return {"case": case, "mlp": mlp, "x": dx, "t": dt}
    if flow == "ensemble":
        import sympy as sp
        omega = sp.Symbol("omega")
        sides, nu, seeds = _members(case, seed)
        dicos = [W.shear_layer(n=n, u0=U0, omega=omega, seed=s) for n, s in zip(sides, seeds)]
        ens = Ensemble(dicos, [{"omega": W.omega_from_nu(float(v))} for v in nu], dtype=case["dtype"])
        return {"case": case, "ens": ens}
    shifted = case["dtype"] != "float64"
    sim = Simulation(_dico(case, seed), dtype=case["dtype"], c0=_reference_state(case) if shifted else None)
    state = {"case": case, "sim": sim, "symbols": (W.RHO, W.QX, W.QY, W.QZ)[:sim.scheme.nconsm]}
    if flow == "learned":
        sim.set_closure(closure.ClosureModel.load(MODEL))
    if case["read"] != "moments":
        state["out"] = pinned_empty((sim.scheme.nconsm,) + tuple(sim.domain.shape_in))
        state["out"][...] = 0.0
    if case["read"] == "restart":
        coords = np.meshgrid(*sim.domain.coords_halo, sparse=True, indexing="ij")
        host = pinned_empty((sim.scheme.nconsm,) + tuple(sim.domain.shape_halo))
        for i, fn in enumerate(_start(case, seed)[0]):
            host[i] = fn(*coords)
        state["in"] = host
    return state


# ------------------------------------------------------------------ the pass
def run(state):
    case = state["case"]
    if case["flow"] == "training":
        mlp = state["mlp"]
        for _ in range(case["steps"] - 1):
            mlp.train_step_device(state["x"], state["t"], case["batch"], lr=1e-4, read_loss=False)
        loss = mlp.train_step_device(state["x"], state["t"], case["batch"], lr=1e-4)
        return {"params": mlp.params_host(), "loss": np.float32(loss)}
    if case["flow"] == "ensemble":
        ens = state["ens"]
        ens.run(case["steps"])
        return [ens.moments(i, keys=range(3)) for i in range(case["count"])]
    sim = state["sim"]
    if case["read"] == "moments":
        for _ in range(case["steps"]):
            sim.one_time_step()
        return [sim.m[s] for s in state["symbols"]]
    if case["read"] == "restart":
        sim.m_halo[0:len(state["symbols"])] = state["in"]
        sim.equilibrium()
        sim.m2f()
    sim.run(case["steps"])
    sim.fields(out=state["out"])
    return state["out"]


# arithmetic of one node's collision (additions and multiplications), D2Q9
# MRT, D2Q9 Geier with relative velocity, D3Q19 MRT
FLOPS = {"mrt2": 130, "geier": 260, "mrt3": 313}


def work(case):
    """Populations (or parameters) read once and written once, host moments
    in and out, and the arithmetic of every step."""
    flow = case["flow"]
    if flow == "training":
        per_sample = 2 * (16 * 64 + 64 * 64 + 64 * 8)
        return {"bytes": case["batch"] * (32 + 32) + 4 * 5768 * 8, "flops": 3 * per_sample * case["batch"] * case["steps"]}
    es = BYTES[case["dtype"]]
    if flow == "ensemble":
        nodes, q, nc, flops = sum(s * s for s in _members(case, 0)[0]), 9, 3, FLOPS["mrt2"]
    elif flow in ("tgv", "cube"):
        nodes, q, nc, flops = case["n"] ** 3, 19, 4, FLOPS["mrt3"]
    elif flow == "disc":
        nodes, q, nc, flops = case["nx"] * case["ny"], 9, 3, FLOPS["mrt2"]
    elif flow == "karman":
        nodes, q, nc, flops = 2 * case["ny"] ** 2, 9, 3, FLOPS["geier"]
    else:
        nodes, q, nc, flops = case["n"] ** 2, 9, 3, FLOPS["mrt2"]
        if flow == "learned":
            flops += 2 * (16 * 64 + 64 * 64 + 64 * 8)
    fields = 8 * nc * nodes
    return {"bytes": 2 * q * es * nodes + fields * (2 if case.get("read") == "restart" else 1),
            "flops": flops * nodes * case["steps"]}


# ------------------------------------------------- the same in 64 bits, on its own
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _grid(shape, length):
    return [((np.arange(n) + 0.5) * (l / n)).reshape([-1 if d == i else 1 for d in range(len(shape))])
            for i, (n, l) in enumerate(zip(shape, length))]


class _Mrt:
    """Multiple-relaxation-time collision: moment polynomials over the
    velocities, equilibria in the conserved moments, rates."""

    def __init__(self, velocities, polynomials, equilibrium, rates, conserved):
        self.v = velocities
        dev = _device()
        m = np.array([[float(p(*v)) for v in velocities] for p in polynomials])
        self.m = torch.tensor(m, dtype=torch.float64, device=dev)
        self.mi = torch.tensor(np.linalg.inv(m), dtype=torch.float64, device=dev)
        self.eq, self.rates, self.conserved = equilibrium, rates, conserved
        self.opposite = [velocities.index(tuple(-c for c in v)) for v in velocities]

    def from_conserved(self, cons):
        return torch.tensordot(self.mi, torch.stack(self.eq(*cons)), dims=1)

    def moments(self, f):
        return torch.tensordot(self.m, f, dims=1)

    def collide(self, f, correct=None):
        m = self.moments(f)
        eq = self.eq(*[m[i] for i in self.conserved])
        before = m.clone() if correct is not None else None
        for i, s in enumerate(self.rates):
            if s:
                m[i] += s * (eq[i] - m[i])
        if correct is not None:
            correct(before, m)
        return torch.tensordot(self.mi, m, dims=1)

    def read(self, f):
        return [self.moments(f)[i] for i in self.conserved]


class _Geier:
    """D2Q9 central-moment collision in the frame of the flow (basis 1, X, Y,
    X^2 + Y^2, X Y^2, X^2 Y, X^2 Y^2, X^2 - Y^2, X Y; product equilibrium)."""

    v = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]
    opposite = list(range(8, -1, -1))

    def __init__(self, rates):
        self.rates = rates

    @staticmethod
    def _central(f, u):
        """Central moments 0, 1, 2 along the leading axis (velocities -1, 0, 1)."""
        lo, mid, hi = f[0] * 1.0, f[1] * 1.0, f[2] * 1.0
        return torch.stack([lo + mid + hi, (-1 - u) * lo - u * mid + (1 - u) * hi,
                            (1 + u) ** 2 * lo + u ** 2 * mid + (1 - u) ** 2 * hi])

    @staticmethod
    def _back(k, u):
        r1 = k[1] + u * k[0]
        r2 = k[2] + 2 * u * k[1] + u * u * k[0]
        return torch.stack([(r2 - r1) / 2, k[0] - r2, (r2 + r1) / 2])

    def _to_populations(self, k, ux, uy):
        g = torch.stack([self._back(k[a], uy) for a in range(3)])
        return self._back(g, ux).reshape(9, *ux.shape)

    def from_conserved(self, cons):
        rho, qx, qy = cons
        z = torch.zeros_like(rho)
        k = torch.stack([torch.stack([rho, z, rho / 3]), torch.stack([z, z, z]), torch.stack([rho / 3, z, rho / 9])])
        return self._to_populations(k, qx / rho, qy / rho)

    def read(self, f):
        g = f.reshape(3, 3, *f.shape[1:])
        return [f.sum(0), (g[2] - g[0]).sum(0), (g[:, 2] - g[:, 0]).sum(0)]

    def collide(self, f):
        rho, qx, qy = self.read(f)
        ux, uy = qx / rho, qy / rho
        k = self._central(f.reshape(3, 3, *f.shape[1:]), ux)
        k = torch.stack([self._central(k[a], uy) for a in range(3)])
        s = self.rates
        plus, minus = k[2, 0] + k[0, 2], k[2, 0] - k[0, 2]
        plus = plus + s[3] * (2 * rho / 3 - plus)
        minus = minus + s[7] * (0 - minus)
        k[2, 0], k[0, 2] = (plus + minus) / 2, (plus - minus) / 2
        k[1, 2] *= 1 - s[4]
        k[2, 1] *= 1 - s[5]
        k[2, 2] += s[6] * (rho / 9 - k[2, 2])
        k[1, 1] *= 1 - s[8]
        return self._to_populations(k, ux, uy)


def _mrt2(omega):
    v = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]
    polys = [lambda x, y: 1, lambda x, y: x, lambda x, y: y, lambda x, y: 3 * (x * x + y * y) - 4,
             lambda x, y: (9 * (x * x + y * y) ** 2 - 21 * (x * x + y * y) + 8) / 2,
             lambda x, y: 3 * x * (x * x + y * y) - 5 * x, lambda x, y: 3 * y * (x * x + y * y) - 5 * y,
             lambda x, y: x * x - y * y, lambda x, y: x * y]

    def eq(r, qx, qy):
        q2 = qx * qx + qy * qy
        return [r, qx, qy, -2 * r + 3 * q2, r - 3 * q2, -qx, -qy, qx * qx - qy * qy, qx * qy]

    return _Mrt(v, polys, eq, RATES_2D + [omega, omega], [0, 1, 2])


def _mrt3(omega):
    v = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if abs(a) + abs(b) + abs(c) < 3]
    polys = [lambda x, y, z, c: 1, lambda x, y, z, c: 19 * c - 30,
             lambda x, y, z, c: (21 * c * c - 53 * c + 24) / 2,
             lambda x, y, z, c: x, lambda x, y, z, c: (5 * c - 9) * x,
             lambda x, y, z, c: y, lambda x, y, z, c: (5 * c - 9) * y,
             lambda x, y, z, c: z, lambda x, y, z, c: (5 * c - 9) * z,
             lambda x, y, z, c: 3 * x * x - c, lambda x, y, z, c: (3 * c - 5) * (3 * x * x - c),
             lambda x, y, z, c: y * y - z * z, lambda x, y, z, c: (3 * c - 5) * (y * y - z * z),
             lambda x, y, z, c: x * y, lambda x, y, z, c: y * z, lambda x, y, z, c: x * z,
             lambda x, y, z, c: (y * y - z * z) * x, lambda x, y, z, c: (z * z - x * x) * y,
             lambda x, y, z, c: (x * x - y * y) * z]
    polys = [(lambda x, y, z, p=p: p(x, y, z, x * x + y * y + z * z)) for p in polys]

    def eq(r, qx, qy, qz):
        j2 = qx * qx + qy * qy + qz * qz
        pxx, pww, zero = 2 * qx * qx - qy * qy - qz * qz, qy * qy - qz * qz, torch.zeros_like(r)
        return [r, -11 * r + 19 * j2, 3 * r - 5.5 * j2, qx, -2 / 3 * qx, qy, -2 / 3 * qy, qz, -2 / 3 * qz,
                pxx, -pxx / 2, pww, -pww / 2, qx * qy, qy * qz, qx * qz, zero, zero, zero]

    e, eps, q, pi, m = 1.2, 1.4, 1.5, 1.6, 1.8
    rates = [0, e, eps, 0, q, 0, q, 0, q, omega, pi, omega, pi, omega, omega, omega, m, m, m]
    return _Mrt(v, polys, eq, rates, [0, 3, 5, 7])


def _omega(nu):
    return 1.0 / (0.5 + 3.0 * nu)


def _start_values(case, seed, shape):
    fns, length = _start(case, seed)
    x = _grid(shape, length)
    return [torch.tensor(np.broadcast_to(np.asarray(fn(*x), dtype=np.float64), shape).copy(), device=_device())
            for fn in fns]


def _periodic(scheme, cons, steps, correct=None):
    f = scheme.from_conserved(cons)
    dims = tuple(range(cons[0].dim()))
    for _ in range(steps):
        f = torch.stack([torch.roll(f[k], v, dims) for k, v in enumerate(scheme.v)])
        f = scheme.collide(f) if correct is None else scheme.collide(f, correct)
    return scheme.read(f)


def _boxed(scheme, cons, steps, lid_axis, u):
    """Bounce-back on every wall of the box; the upper wall of ``lid_axis`` moves along x."""
    f = scheme.from_conserved(cons)
    dim = cons[0].dim()
    one = torch.ones([1] * dim, dtype=torch.float64, device=f.device)
    wall = scheme.from_conserved([one, u * one] + [0 * one] * (dim - 1))
    shape = cons[0].shape
    for _ in range(steps):
        g = torch.empty_like(f)
        for k, v in enumerate(scheme.v):
            r = g[k]
            r.copy_(torch.roll(f[k], v, tuple(range(dim))))
            back = f[scheme.opposite[k]]
            for d in range(dim):
                if v[d]:
                    edge = [slice(None)] * dim
                    edge[d] = slice(0, 1) if v[d] > 0 else slice(shape[d] - 1, shape[d])
                    r[tuple(edge)] = back[tuple(edge)]
            if v[lid_axis] < 0:
                # slots beyond the lid; those beyond a side wall too belong to the
                # wall whose axis comes first
                part = [slice(None)] * dim
                for d in range(dim):
                    if d != lid_axis and v[d]:
                        part[d] = slice(1, None) if v[d] > 0 else slice(0, shape[d] - 1)
                part[lid_axis] = slice(shape[lid_axis] - 1, shape[lid_axis])
                r[tuple(part)] += (wall[k] - wall[scheme.opposite[k]]).reshape(-1)[0]
        f = scheme.collide(g)
    return scheme.read(f)


def _past_disc(scheme, cons, steps, center, radius, channel):
    """Flow past a disc (lattice units) with one ghost layer: inflow on the
    left, Neumann outflow on the right; ``channel``: Bouzidi on the walls, the
    inflow and the disc, else periodic in y, anti-bounce-back inflow and
    bounce-back on the disc."""
    nx, ny = cons[0].shape
    dev = cons[0].device
    one = torch.ones((1, 1), dtype=torch.float64, device=dev)
    inflow = scheme.from_conserved([one, U0 * one, 0 * one]).reshape(-1)
    f = scheme.from_conserved(cons)
    x, y = np.meshgrid(np.arange(nx) + 0.5 - center[0], np.arange(ny) + 0.5 - center[1], indexing="ij")
    solid = x * x + y * y <= radius * radius * (1 + 1e-12)
    links = []
    for k, (a, b) in enumerate(scheme.v):
        if a == 0 and b == 0:
            continue
        # fluid nodes whose neighbour against v_k is solid
        hit = ~solid & np.roll(solid, (a, b), (0, 1))
        i, j = np.nonzero(hit)
        # distance to the disc along -v_k
        px, py = x[i, j], y[i, j]
        c2, c1, c0 = a * a + b * b, -(a * px + b * py), px * px + py * py - radius * radius
        q = (-c1 - np.sqrt(np.maximum(c1 * c1 - c2 * c0, 0.0))) / c2
        links.append((k, a, b, torch.tensor(i, device=dev), torch.tensor(j, device=dev), torch.tensor(q, device=dev)))
    for _ in range(steps):
        g = torch.zeros((9, nx + 2, ny + 2), dtype=torch.float64, device=dev)
        g[:, 1:-1, 1:-1] = f
        if not channel:
            g[:, :, 0], g[:, :, -1] = g[:, :, -2].clone(), g[:, :, 1].clone()
        old = g.clone()
        for k, (a, b) in enumerate(scheme.v):
            o = scheme.opposite[k]
            if channel:
                jump = inflow[k] - inflow[o]
                if b:
                    at = (1, 0) if b > 0 else (ny, ny + 1)
                    i0, i1 = (1, nx + 1)
                    g[k, i0 - a:i1 - a, at[1]] = old[o, i0:i1, at[0]] + jump
                if a > 0:
                    g[k, 0, 1 - b:ny + 1 - b] = old[o, 1, 1:ny + 1] + jump
            elif a > 0:
                g[k, 0, 1 - b:ny + 1 - b] = inflow[k] + inflow[o] - old[o, 1, 1:ny + 1]
        for k, (a, b) in enumerate(scheme.v):
            if a < 0:
                g[k, nx + 1, 1 - b:ny + 1 - b] = g[k, nx, 1 - b:ny + 1 - b]
        for k, a, b, i, j, q in links:
            o = scheme.opposite[k]
            value = old[o, i + 1, j + 1]
            if channel:
                near = 2 * q * value + (1 - 2 * q) * old[o, i + 1 + a, j + 1 + b]
                far = value / (2 * q) + (1 - 1 / (2 * q)) * old[k, i + 1, j + 1]
                value = torch.where(q < 0.5, near, far)
            g[k, i + 1 - a, j + 1 - b] = value
        f = scheme.collide(torch.stack([g[k, 1 - a:nx + 1 - a, 1 - b:ny + 1 - b] for k, (a, b) in enumerate(scheme.v)]))
    return scheme.read(f)


def _network(p, x):
    """The closure network (silu, 16-64-64-8) on rows x."""
    at, parts = 0, []
    for o, i in ((64, 16), (64, 64), (8, 64)):
        parts += [p[at:at + o * i].reshape(o, i), p[at + o * i:at + o * i + o]]
        at += o * i + o
    w1, b1, w2, b2, w3, b3 = parts
    silu = torch.nn.functional.silu
    return silu(silu(x @ w1.T + b1) @ w2.T + b2) @ w3.T + b3


def _closure_correction():
    """The trained closure on the moments around a collision (rate form: the
    network scales each non-conserved moment's own relaxation)."""
    d = np.load(MODEL, allow_pickle=False)
    dev = _device()
    p, norm, rate, guard = (torch.tensor(np.asarray(d[k], dtype=np.float64), device=dev)
                            for k in ("params", "norm", "rate", "guard"))

    def correct(before, after):
        rows = before.reshape(9, -1).T
        x = torch.zeros((rows.shape[0], 16), dtype=torch.float64, device=dev)
        x[:, :9] = (rows - norm[:9]) * norm[16:25]
        z = _network(p, x)[:, :6] * norm[40:46] + norm[32:38]
        change = (after[3:] - before[3:]).reshape(6, -1).T
        extra = (rate[:6] + (rate[8:14] - rate[:6]) * torch.sigmoid(z)) * change
        limit = guard[0] * change.abs().max(dim=1, keepdim=True).values + guard[1]
        extra = torch.where((extra.abs() <= limit).all(dim=1, keepdim=True), extra, torch.zeros_like(extra))
        after[3:] += extra.T.reshape(after[3:].shape)

    return correct


def _trained(case, seed):
    x, t, params = _samples(case, seed)
    dev = _device()
    x = torch.tensor(x, device=dev).to(torch.bfloat16).double()   # the inputs are handed over in BF16
    t = torch.tensor(t.astype(np.float32), device=dev).double()
    p = torch.tensor(params, device=dev).double().requires_grad_()
    opt = torch.optim.Adam([p], lr=1e-4)
    for _ in range(case["steps"]):
        opt.zero_grad()
        loss = ((_network(p, x)[:, :6] - t[:, :6]) ** 2).mean()
        loss.backward()
        opt.step()
    return {"params": p.detach(), "loss": loss.detach().reshape(())}


def exact(case, seed):
    flow = case["flow"]
    if flow == "training":
        return _trained(case, seed)
    if flow == "ensemble":
        if sum(s * s for s in _members(case, seed)[0]) * case["steps"] > 2e9:
            return None   # too long in 64 bits
        out = []
        for n, nu, s in zip(*_members(case, seed)):
            init = W.shear_layer(n=n, u0=U0, seed=s)["init"]
            x = _grid((n, n), (1.0, 1.0))
            cons = [torch.tensor(np.broadcast_to(a, (n, n)).copy(), dtype=torch.float64, device=_device())
                    for a in (np.ones((n, n)), init[W.QX](*x), init[W.QY](*x))]
            out.append(torch.stack(_periodic(_mrt2(_omega(float(nu))), cons, case["steps"])))
        return out
    if flow in ("tgv", "cube"):
        shape = (case["n"],) * 3
        cons = _start_values(case, seed, shape)
        if flow == "tgv":
            got = _periodic(_mrt3(_omega(2e-3)), cons, case["steps"])
        else:
            got = _boxed(_mrt3(_omega(1e-3)), cons, case["steps"], 2, U0)
    elif flow == "disc":
        cons = _start_values(case, seed, (case["nx"], case["ny"]))
        nu = U0 * 2 * case["radius"] / _disc_re(case)
        got = _past_disc(_mrt2(_omega(nu)), cons, case["steps"], _disc_center(case), case["radius"], False)
    elif flow == "karman":
        ny = case["ny"]
        cons = _start_values(case, seed, (2 * ny, ny))
        mu, c = 5.0e-6, 3.0 * ny
        s1, s2 = 1 / (0.5 + c * (10 * mu - 2 * mu / 3)), 1 / (0.5 + c * mu)
        got = _past_disc(_Geier([0, 0, 0, s1, s1, s1, s1, s2, s2]), cons, case["steps"],
                         (0.3 * ny, 0.5 * ny + 2), ny / 32, True)
    else:
        shape = (case["n"],) * 2
        cons = _start_values(case, seed, shape)
        if flow == "cavity":
            got = _boxed(_mrt2(_omega(1e-3)), cons, case["steps"], 1, U0)
        elif flow == "shear":
            got = _periodic(_mrt2(_omega(1e-3)), cons, case["steps"])
        else:
            nu = U0 * case["n"] / 30000.0
            got = _periodic(_mrt2(_omega(nu)), cons, case["steps"], _closure_correction())
    return list(got) if case["read"] == "moments" else torch.stack(got)
