"""The work that a relaxation run has this library do, as cases to measure.

A user's program advances a context in time (``Relax.step``) and reads the
fields at output steps; it runs whole short solves (create, run, read,
destroy); it advances ensembles; and a Fortran host calls the operators one
by one on its own device buffers.  Each listed case is one of these, on a
grid of the benchmark configurations, of the tutorial decks or of a ragged
size (FFT lengths are products of 2 and 3).

    kind "steps"      `steps` time steps of a context, then u, tau, gamma
    kind "solve"      context, coseismic solve, `steps` steps, fields, destroy
    kind "ensemble"   `steps` steps of `members` uneven members, each one's u
    kind "operators"  stressupdate, viscouseigenstress, equivalentbodyforce
                      and the Green's function on device buffers

``exact`` evaluates the same method in 64 bits with plain torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from relax_b200 import _lib
from relax_b200.api import Ensemble, Relax
from relax_b200.config import Event, Fault, Plane, Simulation, ensemble_uneven, relax_layer

TWO_PI = 2.0 * math.pi
GRAVITY = 8.3e-4


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------

def _steps(name, sx, dx, rheology, steps, faults=1, gravity=False, afterslip=False, kind="steps"):
    return {"name": name, "kind": kind, "sx1": sx[0], "sx2": sx[1], "sx3": sx[2], "dx": dx, "rheology": rheology,
            "power": 3.0, "faults": faults, "gravity": gravity, "afterslip": afterslip, "steps": steps}


def listed():
    return [
        # the smallest member shape of the ensembles, on its own: launches and host latency count
        _steps("steps 64x64x64 maxwell", (64, 64, 64), 1.0, "maxwell", 40),
        # the linear Maxwell benchmark box
        _steps("steps 128x128x128 maxwell", (128, 128, 128), 0.8, "maxwell", 40),
        # the headline benchmark: power law with an afterslip plane, adaptive time step
        _steps("steps 256x256x128 afterslip", (256, 256, 128), 0.5, "powerlaw", 40, afterslip=True),
        # the large instance: three faults, gravity, a stress exponent that needs powf
        dict(_steps("steps 512x512x256 gravity", (512, 512, 256), 0.4, "powerlaw", 16, faults=3, gravity=True),
             power=3.5),
        # the tutorials' 256^3 box, power law with gravity
        _steps("steps 256x256x256 gravity", (256, 256, 256), 0.4, "powerlaw", 24, gravity=True),
        # transient (Burgers) rheology on top of the viscous one
        _steps("steps 128x128x128 burgers", (128, 128, 128), 0.8, "burgers", 40),
        # ragged boxes, as chosen to fit a region rather than a power of two
        _steps("steps 108x72x54 powerlaw", (108, 72, 54), 0.9, "powerlaw", 40),
        _steps("steps 288x216x144 powerlaw", (288, 216, 144), 0.5, "powerlaw", 20, faults=2, gravity=True),
        # one short solve from a deck to its fields (parameter sweeps, inversions)
        _steps("solve 96x96x64 maxwell", (96, 96, 64), 1.0, "maxwell", 10, kind="solve"),
        # an uneven ensemble: members of 64^3, 128^2 x 64, 128^3 and 192^2 x 96
        {"name": "ensemble of 16", "kind": "ensemble", "members": 16, "steps": 10},
        # the operators, as a Fortran host calls them for one stress and velocity evaluation
        {"name": "operators 128x128x128", "kind": "operators", "sx1": 128, "sx2": 128, "sx3": 128, "dx": 0.8,
         "power": 3.0, "gravity": True},
        {"name": "operators 72x48x36", "kind": "operators", "sx1": 72, "sx2": 48, "sx3": 36, "dx": 1.0,
         "power": 1.0, "gravity": False},
    ]


def _lengths(lo, hi, multiple=1):
    """The products of 2 and 3 in [lo, hi]."""
    both = sorted(2 ** a * 3 ** b for a in range(12) for b in range(8))
    return [n for n in both if lo <= n <= hi and n % multiple == 0]


def _length(rng, lo, hi, multiple=1):
    """A product of 2 and 3, log-uniform over [lo, hi]."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_lengths(lo, hi, multiple), key=lambda n: abs(math.log(n / want)))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "solve", "ensemble", "operators"])
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 16), "steps": rng.randint(4, 10)}
    # sx1 / 2 is the FFT length along x1: sx1 a multiple of 4
    sx1, sx2 = _length(rng, 32, 512, 4), _length(rng, 24, 512)
    sx3 = _length(rng, 24, 256, 2)
    dx = round(rng.uniform(0.4, 1.2), 2)
    gravity = rng.random() < 0.5
    if kind == "operators":
        return {"kind": kind, "sx1": min(sx1, 256), "sx2": min(sx2, 256), "sx3": min(sx3, 144), "dx": dx,
                "power": rng.choice([1.0, 3.0, 3.5]), "gravity": gravity}
    rheology = rng.choice(["maxwell", "powerlaw", "powerlaw", "burgers"])
    c = _steps("", (sx1, sx2, sx3), dx, rheology, rng.randint(6, 12) if sx1 * sx2 * sx3 > 1 << 24 else rng.randint(8, 40),
               faults=rng.randint(1, 3), gravity=gravity, afterslip=rng.random() < 0.3, kind=kind)
    del c["name"]
    c["power"] = rng.choice([2.0, 3.0, 3.5])
    return c


# --------------------------------------------------------------------------
# decks and inputs, from the seed alone
# --------------------------------------------------------------------------

def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7fffffff, case.get("sx1", 0), case.get("sx3", 0)])


def _lid(case):
    """Depth of the top of the viscous substrate, on a grid plane."""
    return round(0.35 * (case["sx3"] // 2)) * case["dx"]


def _rheology(case, seed):
    """{mechanism: (fluidity, stress exponent, Gk)} below the lid."""
    g = float(10.0 ** _rng(case, seed + 1).uniform(-0.3, 0.3))
    if case["rheology"] == "maxwell":
        return {"linear": (g, 1.0, 0.0)}
    if case["rheology"] == "powerlaw":
        return {"nonlinear": (g, case["power"], 0.0)}
    return {"linear": (0.5 * g, 1.0, 0.0), "ltransient": (g, 1.0, 0.5)}


def _faults(case, seed):
    """Faults (slip, x, y, z, length, width, strike, dip, rake) around the
    box's centre, slip about 3 dx (lognormal, sigma 0.3)."""
    rng = _rng(case, seed)
    dx, depth = case["dx"], case["dx"] * case["sx3"] / 2
    side = dx * min(case["sx1"], case["sx2"])
    out = []
    for _ in range(case["faults"]):
        length = max(4.0 * dx, min(side, 4.0 * depth) * float(rng.uniform(0.15, 0.35)))
        width = max(3.0 * dx, min(0.5 * length, 0.5 * depth))
        slip = 3.0 * dx * float(np.exp(rng.normal(0.0, 0.3)))
        strike = float(rng.uniform(0.0, 360.0))
        a = math.radians(strike)
        x, y = float(rng.uniform(-0.1, 0.1)) * side, float(rng.uniform(-0.1, 0.1)) * side
        dip, rake = ((90.0, 0.0), (float(rng.uniform(20.0, 60.0)), 90.0))[int(rng.integers(2))]
        out.append((slip, x - 0.5 * length * math.cos(a), y - 0.5 * length * math.sin(a),
                    float(rng.uniform(0.5, 2.0)) * dx, length, width, strike, dip, rake))
    return out


def _plane(case, seed):
    """One afterslip plane on the first fault's lower edge, continuing down
    its dip, with a free rake."""
    if not case["afterslip"]:
        return None
    _, x, y, z, length, width, strike, dip, _ = _faults(case, seed)[0]
    a, b = math.radians(strike), math.radians(dip)
    return (x - width * math.cos(b) * math.sin(a), y + width * math.cos(b) * math.cos(a), z + width * math.sin(b),
            length, 0.5 * width, strike, dip, 900.0)


def _deck(case, seed):
    r, lid = _rheology(case, seed), _lid(case)
    plane = _plane(case, seed)
    return Simulation(
        sx1=case["sx1"], sx2=case["sx2"], sx3=case["sx3"], dx1=case["dx"], dx2=case["dx"], dx3=case["dx"], beta=0.2,
        nyquist=2.0, lambda_=1.0, mu=1.0, gam=GRAVITY if case["gravity"] else 0.0, interval=1.0e30, odt=-1, tscale=1.0,
        linear=[(lid, r["linear"][0])] if "linear" in r else [],
        nonlinear=[(lid, r["nonlinear"][0], r["nonlinear"][1], 0.0)] if "nonlinear" in r else [],
        ltransient=[(lid, r["ltransient"][0], r["ltransient"][2])] if "ltransient" in r else [],
        faultcreep=[(0.0, 1.0, 2.0, 0.0, 0.0)] if plane else [], planes=[Plane(*plane)] if plane else [],
        events=[Event(0.0, [Fault(*f) for f in _faults(case, seed)])], name="deck")


def _members(case, seed):
    """The first members of the uneven ensemble (their grids, lids and
    exponents), with slip and fluidity drawn from the seed."""
    rng = _rng(case, seed)
    sims = ensemble_uneven(seed=4, n=case["members"])
    for s in sims:
        depth, g0, n, coh = s.nonlinear[0]
        s.nonlinear = [(depth, g0 * float(10.0 ** rng.uniform(-0.2, 0.2)), n, coh)]
        s.events[0].faults[0].slip *= float(np.exp(rng.normal(0.0, 0.2)))
        s.interval = 1.0e30
    return sims


def _host(shape):
    """A page-locked host buffer to read a field into."""
    return torch.zeros(shape, dtype=torch.float32, pin_memory=torch.cuda.is_available())


def _outputs(sim):
    return {"u": _host(sim.vec_shape()), "tau": _host(sim.tensor_shape() + (6,)), "gamma": _host(sim.vec_shape()[1:])}


def _smooth(rng, shape, dev, n=24):
    """n random plane waves, decaying with depth: (components, z, y, x)."""
    nc, nz, ny, nx = shape
    z, y, x = (torch.arange(m, device=dev, dtype=torch.float32) for m in (nz, ny, nx))
    out = torch.zeros(shape, device=dev)
    for c in range(nc):
        for _ in range(n // nc):
            kx, ky = int(rng.integers(0, max(2, nx // 8))), int(rng.integers(0, max(2, ny // 8)))
            amp, ph, dec = float(rng.normal()), float(rng.uniform(0, TWO_PI)), float(rng.uniform(1.0, 4.0))
            wave = torch.cos(TWO_PI * (kx * x[None, :] / nx + ky * y[:, None] / ny) + ph)
            out[c] += amp * torch.exp(-dec * z / nz)[:, None, None] * wave[None]
    return out


def _operator_inputs(case, seed, dev):
    """Displacement (3, z, y, x) and stored stress (z, y, x, 6), and the
    substrate's fluidity per layer."""
    rng = _rng(case, seed)
    nz, ny, nx = case["sx3"] // 2, case["sx2"], case["sx1"]
    u = _smooth(rng, (3, nz, ny, nx), dev)
    tau = 0.1 * _smooth(rng, (6, nz, ny, nx), dev).permute(1, 2, 3, 0).contiguous()
    return u, tau, 10.0 ** rng.uniform(-0.3, 0.3, nz)


def _pad(u):
    return torch.nn.functional.pad(u, (0, 2)).contiguous()


# --------------------------------------------------------------------------
# preparation and one pass
# --------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "solve":
        sim = _deck(case, seed)
        return {"case": case, "sim": sim, "out": _outputs(sim)}
    if case["kind"] == "steps":
        sim = _deck(case, seed)
        r = Relax(sim)
        r.coseismic()
        return {"case": case, "r": r, "out": _outputs(sim)}
    if case["kind"] == "ensemble":
        sims = _members(case, seed)
        e = Ensemble(sims)
        e.coseismic()
        return {"case": case, "e": e, "members": [e.member(k) for k in range(e.n)],
                "out": [_host(s.vec_shape()) for s in sims]}
    nz, ny, nx = case["sx3"] // 2, case["sx2"], case["sx1"]
    u, tau, fluidity = _operator_inputs(case, seed, "cuda")
    layers = (relax_layer * nz)(*[relax_layer(z=0.0, gammadot0=float(g), stressexponent=case["power"], cohesion=0.0,
                                              friction=0.0, Gk=0.0) for g in fluidity])
    return {"case": case, "u": _pad(u), "tau": tau, "layers": layers, "sig": torch.empty_like(tau),
            "moment": torch.empty_like(tau), "c": torch.empty((3, case["sx3"], ny, nx + 2), device="cuda"),
            "t": torch.empty((3, ny, nx + 2), device="cuda")}


def _log_row(t):
    """Dt, time, power and C:E of a step's log."""
    return (t[1], t[5], t[6], t[7])


def _read(r, out):
    for name, buf in out.items():
        r.field_into(name, buf)
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "steps":
        r = state["r"]
        log = [_log_row(r.step()) for _ in range(case["steps"])]
        return dict(_read(r, state["out"]), log=np.array(log, np.float32))
    if case["kind"] == "solve":
        with Relax(state["sim"]) as r:
            log = [_log_row(t) for t in r.run(case["steps"])[1:]]
            return dict(_read(r, state["out"]), log=np.array(log, np.float32))
    if case["kind"] == "ensemble":
        log = [[_log_row(t) for t in state["e"].step()] for _ in range(case["steps"])]
        for m, buf in zip(state["members"], state["out"]):
            m.field_into("u", buf)
        return {"u": state["out"], "log": np.array(log, np.float32)}
    return _run_operators(state, case)


def _run_operators(s, case):
    """sig = -tau + C:E(u); m = eigenstress(sig); c = -div m; c = G c."""
    lib, st = _lib.load(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    sx1, sx2, sx3, dx = case["sx1"], case["sx2"], case["sx3"], case["dx"]
    ptr = [C.c_void_p(s["u"][k].data_ptr()) for k in range(3)]
    c = [C.c_void_p(s["c"][k].data_ptr()) for k in range(3)]
    t = [C.c_void_p(s["t"][k].data_ptr()) for k in range(3)]
    sig, mom = C.c_void_p(s["sig"].data_ptr()), C.c_void_p(s["moment"].data_ptr())
    torch.neg(s["tau"], out=s["sig"])
    for name in ("moment", "c", "t"):
        s[name].zero_()
    tm = C.c_double(1.0e7)
    _lib.check(lib.relax_op_stressupdate(*ptr, 1.0, 1.0, dx, dx, dx, sx1, sx2, sx3 // 2, sig, st))
    _lib.check(lib.relax_op_viscouseigenstress(1.0, C.cast(s["layers"], C.c_void_p), None, sig, sx1, sx2, sx3 // 2, mom,
                                               C.byref(tm), None, None, st))
    _lib.check(lib.relax_op_bodyforce(mom, dx, dx, dx, sx1, sx2, sx3 // 2, *c, *t, st))
    _lib.check(lib.relax_op_green(*c, *t, sx1, sx2, sx3, dx, dx, dx, 1.0, 1.0, GRAVITY if case["gravity"] else 0.0, st))
    return {"sig": s["sig"], "moment": s["moment"], "c": s["c"], "tm": np.array([tm.value], np.float32)}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _green_flops(sx1, sx2, sx3):
    n = sx1 * sx2 * sx3
    return 6 * 2.5 * n * math.log2(n)


def _step_work(sx1, sx2, sx3, steps, burgers=False):
    """The state (u, tau, gamma; epsilonik) read and written once a step."""
    nh = sx1 * sx2 * (sx3 // 2)
    return steps * nh * 8.0 * (16 if burgers else 10), steps * (2 * _green_flops(sx1, sx2, sx3) + 400.0 * nh)


def work(case):
    if case["kind"] == "ensemble":
        parts = []
        for s in ensemble_uneven(seed=4, n=case["members"]):
            b, f = _step_work(s.sx1, s.sx2, s.sx3, case["steps"])
            parts.append((b + 12.0 * s.sx1 * s.sx2 * s.sx3h, f))
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    sx = case["sx1"], case["sx2"], case["sx3"]
    nh = sx[0] * sx[1] * (sx[2] // 2)
    if case["kind"] == "operators":
        # u, tau, sig, moment once, the body force (half box) and the displacement (whole box) once
        return {"bytes": nh * 4.0 * (3 + 6 + 6 + 6 + 3 + 6), "flops": _green_flops(*sx) + 300.0 * nh}
    b, f = _step_work(*sx, case["steps"], case["rheology"] == "burgers")
    return {"bytes": b + 40.0 * nh, "flops": f}


# --------------------------------------------------------------------------
# the same method in 64 bits
# --------------------------------------------------------------------------

class _Grid:
    """Coordinates, wavenumbers and operators of one box in 64 bits; fields
    are (components, z, y, x), the physical half-space nz = sx3/2 layers."""

    def __init__(self, sx, dx, lam, mu, gam, dev):
        self.sx1, self.sx2, self.sx3 = sx
        self.nz = self.sx3 // 2
        self.dx, self.lam, self.mu, self.gam, self.dev = dx, lam, mu, gam, dev
        self.k1 = torch.arange(self.sx1 // 2 + 1, device=dev, dtype=torch.float64) / (self.sx1 * dx)
        self.k2, self.k3 = (self._wave(n) for n in (self.sx2, self.sx3))

    def _wave(self, n):
        i = torch.arange(n, device=self.dev, dtype=torch.float64)
        return torch.where(i < n // 2, i, i - n) / (n * self.dx)

    def points(self):
        """(x3, x2, x1) of the physical points, origin at the box's corner 0."""
        def axis(n):
            i = torch.arange(n, device=self.dev, dtype=torch.float64)
            return torch.where(i < n // 2, i, i - n) * self.dx
        x3 = torch.arange(self.nz, device=self.dev, dtype=torch.float64) * self.dx
        return x3[:, None, None], axis(self.sx2)[None, :, None], axis(self.sx1)[None, None, :]

    def d1(self, f):
        return (torch.roll(f, -1, -1) - torch.roll(f, 1, -1)) * (0.5 / self.dx)

    def d2(self, f):
        return (torch.roll(f, -1, -2) - torch.roll(f, 1, -2)) * (0.5 / self.dx)

    def d3(self, f):
        out = torch.empty_like(f)
        out[1:-1] = (f[2:] - f[:-2]) * (0.5 / self.dx)
        out[0] = (f[1] - f[0]) / self.dx
        out[-1] = (f[-1] - f[-2]) / self.dx
        return out

    def hooke(self, u):
        """C:E(u), components 11 12 13 22 23 33."""
        e11, e22, e33 = self.d1(u[0]), self.d2(u[1]), self.d3(u[2])
        tr = self.lam * (e11 + e22 + e33)
        mu = self.mu
        return torch.stack([2 * mu * e11 + tr, mu * (self.d1(u[1]) + self.d2(u[0])),
                            mu * (self.d1(u[2]) + self.d3(u[0])), 2 * mu * e22 + tr,
                            mu * (self.d2(u[2]) + self.d3(u[1])), 2 * mu * e33 + tr])

    def body_force(self, m):
        """(-div m, traction m_i3 at the surface)."""
        rows = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
        f = torch.stack([-(self.d1(m[a]) + self.d2(m[b]) + self.d3(m[c])) for a, b, c in rows])
        return f, torch.stack([m[2][0], m[4][0], m[5][0]])

    def green(self, f, t, full=False):
        """Displacement of a body force (physical layers; zero below) and a
        surface traction: elastic response, surface traction (gravity
        included) and its Cerruti correction."""
        dx, n3, lam, mu = self.dx, self.sx3, self.lam, self.mu
        box = torch.zeros((3, n3, self.sx2, self.sx1), dtype=torch.float64, device=self.dev)
        box[:, :f.shape[1]] = f
        c = torch.fft.rfftn(box, dim=(1, 2, 3)) * dx ** 3
        del box
        p = torch.fft.rfftn(t, dim=(1, 2)) * dx ** 2
        k1, k2, k3 = self.k1[None, None, :], self.k2[None, :, None], self.k3[:, None, None]
        r2 = k1 ** 2 + k2 ** 2 + k3 ** 2
        inv = torch.where(r2 > 0, 1.0 / torch.where(r2 > 0, r2, 1.0), 0.0)
        ratio1 = (lam + mu) / (lam + 2 * mu) / mu / (4 * math.pi ** 2)
        ratio2 = mu / (lam + mu)
        kc = (k1 * c[0] + k2 * c[1] + k3 * c[2]) * (ratio1 * inv * inv)
        c *= (ratio1 * (1 + ratio2)) * inv
        for i, k in enumerate((k1, k2, k3)):
            c[i] -= k * kc
        del kc, inv, r2
        alpha = (lam + mu) / (lam + 2 * mu)
        grav = 2 * mu * alpha * self.gam
        d = n3 * dx
        i2pi = 1j * TWO_PI
        p[0] -= (i2pi * mu * (k3 * c[0] + k1 * c[2])).sum(0) / d
        p[1] -= (i2pi * mu * (k3 * c[1] + k2 * c[2])).sum(0) / d
        p[2] -= (i2pi * ((lam + 2 * mu) * k3 * c[2] + lam * (k1 * c[0] + k2 * c[1])) - grav * c[2]).sum(0) / d
        k1, k2 = k1[0], k2[0]
        beta = TWO_PI * torch.sqrt(k1 ** 2 + k2 ** 2)
        on = beta > 0
        beta = torch.where(on, beta, 1.0)
        b1, b2 = (torch.where(on, q, 0.0) / (2 * mu * beta ** 3) for q in (p[0], p[1]))
        q = TWO_PI * (k1 * p[0] + k2 * p[1])
        b3 = torch.where(on, beta * p[2] - 1j * (1 - alpha) * q, 0.0) / \
            (2 * alpha * mu * beta ** 4 * (1 + self.gam / beta))
        bq = b1 * k1 + b2 * k2
        fi = 2 * beta / ((TWO_PI * k3) ** 2 + beta ** 2)
        g = TWO_PI * k3 * fi
        h = alpha * 1j * beta * TWO_PI * b3 * (1 - 1 / alpha - 1j * g) + alpha * TWO_PI ** 2 * bq * (1 - 1j * g)
        c[0] += fi * (k1 * h - 2 * beta ** 2 * b1)
        c[1] += fi * (k2 * h - 2 * beta ** 2 * b2)
        c[2] += fi * (-alpha * beta ** 2 * b3 * (1 / alpha - 1j * g) + alpha * beta * TWO_PI ** 2 * k3 * fi * bq)
        del h
        u = torch.fft.irfftn(c, s=(n3, self.sx2, self.sx1), dim=(1, 2, 3)) / dx ** 3
        return u if full else u[:, :self.nz].contiguous()


def _norm(s):
    return torch.sqrt(0.5 * (s[0] ** 2 + 2 * s[1] ** 2 + 2 * s[2] ** 2 + s[3] ** 2 + 2 * s[4] ** 2 + s[5] ** 2))


def _deviator(s):
    tr = (s[0] + s[3] + s[5]) / 3.0
    d = s.clone()
    for i in (0, 3, 5):
        d[i] -= tr
    return d


def _eigenstress(s, fluidity, power, mu):
    """(2 gd s', gd |s'|/mu, min 1/gd) of a viscous mechanism."""
    d = _deviator(s)
    x = _norm(d) / mu
    gd = fluidity * x ** (power - 1.0)
    top = float(gd.max())
    return 2.0 * gd * d, gd * x, 1.0 / top if top > 0 else 3.0e38


def _internal(g):
    """Upper end of the top edge, degrees -> centre, radians (wangconvention)."""
    slip, x, y, z, length, width, strike, dip, rake = g
    a, b = math.radians(-90.0 - strike), math.radians(90.0 - dip)
    return (-slip, x - 0.5 * length * math.sin(a) + 0.5 * width * math.sin(b) * math.cos(a),
            y - 0.5 * length * math.cos(a) - 0.5 * width * math.sin(b) * math.sin(a), z + 0.5 * width * math.cos(b),
            length, width, a, b, math.radians(rake))


def _gauss(x, s):
    return torch.exp(-0.5 * (x / s) ** 2) / math.sqrt(TWO_PI) / s


def _taper(x, beta, derivative=False):
    """The cosine-tapered boxcar omega, or its derivative."""
    ax = x.abs()
    edge = (ax > (1 - 2 * beta) / (1 - beta) / 2) & (ax < 1 / (1 - beta) / 2)
    ph = math.pi * ((1 - beta) * ax - 0.5 + beta) / beta
    if derivative:
        return torch.where(edge, -torch.sign(x) * math.pi * (1 - beta) / 2 / beta * torch.sin(ph), 0.0)
    return torch.where(edge, torch.cos(0.5 * ph) ** 2, torch.where(ax < 0.5 / (1 - beta), 1.0, 0.0))


class _Patch:
    """A rectangular source in its own frame and in its image's."""

    def __init__(self, g, geometry, beta=0.2, surface=False):
        self.slip, x, y, z, self.W, self.L, strike, dip, rake = _internal(geometry)
        self.dx, self.beta = g.dx, beta
        cs, ss, cd, sd = math.cos(strike), math.sin(strike), math.cos(dip), math.sin(dip)
        self.cr, self.sr = math.cos(rake), math.sin(rake)
        self.cs, self.ss, self.cd, self.sd, self.dip = cs, ss, cd, sd, dip
        x3, x2, x1 = g.points()
        x3 = x3[:1] if surface else x3
        c2 = cs * x - ss * y
        xr, yr, zr = cd * c2 - sd * z, ss * x + cs * y, sd * c2 + cd * z
        x2r = cs * x1 - ss * x2
        self.n, self.ni = cd * x2r - sd * x3 - xr, cd * x2r + sd * x3 - xr
        self.a = ss * x1 + cs * x2 - yr
        self.d, self.di = sd * x2r + cd * x3 - zr, -sd * x2r + cd * x3 + zr
        self.wp, self.lp = (q * (1 + 2 * beta) / 2 for q in (self.W, self.L))
        self.near = ~(((x3 - z).abs() > self.lp) & ((x3 + z).abs() > self.lp))
        self.above = (x3 - z).abs() <= self.lp
        self.off1, self.off2 = (x1 - x).abs(), (x2 - y).abs()
        self.normal = (cd * cs, -cd * ss, -sd)
        self.rake = (ss * self.cr + cs * sd * self.sr, cs * self.cr - ss * sd * self.sr, cd * self.sr)

    def band(self, cut):
        return ~((self.n.abs() > cut * self.dx) & (self.ni.abs() > cut * self.dx))

    def column(self):
        m = max(self.wp, self.lp)
        return (self.off1 <= m) & (self.off2 <= m)

    def box(self):
        return self.near & self.column()

    def impulse(self):
        along = _taper(self.a / self.W, self.beta)
        return along * (_gauss(self.n, self.dx) * _taper(self.d / self.L, self.beta) +
                        _gauss(self.ni, self.dx) * _taper(self.di / self.L, self.beta))

    def force(self, mu):
        """Equivalent body force of the shear dislocation (3 components)."""
        s = -mu * self.slip
        dx, b = self.dx, self.beta
        def prime(x):
            return -x * torch.exp(-0.5 * (x / dx) ** 2) / math.sqrt(TWO_PI) / dx ** 3
        along, along1 = _taper(self.a / self.W, b), _taper(self.a / self.W, b, True)
        down, downi = _taper(self.d / self.L, b), _taper(self.di / self.L, b)
        src, img = s * prime(self.n) * along * down, s * prime(self.ni) * along * downi
        cpl = s / self.W * _gauss(self.n, dx) * along1 * down
        cpli = s / self.W * _gauss(self.ni, dx) * along1 * downi
        dcs = s / self.L * _gauss(self.n, dx) * along * _taper(self.d / self.L, b, True)
        cr, sr, cs, ss, cd, sd = self.cr, self.sr, self.cs, self.ss, self.cd, self.sd
        shallow = math.radians(2.01) > self.dip
        q, w, v = (src + img, cpl + cpli, cpl - cpli) if shallow else (src, cpl, cpl)
        f = torch.stack([cr * ss * q + cr * cd * cs * w + cd * sr * cs * dcs + sd * sr * cs * src,
                         cr * cs * q - cr * cd * ss * w - cd * sr * ss * dcs - sd * sr * ss * src,
                         -cr * sd * v + cd * sr * src - sd * sr * dcs])
        return f * (self.box() & self.band(7.01))

    def dyad(self, weight, amount):
        """Symmetric normal x slip tensor times a weight field."""
        n, r = self.normal, self.rake
        e = [0.5 * (n[i] * r[j] + n[j] * r[i]) for i, j in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
        return torch.stack([amount * v * weight for v in e])

    def traction(self, mu):
        t = self.dyad(self.impulse() * (self.column() & self.band(7.01)), mu * self.slip)
        return torch.stack([t[2][0], t[4][0], t[5][0]])

    def moment(self, mu):
        on = self.above & (self.off1 <= self.wp) & (self.off2 <= self.wp) & self.band(7.01)
        return self.dyad(self.impulse() * on, 2.0 * mu * self.slip)

    def creep(self, sig, v0, ab, mu):
        """(eigenstress rate, Maxwell time) of rate-strengthening friction
        with a free rake; no coefficient of friction, no cohesion."""
        on = self.box() & self.band(7.01)
        n = self.normal
        t = [sig[0] * n[0] + sig[1] * n[1] + sig[2] * n[2], sig[1] * n[0] + sig[3] * n[1] + sig[4] * n[2],
             sig[2] * n[0] + sig[4] * n[1] + sig[5] * n[2]]
        tn = t[0] * n[0] + t[1] * n[1] + t[2] * n[2]
        t = [q - tn * m for q, m in zip(t, n)]
        ts = torch.sqrt(t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
        gd = v0 * 2.0 * torch.sinh(torch.clamp(ts / ab, max=11.0))
        b = torch.where(on, 2.0 * mu * self.impulse() * gd / ts, 0.0)
        pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
        m = torch.stack([0.5 * b * (t[i] * n[j] + t[j] * n[i]) for i, j in pairs])
        tm = torch.where(on, ts / mu / gd * (min(self.L, self.W) / self.dx), 3.0e38)
        return m, float(tm.min())


class _Solve:
    """The relaxation in 64 bits: coseismic solve, then RK2 steps."""

    def __init__(self, sx, dx, lam, mu, gam, faults, mechanisms, dev, plane=None):
        """mechanisms: {"linear" | "nonlinear" | "ltransient": (fluidity, power, Gk, top depth)}"""
        self.g = g = _Grid(sx, dx, lam, mu, gam, dev)
        self.mu, self.mech = mu, []
        for name in ("linear", "nonlinear", "ltransient"):
            if name in mechanisms:
                flu, power, gk, lid = mechanisms[name]
                z = torch.arange(g.nz, device=dev)
                self.mech.append((name, torch.where(z >= round(lid / dx), flu, 0.0).double()[:, None, None], power, gk))
        f = torch.zeros((3, g.nz, g.sx2, g.sx1), dtype=torch.float64, device=dev)
        t = torch.zeros((3, g.sx2, g.sx1), dtype=torch.float64, device=dev)
        self.tau = torch.zeros((6,) + f.shape[1:], dtype=torch.float64, device=dev)
        for geometry in faults:
            p = _Patch(g, geometry)
            f += p.force(mu)
            self.tau += p.moment(mu)
            t += _Patch(g, geometry, surface=True).traction(mu)
        self.plane = None
        if plane is not None:   # the plane's rake is reversed on input, 0 slip
            self.plane = _Patch(g, (0.0,) + plane[:7] + (plane[7] - 180.0,))
        self.u = g.green(f, t)
        self.gamma = torch.zeros_like(self.u[0])
        self.eps = torch.zeros_like(self.tau)
        self.epsdot = None
        self.t, self.log = 0.0, []
        self.sig = g.hooke(self.u) - self.tau

    def rates(self, sig, eps, corrector=False):
        """(moment rate, gamma rate, Maxwell time, transient strain rate)."""
        m, gd, inv, rate = torch.zeros_like(sig), torch.zeros_like(sig[0]), 0.0, None
        for name, flu, power, gk in self.mech:
            if name == "ltransient":
                q = _deviator(sig) - 2.0 * gk * eps
                g = flu * (_norm(q) / self.mu) ** (power - 1.0)
                rate = g / self.mu * q
                m += 2.0 * g * q
                inv += float(g.max())
            else:
                dm, dg, tm = _eigenstress(sig, flu, power, self.mu)
                m += dm
                gd += dg
                inv += 1.0 / min(1.0e7, tm)
        if self.plane is not None:
            dm, tm = self.plane.creep(sig, 1.0, 2.0, self.mu)
            m += dm
            inv += 1.0 / min(1.0e7, tm)
        return m, gd, 1.0 / inv, rate

    def step(self):
        g = self.g
        m, _, tm, rate = self.rates(self.sig, self.eps)
        dt = min(tm, 1.0e7) / 10.0
        v = self.u + 0.5 * dt * g.green(*g.body_force(m))
        sig = g.hooke(v) - self.tau - 0.5 * dt * m
        eps = self.eps + 0.5 * dt * rate if rate is not None else self.eps
        m, gd, _, rate = self.rates(sig, eps)
        del sig, v
        self.gamma += dt * gd
        if rate is not None:
            self.eps = self.eps + dt * rate
        self.u = self.u + dt * g.green(*g.body_force(m))
        self.tau = self.tau + dt * m
        self.sig = g.hooke(self.u) - self.tau
        self.t += dt
        dv = g.dx ** 3
        self.log.append((dt, self.t, float(_norm(m).sum()) * dv, float(_norm(self.tau).sum()) * dv))


def _single(v):
    """A layer's parameter as the library holds it."""
    return float(np.float32(v))


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "operators":
        return _exact_operators(case, seed, dev)
    if case["kind"] == "ensemble":
        us, logs = [], []
        for s in _members(case, seed):
            depth, g0, n, _ = s.nonlinear[0]
            fs = [(f.slip, f.x, f.y, f.z, f.length, f.width, f.strike, f.dip, f.rake) for f in s.events[0].faults]
            # an interface acts from the grid plane nearest to its depth (a tie rounds down)
            lid = math.ceil(depth / s.dx1 - 0.5) * s.dx1
            q = _Solve((s.sx1, s.sx2, s.sx3), s.dx1, 1.0, 1.0, 0.0, fs,
                       {"nonlinear": (_single(g0), _single(n), 0.0, lid)}, dev)
            for _ in range(case["steps"]):
                q.step()
            us.append(_pad(q.u))
            logs.append(q.log)
        return {"u": us, "log": np.array(logs).transpose(1, 0, 2)}
    mech = {k: (_single(v[0]), v[1], v[2], _lid(case)) for k, v in _rheology(case, seed).items()}
    q = _Solve((case["sx1"], case["sx2"], case["sx3"]), case["dx"], 1.0, 1.0, GRAVITY if case["gravity"] else 0.0,
               _faults(case, seed), mech, dev, _plane(case, seed))
    for _ in range(case["steps"]):
        q.step()
    return {"u": _pad(q.u), "tau": q.tau.permute(1, 2, 3, 0).contiguous(), "gamma": _pad(q.gamma),
            "log": np.array(q.log)}


def _exact_operators(case, seed, dev):
    u, tau, fluidity = _operator_inputs(case, seed, dev)
    g = _Grid((case["sx1"], case["sx2"], case["sx3"]), case["dx"], 1.0, 1.0, GRAVITY if case["gravity"] else 0.0, dev)
    sig = g.hooke(u.double()) - tau.double().permute(3, 0, 1, 2)
    flu = torch.tensor([_single(f) for f in fluidity], dtype=torch.float64, device=dev)[:, None, None]
    m, _, tm = _eigenstress(sig, flu, case["power"], 1.0)
    c = g.green(*g.body_force(m), full=True)
    return {"sig": sig.permute(1, 2, 3, 0).contiguous(), "moment": m.permute(1, 2, 3, 0).contiguous(), "c": _pad(c),
            "tm": np.array([min(tm, 1.0e7)])}
