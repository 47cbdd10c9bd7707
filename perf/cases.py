"""Performance cases of the Allen-Cahn phase-field LBM solver.

Every case goes through the package's public surface (``FEConfig``,
``AllenCahnSolver``, ``AllenCahnBatch``, ``measure_spread_factor``), as the
sweep, serving and verification drivers use it.  One pass of

  kind "step"   advances a solver that the program keeps by ``steps`` time
                steps in one ``run`` call and reads phi and u, as a driver does
                at its check points (``loop``: through one ``step()`` call per
                time step, as the reference's scripts do);
  kind "batch"  the same for ``count`` grids of different extents, substrates
                and contact angles in one ``AllenCahnBatch``;
  kind "watch"  takes a few steps and then reads everything a monitored run looks
                at: the six fields, both populations, the device diagnostics;
  kind "solve"  is a whole solve from host arrays: construct, ``set_solid``,
                ``init_fields``, ``steps`` steps, phi back to the host and the
                spread diagnostics.

Inputs are droplets with a tanh profile and an impact velocity above a flat,
ridge, convex or concave substrate with a smooth solid fraction, at the
parameters of the impact sweep (density ratio 828, xi = 4, tau = 0.53), each
seed with its own droplet and substrate.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pytorch-lbm_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from lbm.batch import AllenCahnBatch  # noqa: E402
from lbm.fe_ac_solver import AllenCahnSolver  # noqa: E402
from lbm.fe_config import FEConfig  # noqa: E402
from lbm.fe_measure import measure_spread_factor  # noqa: E402

_DEV = "cuda"
_DTYPES = {"float32": torch.float32, "float64": torch.float64, "float16": torch.float16}
_SUBSTRATES = ("flat", "ridge", "convex", "concave")
# extents of the impact sweep's and the serving loop's grids
_SWEEP = ((96, 96, 96), (128, 128, 96), (150, 150, 107), (192, 192, 128))


def _case(name, kind="step", grid=(0, 0, 0), substrate="ridge", theta=162.0, dtype="float32", steps=5, **more):
    c = {"kind": kind, "nx": grid[0], "ny": grid[1], "nz": grid[2], "substrate": substrate, "theta": theta,
         "dtype": dtype, "steps": steps, "tau_h": 1.0, "tau_g": 0.53, "interface": "allen-cahn", "loop": False,
         "count": 1}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one step() of the 24x24x20 flat-wall droplet, where launches and the host count
        _case("step_24", grid=(24, 24, 20), substrate="flat", theta=120.0, steps=1, loop=True),
        # the reference's validation script: an 80x80x65 ridge impact stepped one step() at a time
        _case("loop_80", grid=(80, 80, 65), theta=162.0, steps=5, loop=True),
        # the headline workload: the 150x150x107 ridge impact in float32
        _case("ridge_150", grid=(150, 150, 107), theta=162.0, steps=8),
        # odd extents, every option away from its default: tau_h != 1, tau_g != tau_l, quadratic wetting
        _case("concave_tau_121", grid=(121, 97, 85), substrate="concave", theta=100.0, steps=5, tau_h=0.57, tau_g=0.6),
        # the Cahn-Hilliard interface mode (two more passes per step) at a sweep size
        _case("cahn_hilliard_128", grid=(128, 128, 96), substrate="flat", theta=120.0, steps=5,
              interface="cahn-hilliard"),
        # float64, the mode of the verification scripts and the error runs
        _case("double_96", grid=(96, 96, 96), substrate="ridge", theta=150.0, dtype="float64", steps=5),
        # the largest grid of the serving workload, float32
        _case("convex_256", grid=(256, 256, 192), substrate="convex", theta=150.0, steps=4),
        # the precision workload: 384x384x256 in half-precision storage, the largest case
        _case("half_384", grid=(384, 384, 256), substrate="convex", theta=150.0, dtype="float16", steps=2),
        # the batched sweep: grids of uneven extents and substrates in half-precision storage
        _case("batch_sweep_8", kind="batch", dtype="float16", steps=2, count=8),
        # the 2-D path on its bench grid
        _case("ridge2d_2048", grid=(2048, 1024, 1), theta=150.0, steps=8),
        # a check point of a monitored run: a few steps, then every read-out
        _case("watch_128", kind="watch", grid=(128, 128, 96), substrate="ridge", theta=150.0, steps=3),
        # a short solve from host arrays, set-up and read-back included
        _case("solve_150", kind="solve", grid=(150, 150, 107), theta=162.0, steps=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "step", "batch", "watch", "solve"))
    dtype = rng.choice(("float32", "float32", "float32", "float16", "float64"))
    theta = round(rng.uniform(92.0, 162.0), 1)
    substrate = rng.choice(_SUBSTRATES)
    tau_h = rng.choice((1.0, 1.0, 1.0, 0.57))
    if kind == "batch":
        return _case("", kind="batch", dtype=rng.choice(("float16", "float32")), steps=rng.choice((1, 2, 3)),
                     count=rng.randint(2, 10), theta=theta)
    if kind == "step" and dtype != "float16" and rng.random() < 0.25:  # the 2-D path
        n = _log_int(rng, 4000, 2200000)
        ny = max(40, int(math.sqrt(n / rng.uniform(1.0, 3.0))))
        return _case("", grid=(max(40, n // ny), ny, 1), substrate=substrate, theta=theta, dtype=dtype,
                     steps=rng.randint(1, 8), tau_h=tau_h)
    n = _log_int(rng, 12000, {"float64": 1500000, "float16": 24000000}.get(dtype, 12000000))
    if kind != "step":
        n = min(n, 2500000)
    s = (n / 0.75) ** (1.0 / 3.0)
    nx = max(22, int(s * rng.uniform(0.85, 1.2)))
    ny = max(22, int(s * rng.uniform(0.85, 1.2)))
    nz = max(20, n // (nx * ny))
    steps = rng.randint(2, 4) if kind == "watch" else rng.randint(2, 10) if kind == "solve" else rng.randint(1, 2 if dtype == "float16" else 6)
    interface = "cahn-hilliard" if dtype != "float16" and rng.random() < 0.15 else "allen-cahn"
    return _case("", kind=kind, grid=(nx, ny, nz), substrate=substrate, theta=theta, dtype=dtype, steps=steps,
                 tau_h=tau_h, interface=interface, loop=kind == "step" and n < 400000 and rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _parts(case, seed):
    """The grids of a case: one dict of plain values per solver."""
    r = np.random.default_rng([int(seed), 77])
    parts = []
    for i in range(case["count"]):
        if case["kind"] == "batch":
            grid = _SWEEP[i % len(_SWEEP)] if i < len(_SWEEP) else _SWEEP[(3 * i + 1) % len(_SWEEP)]
            substrate, theta = _SUBSTRATES[(i + i // 4) % 4], (case["theta"] - 92.0 + 19.0 * i) % 70.0 + 92.0
        else:
            grid, substrate, theta = (case["nx"], case["ny"], case["nz"]), case["substrate"], case["theta"]
        two_d = grid[2] == 1
        span = grid[:2] if two_d else grid
        R = min(30.0 if not two_d else 150.0, 0.21 * min(span)) * r.uniform(0.94, 1.04)
        R_g = R * r.uniform(0.95, 1.05)
        h = {"flat": 1.0, "ridge": R_g, "convex": 2.0 * R_g, "concave": 0.55 * R_g}[substrate]
        c = [s / 2.0 + r.uniform(-0.8, 0.8) for s in span[:-1]]
        c.append(min(h + 1.5 + R, span[-1] - R - 2.0) + r.uniform(-0.4, 0.4))
        u = list(r.uniform(-0.012, 0.012, len(span) - 1)) + [-r.uniform(0.03, 0.06)]
        parts.append(dict(grid=grid, span=span, substrate=substrate, theta=theta, R=R, R_g=R_g, center=c, u=u))
    return parts


def _fields(p):
    """(solid, fraction, phi, u) of one grid on the device, in the types of the generators users call: bool,
    float64, float32, float32."""
    span = p["span"]
    ax = [torch.arange(s, dtype=torch.float64, device=_DEV).reshape([-1 if a == d else 1 for a in range(len(span))])
          for d, s in enumerate(span)]
    up, R_g = ax[-1], p["R_g"]
    frac = (up == 0).to(torch.float64).expand(span).contiguous()
    if p["substrate"] != "flat":
        r2 = (ax[0] - span[0] / 2.0) ** 2
        if p["substrate"] == "ridge":
            r2 = r2 + up ** 2
        else:
            r2 = r2 + (up - R_g) ** 2
            if len(span) == 3:
                r2 = r2 + (ax[1] - span[1] / 2.0) ** 2
        sd = R_g - torch.sqrt(r2)
        if p["substrate"] == "concave":
            frac = torch.where((up < R_g).expand(span), torch.maximum(frac, (0.5 - sd).clamp(0.0, 1.0)), frac)
        else:
            frac = torch.maximum(frac, (sd + 0.5).clamp(0.0, 1.0))
    r2 = sum((a - c) ** 2 for a, c in zip(ax, p["center"]))
    phi = (0.5 + 0.5 * torch.tanh(2.0 * (p["R"] - torch.sqrt(r2)) / 4.0)).clamp(0.0, 1.0).to(torch.float32)
    u = torch.stack([v * phi for v in p["u"]])
    return frac >= 0.5, frac, phi, u


def _config(case, p):
    nx, ny, nz = p["grid"]
    return FEConfig(nx=nx, ny=ny, nz=nz, rho_l=1.0, rho_g=1.0 / 828.0, sigma=0.01424, xi=4.0, tau_l=0.53,
                    tau_g=case["tau_g"], tau_h=case["tau_h"], theta_eq=p["theta"], device=_DEV)


def _solver(case, p):
    return AllenCahnSolver(_config(case, p), dtype=_DTYPES[case["dtype"]], geo_amplification=1.5,
                           geometric_wetting=True, interface_mode=case["interface"])


def prepare(case, seed):
    state = {"case": case, "parts": _parts(case, seed)}
    if case["kind"] == "solve":
        state["host"] = [x.cpu().numpy() for x in _fields(state["parts"][0])]
        return state
    solvers = []
    for p in state["parts"]:
        solid, frac, phi, u = _fields(p)
        s = _solver(case, p)
        s.set_solid(solid, frac)
        s.init_fields(phi, u)
        solvers.append(s)
    state["solvers"] = solvers
    if case["kind"] == "batch":
        state["batch"] = AllenCahnBatch(solvers)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        solid, frac, phi, u = state["host"]
        s = _solver(case, state["parts"][0])
        s.set_solid(solid, frac)
        s.init_fields(phi, u)
        s.run(case["steps"])
        m = s.measure()
        out = {"phi": s.phi.cpu().numpy(), "extent": np.array([m["Dx"], m["Dy"], m["Dz"]]), "volume": m["volume"]}
        s.close()
        return out
    if case["kind"] == "batch":
        state["batch"].run(case["steps"])
        return [dict(zip(("phi", "u"), s.fields("phi", "u"))) for s in state["solvers"]]
    s = state["solvers"][0]
    if case["loop"]:
        for _ in range(case["steps"]):
            s.step()
    else:
        s.run(case["steps"])
    if case["kind"] == "step":
        return dict(zip(("phi", "u"), s.fields("phi", "u")))
    names = ("phi", "rho", "u", "P", "p", "mu_phi")
    out = dict(zip(names, s.fields(*names)))
    out["f"], out["g"] = s.f, s.g
    m, r = s.measure(), s.reduce()
    spread = measure_spread_factor(out["phi"], s.solid)
    out["measure"] = np.array([m["volume"], m["z_com"], m["C_max"], m["Dx"], m["Dy"], m["Dz"]])
    out["momentum"] = np.array(r["momentum"])
    out["spread"] = np.array([spread["volume"], spread["Dx"], spread["Dy"], spread["Dz"]])
    return out


def work(case):
    """Bytes and operations one pass cannot do without: per time step each value of the state read once and written
    once.  The state of a node is g (one value per lattice velocity), u, phi, and f; with tau_h = 1 the
    post-collision f follows from phi, u and the vector of the interface source, so that vector counts in its place.
    A class byte is read.  Operations: about 450 (19 velocities) and 230 (9) per node and step.  The read-outs and
    set-up inputs are added once."""
    T = 8 if case["dtype"] == "float64" else 4
    S = 2 if case["dtype"] == "float16" else T
    nbytes = flops = 0.0
    for p in _parts(case, 0):
        nx, ny, nz = p["grid"]
        N, D, q = float(nx * ny * nz), (2 if nz == 1 else 3), (9 if nz == 1 else 19)
        f = 2 * D * T if case["tau_h"] == 1.0 else 2 * q * S
        nbytes += N * case["steps"] * (2 * q * S + 2 * D * T + 2 * T + f + 1)
        flops += N * case["steps"] * (230.0 if D == 2 else 450.0)
        if case["kind"] == "solve":
            nbytes += N * (1 + 8 + 4 * (1 + D)) + N * (2 * q * S + (1 + D) * T) + N * T
        elif case["kind"] == "watch":
            nbytes += N * T * 2 * (2 * q + D + 5)
        else:
            nbytes += N * T * 2 * (1 + D)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The same passes in float64, plain torch
# ---------------------------------------------------------------------------
_E3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
       (-1, -1, 0), (1, -1, 0), (1, 0, 1), (-1, 0, 1), (-1, 0, -1), (1, 0, -1), (0, 1, 1), (0, -1, 1), (0, -1, -1),
       (0, 1, -1)]
_E2 = [(0, 0), (1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]


class _Exact:
    """The solver's equations in float64: the lattice weights and the wall tables are the float32 values the method
    uses in every precision."""

    def __init__(self, case, p):
        self.case, self.cfg, self.theta = case, _config(case, p), p["theta"]
        solid, frac, phi, u = _fields(p)
        self.solid, self.D = solid, solid.dim()
        self.E = _E2 if self.D == 2 else _E3
        self.opp = [self.E.index(tuple(-x for x in e)) for e in self.E]
        w = {0: 1 / 3 if self.D == 3 else 4 / 9, 1: 1 / 18 if self.D == 3 else 1 / 9, 2: 1 / 36}
        self.w = [float(np.float32(w[sum(abs(x) for x in e)])) for e in self.E]
        self.cs2 = 1.0 / 3.0
        self._geometry(frac)
        self.phi = phi.double().clamp(0.0, 1.0)
        self.u = u.double()
        self.mass = float(self.phi.sum())
        self.f = torch.stack([self.phi * x for x in self._equilibrium(self.u, 1.0)])
        self.g = torch.stack(self._equilibrium(self.u, 0.0))
        self.phi_u = None

    def _at(self, a, e, sign=1):
        """a(x + sign e), periodic."""
        return torch.roll(a, tuple(-sign * x for x in e), tuple(range(self.D)))

    def _dot(self, e, v):
        return sum(x * v[d] for d, x in enumerate(e) if x)

    def _geometry(self, frac):
        solid, D = self.solid, self.D
        self.partial = (frac > 0.01) & (frac < 0.99) & ~solid
        self.eps = frac
        b = torch.zeros_like(solid)
        for e in self.E[1:]:
            b |= self._at(solid, e) & ~solid
        self.boundary = b
        grad = torch.gradient(frac)
        mag = torch.sqrt(sum(x * x for x in grad)).clamp_min(1e-10)
        self.normal = [((-x / mag) * b).float() for x in grad]
        dist = torch.where(b, 0.0, 100.0)
        for _ in range(11):
            near = dist
            for d in range(D):
                near = torch.minimum(near, torch.minimum(torch.roll(dist, 1, d), torch.roll(dist, -1, d)) + 1.0)
            dist = near
        weight = torch.exp((-dist / 2.5).double()).float()  # float32 argument and value
        self.weight = torch.where(solid, 0.0, weight).double()
        n = [x.double() for x in self.normal]
        size = torch.sqrt(sum(x * x for x in n)).clamp_min(1e-10)
        self.top = b & (n[-1].abs() / size > 0.5)
        self.linear = self.theta > 130.0 or self.theta < 50.0
        h = self.cfg.sigma * math.cos(math.radians(self.theta))
        scale = h / self.cfg.kappa * (3.0 if abs(self.theta - 90.0) > 60.0 else 2.0) if self.linear \
            else self.cfg.phi_c / self.cfg.kappa
        self.mu_wall = -2.0 * h
        self.ghost = []
        for e in self.E:
            nde = sum(float(x) * self.normal[d] for d, x in enumerate(e)) * float(np.float32(scale))
            self.ghost.append((self._at(solid, e) & b, nde.double()))
        c = math.cos(math.radians(self.theta))
        disc = 1.0 + 4.0 * c / 3.0
        self.target = 0.5 * (1.0 - math.sqrt(disc)) if disc >= 0 else 0.5 * (1.0 + c)

    def _neighbour(self, a, q):
        mask, nde = self.ghost[q]
        v = self._at(a, self.E[q])
        return torch.where(mask, a - nde if self.linear else a + nde * a * (1.0 - a), v)

    def _equilibrium(self, u, one):
        """w (one + e.u/cs2 + (e.u/cs2)^2/2 - u.u/(2 cs2)) for every velocity."""
        sq = sum(x * x for x in u) / (2.0 * self.cs2)
        out = []
        for q, e in enumerate(self.E):
            eu = self._dot(e, u) / self.cs2
            out.append(self.w[q] * (one + eu + 0.5 * eu * eu - sq))
        return out

    def _gradient(self, a):
        grad = [torch.zeros_like(a) for _ in range(self.D)]
        lap = torch.zeros_like(a)
        for q in range(1, len(self.E)):
            v = self._neighbour(a, q)
            for d, x in enumerate(self.E[q]):
                if x:
                    grad[d] += (self.w[q] / self.cs2 * x) * v
            lap += (2.0 * self.w[q] / self.cs2) * (v - a)
        return grad, lap

    def step(self):
        cfg, E, cs2, D, solid = self.cfg, self.E, self.cs2, self.D, self.solid
        phi = torch.where(solid, 0.0, self.f.sum(0).clamp(0.0, 1.0))
        self.rho = phi * cfg.rho_l + (1.0 - phi) * cfg.rho_g
        rho_e = self.rho.clamp_min(0.5 * cfg.rho_l)
        grad, lap = self._gradient(phi)
        mu = 4.0 * cfg.beta * phi * (phi - 1.0) * (phi - 0.5) - cfg.kappa * lap
        mu = mu + self.boundary.double() * (self.mu_wall if self.linear else cfg.phi_c * phi * (1.0 - phi))
        self.mu = mu
        # geometric contact-angle correction
        n = [x.double() for x in self.normal]
        gn = sum(a * b for a, b in zip(n, grad))
        gt = [b - gn * a for a, b in zip(n, grad)]
        size = torch.sqrt(sum(x * x for x in gt)).clamp_min(1e-10)
        want = -size * math.cos(math.radians(self.theta)) / math.sin(math.radians(self.theta))
        want = gn + (want - gn) * 1.5
        on = self.boundary & (torch.sqrt(sum(x * x for x in grad)) > 1e-6)
        grad = [torch.where(on, b + self.weight * (t + want * a - b), b) for a, b, t in zip(n, grad, gt)]
        # pressure, non-equilibrium stress, forces, velocity
        P = self.g.sum(0)
        self.P = P
        eq = self._equilibrium(self.u, 0.0)
        drho = cfg.rho_l - cfg.rho_g
        visc = (0.5 - cfg.tau_g) / cfg.tau_g
        F = [(mu - P * drho * cs2) * x for x in grad]
        for q in range(1, len(E)):
            off = (self.g[q] - eq[q] - P * self.w[q]) * self._dot(E[q], grad) * (visc * drho)
            for d, x in enumerate(E[q]):
                if x:
                    F[d] = F[d] + x * off
        u = [sum(E[q][d] * self.g[q] for q in range(len(E)) if E[q][d]) + 0.5 * F[d] / rho_e for d in range(D)]
        u = torch.stack([torch.where(solid, 0.0, x) for x in u])
        # interface source
        now = phi * u
        source = now - self.phi_u if self.phi_u is not None else torch.zeros_like(now)
        self.phi_u = now
        if self.case["interface"] == "cahn-hilliard":
            gmu, _ = self._gradient(mu)
            m = cs2 * (cfg.tau_h - 0.5) * cfg.tau_h / (cfg.tau_h - 0.5)
            source = source + torch.stack([m * (a - b) for a, b in zip(gmu, grad)])
        else:
            size = torch.sqrt(sum(x * x for x in grad)).clamp_min(1e-10)
            lam = cs2 * 4.0 * phi * (1.0 - phi) / cfg.xi * (1.0 - 0.8 * self.weight)
            source = source + torch.stack([lam * x / size for x in grad])
        # collisions
        if cfg.tau_g != cfg.tau_l:
            eta = phi * cfg.rho_l * (cfg.tau_l - 0.5) + (1.0 - phi) * cfg.rho_g * (cfg.tau_g - 0.5)
            om = 1.0 / (0.5 + eta / (phi * cfg.rho_l + (1.0 - phi) * cfg.rho_g))
        else:
            om = torch.full_like(phi, 1.0 / cfg.tau_l)
        feq, geq = self._equilibrium(u, 1.0), self._equilibrium(u, 0.0)
        f, g = torch.empty_like(self.f), torch.empty_like(self.g)
        for q, e in enumerate(E):
            f[q] = self.f[q] - (self.f[q] - phi * feq[q]) / cfg.tau_h
            g[q] = self.g[q] - om * (self.g[q] - geq[q] - P * self.w[q])
            if q:
                f[q] += (1.0 - 0.5 / cfg.tau_h) * self.w[q] / cs2 * self._dot(e, source)
                g[q] += (1.0 - 0.5 * om) * self.w[q] * self._dot(e, F) / (rho_e * cs2)
        # streaming, bounce-back, volume penalisation
        for q, e in enumerate(E):
            for old, new in ((f, self.f), (g, self.g)):
                v = self._at(old[q], e, -1)
                v = torch.where(self.partial, (1.0 - self.eps) * v + self.eps * old[self.opp[q]], v)
                new[q] = torch.where(solid, old[self.opp[q]], v)
        # mass correction, boundary-phi relaxation
        corr = self.mass / float(phi.sum())
        self.u, self.phi = u, (phi * corr).clamp(0.0, 1.0)
        self.f *= corr
        if abs(self.target - 0.5) > 0.05:
            on = self.top & (self.phi > 0.15) & (self.phi < 0.85)
            new = (self.phi + 0.3 * (self.target - self.phi)).clamp(0.0, 1.0)
            scale = (new / self.f.sum(0).clamp_min(1e-10)).clamp(0.5, 2.0)
            self.f *= torch.where(on, scale, 1.0)
            self.phi = torch.where(on, new, self.phi)


def _extents(phi, solid):
    inside = (phi > 0.5) & ~solid
    hits = []
    for d in range(phi.dim()):
        i = torch.nonzero(inside.any(dim=tuple(a for a in range(phi.dim()) if a != d))).flatten()
        hits.append(float(i[-1] - i[0] + 1) if len(i) else 0.0)
    return hits, torch.nonzero(inside)[:, -1].double().mean().item()


def exact(case, seed):
    outs = []
    for p in _parts(case, seed):
        s = _Exact(case, p)
        for _ in range(case["steps"]):
            s.step()
        phi = torch.where(s.solid, 0.0, s.phi)
        if case["kind"] == "solve":
            return {"phi": s.phi, "extent": np.array(_extents(phi, s.solid)[0]), "volume": float(phi.sum())}
        if case["kind"] == "watch":
            ext, z = _extents(phi, s.solid)
            vol = float(phi.sum())
            # the momentum's density is that of the phi that is read
            rho = s.phi * s.cfg.rho_l + (1.0 - s.phi) * s.cfg.rho_g
            return {"phi": s.phi, "rho": s.rho, "u": s.u, "P": s.P, "p": s.P * s.cs2, "mu_phi": s.mu, "f": s.f,
                    "g": s.g, "measure": np.array([vol, z, float(phi.max())] + ext),
                    "momentum": np.array([float((rho * x).sum()) for x in s.u]), "spread": np.array([vol] + ext)}
        outs.append({"phi": s.phi, "u": s.u})
    return outs if case["kind"] == "batch" else outs[0]
