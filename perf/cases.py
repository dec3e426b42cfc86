"""Performance cases of the solver: what a program that designs with it calls.

Every pass goes through ``LbmSolver``, with the design (or the populations)
handed over as host arrays and the results read back as host arrays, as the
provider, the design loop and the unsteady driver do.  A case's ``kind`` is
the call sequence of one pass:

  evaluate    set_design, forward, responses, fields    (provider evaluation)
  steady      set_design, forward, responses, gradient  (design-loop iteration)
  horizon     set_design, gradient over the trajectory  (provider sensitivities)
  stage       set_design, forward, time_average, gradient of the time average
  march       set_populations, advance, populations     (state handed over and back)
  map         set_design, design, design_vjp            (volume constraint of the loop)

The channel is the one of ``implexity_b200.workloads``: plug velocity inlet,
pressure outlet, bounce-back walls, porous design region between the ports.

The library computes in FP32 and widens what it returns to FP64; the program
keeps it as FP32, or as bfloat16 (FP32's range, which gradients need) where
the populations and their cotangents are held in 16 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from implexity_b200 import LbmSolver, workloads


# ------------------------------------------------------------------ cases
def _case(name, kind, shape, steps, **kw):
    c = {"name": name, "kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2], "steps": steps,
         "lattice": 19, "collision": "trt", "storage": "float32", "arithmetic": "float32", "design": "uniform",
         "filter": "box1", "inlet": 0.05, "obstacles": False, "adjoint_steps": 0, "checkpoint_every": 0}
    c.update(kw)
    return c


def listed():
    return [
        # a first look at a problem: the grid of the parity tests, evaluated once;
        # nothing but latency counts
        _case("evaluate_16x10x8_bgk", "evaluate", (16, 10, 8), 120, collision="bgk"),
        # design sensitivities of the small channel over its whole trajectory
        # (the default adjoint), checkpoints every ceil(sqrt(steps)) steps
        _case("horizon_48x24x24_trt", "horizon", (48, 24, 24), 800),
        # ragged grid with obstacles and 16-bit storage of state and adjoint:
        # planes and strides of no 16-byte multiple, a partial last tile
        _case("horizon_61x47x35_trt_f16", "horizon", (61, 47, 35), 300, storage="float16", obstacles=True),
        # one state handed over, marched and read back on a periodic D3Q27 box
        # with a body force and solids (no ports): a coupled solver's use
        _case("march_53x36x30_d3q27", "march", (53, 36, 30), 200, lattice=27, obstacles=True),
        # loop iteration on the grid of the accuracy comparisons: the state fits L2
        _case("steady_64_trt", "steady", (64, 64, 64), 1000, adjoint_steps=1000),
        # provider evaluation with every field read back, in the mode that meets
        # the tightest objective tolerance: FP64 collision on FP32 storage
        _case("evaluate_96x80x80_f64coll", "evaluate", (96, 80, 80), 400, arithmetic="float64"),
        # the design map and its transpose alone, conic filter of radius 2 (the
        # filter and the volume constraint of the full design loop)
        _case("map_192x96x96_conic", "map", (192, 96, 96), 1, filter="conic2"),
        # unsteady design: D3Q27, pulsatile inlet, time-averaged objective,
        # checkpointed adjoint with a stage seed in every state
        _case("stage_128x104x96_d3q27", "stage", (128, 104, 96), 120, lattice=27, inlet=0.04, checkpoint_every=20),
        # the benchmark's iteration at 128^3
        _case("steady_128_trt", "steady", (128, 128, 128), 500, adjoint_steps=800),
        # the benchmark's default iteration, FP32 and 16-bit storage
        _case("steady_256x128x128_trt", "steady", (256, 128, 128), 600, adjoint_steps=1000),
        _case("steady_256x128x128_trt_f16", "steady", (256, 128, 128), 600, adjoint_steps=1000, storage="float16"),
        # the multiple-relaxation-time sphere workload, gradient of a trajectory
        _case("horizon_256x128x128_mrt", "horizon", (256, 128, 128), 200, collision="mrt", design="spheres"),
    ]


def draw(rng):
    kind = rng.choice(["evaluate", "steady", "horizon", "stage", "march", "map"])
    most = 200_000 if kind == "march" else 1_500_000
    cells = math.exp(rng.uniform(math.log(800), math.log(most)))
    a, b = math.exp(rng.uniform(0.0, 1.0)), math.exp(rng.uniform(-0.3, 0.3))
    ny = max(6, round((cells / a) ** (1 / 3) * b))
    nz = max(6, round((cells / a) ** (1 / 3) / b))
    nx = max(8, round(cells / (ny * nz)))
    cells = nx * ny * nz
    # fewer steps on larger grids, as the pass stays near a fifth of a second at most
    steps = max(20, min(rng.randint(60, 600), int(1.2e9 / cells)))
    c = _case("", kind, (nx, ny, nz), steps, inlet=0.04,
              lattice=27 if kind == "stage" else rng.choice([19, 19, 27]),
              collision=rng.choice(["bgk", "trt", "trt", "mrt"]),
              storage=rng.choice(["float32", "float32", "float16", "bfloat16"]),
              filter=rng.choice(["box1", "conic2", "none"]),
              obstacles=rng.random() < 0.4)
    if kind == "steady":
        c["adjoint_steps"] = max(20, steps // 2)
    if kind in ("horizon", "stage"):
        c["checkpoint_every"] = rng.choice([0, max(2, steps // 7)])
    if kind == "evaluate" and c["storage"] == "float32" and rng.random() < 0.3:
        c["arithmetic"] = "float64"
    if kind in ("march", "map"):
        c["storage"] = "float32"
    if kind == "map":
        c["steps"] = 1
    if kind == "stage":
        c["collision"] = "trt"
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _shape(case):
    return (case["nx"], case["ny"], case["nz"])


def _solid(case):
    """Obstacles that touch walls and, on the periodic box, the wrapping faces."""
    nx, ny, nz = _shape(case)
    solid = np.zeros((nx, ny, nz), dtype=bool)
    if case["obstacles"]:
        solid[nx // 3 : nx // 3 + max(1, nx // 8), 0 : max(1, ny // 3), nz // 3 : nz // 3 + max(1, nz // 4)] = True
        solid[2 * nx // 3, ny // 2 :, : max(1, nz // 5)] = True
        if case["kind"] == "march":
            solid[0, ny // 2 : ny // 2 + 2, 0:2] = True
    return solid


def _problem(case):
    shape = _shape(case)
    lattice = "D3Q%d" % case["lattice"]
    tau = 1.0 if case["collision"] == "mrt" else 0.8
    box = 1 if case["filter"] == "box1" else 0
    if case["kind"] == "stage":
        p = workloads.pulsatile_problem(shape=shape, steps=case["steps"], lattice=lattice, u_mean=case["inlet"],
                                        period_steps=100, storage=case["storage"], box_half_width=box)
        solid = _solid(case)
        p["solid_mask"] = solid
        p["design_region"] &= ~solid
    else:
        p = workloads.channel_problem(shape=shape, steps=case["steps"], tau=tau, u_in=case["inlet"],
                                      collision=case["collision"], lattice=lattice, storage=case["storage"],
                                      box_half_width=box, mrt_bulk_rate=1.2 if case["collision"] == "mrt" else None,
                                      ports=case["kind"] != "march", solid=_solid(case))
    if case["filter"] == "conic2":
        p["topology_map"]["filter_radius_m"] = 2.0 * p["spacing_m"]
    if case["kind"] == "march":
        p["periodic_axes"] = [True, False, True]
        p["acceleration_m_s2"] = [2e-5, 0.0, 1e-6]
    p["solver_options"]["collision_arithmetic"] = case["arithmetic"]
    return p


def _lattice(q):
    c = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)
         if (x, y, z) != (0, 0, 0) and (q == 27 or abs(x) + abs(y) + abs(z) < 3)]
    c = np.array([(0, 0, 0)] + c)
    order = np.abs(c).sum(1)
    w = np.array([1 / 3, 1 / 18, 1 / 36] if q == 19 else [8 / 27, 2 / 27, 1 / 54, 1 / 216])[order]
    return c, w


def _design(case, seed):
    if case["design"] == "spheres":
        return workloads.sphere_design(_shape(case), seed)
    return workloads.uniform_design(_shape(case), seed)


def _weights(kind):
    if kind == "stage":  # the time-averaged viscous dissipation
        w = np.zeros(8)
        w[7] = 1.0
        return w
    return workloads.objective_weights()


def _populations(case, seed):
    """A smooth, slightly perturbed state near equilibrium, f[cells, q]."""
    q = case["lattice"]
    c, w = _lattice(q)
    rng = np.random.default_rng(seed)
    n = math.prod(_shape(case))
    rho = 1.0 + 1e-3 * rng.standard_normal((n, 1))
    cu = (0.02 * rng.standard_normal((n, 3))) @ c.T
    return rho * w * (1.0 + 3.0 * cu + 4.5 * cu * cu) * (1.0 + 1e-3 * rng.standard_normal((n, q)))


def prepare(case, seed):
    s = {"case": case, "solver": LbmSolver(_problem(case)), "weights": _weights(case["kind"]),
         "dtype": torch.float32 if case["storage"] == "float32" else torch.bfloat16,
         "design": _design(case, seed)}
    if case["kind"] == "march":
        s["populations"] = _populations(case, seed)
        s["solver"].set_design(s["design"])
    if case["kind"] == "map":
        cells = math.prod(_shape(case))
        s["phi_bar"] = np.random.default_rng(seed + 1).uniform(0.5, 1.5, _shape(case)) / (0.4 * cells)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case, solver, w = s["case"], s["solver"], s["weights"]
    kind = case["kind"]

    def keep(a):
        return torch.from_numpy(a).to(s["dtype"])

    if kind == "march":
        solver.set_populations(s["populations"])
        d = solver.advance(case["steps"])
        return {"populations": keep(solver.populations()), "mach": d.maximum_mach,
                "minimum_population": d.minimum_population}
    solver.set_design(s["design"])
    if kind == "evaluate":
        d = solver.forward()
        r, f = solver.responses(), solver.fields()
        return {"responses": keep(r), "velocity": keep(f["velocity_m_s"]), "pressure": keep(f["gauge_pressure_Pa"]),
                "density": keep(f["density_kg_m3"]), "mach": d.maximum_mach,
                "minimum_population": d.minimum_population}
    if kind == "steady":
        # an iteration of an early design: a loose tolerance, met at the first residual check
        solver.forward()
        r = solver.responses()
        g, rep = solver.gradient(w, mode="steady", tolerance=0.9, lambda_storage=case["storage"],
                                 check_every=case["adjoint_steps"])
        return {"responses": keep(r), "gradient": keep(g), "iterations": rep.iterations}
    if kind == "horizon":
        g, rep = solver.gradient(w, mode="horizon", lambda_storage=case["storage"],
                                 checkpoint_every=case["checkpoint_every"])
        return {"gradient": keep(g), "iterations": rep.iterations}
    if kind == "stage":
        solver.forward()
        r = solver.time_average()
        g, rep = solver.gradient(w, mode="horizon", lambda_storage=case["storage"], objective="time_average",
                                 checkpoint_every=case["checkpoint_every"])
        return {"responses": keep(r), "gradient": keep(g), "iterations": rep.iterations}
    phi, alpha = solver.design()
    return {"phi": keep(phi), "alpha": keep(alpha), "gradient": keep(solver.design_vjp(s["phi_bar"]))}


# ------------------------------------------------------------------ the work of one pass
def work(case):
    n, q = math.prod(_shape(case)), case["lattice"]
    sb = 4 if case["storage"] == "float32" else 2
    T = case["steps"]
    records = 40 if case["kind"] == "stage" else 16
    forward = n * (2 * q * sb + 4)                    # populations in and out, alpha
    adjoint = n * (2 * q * sb + 4 + records + 8)      # cotangents in and out, alpha, the record, alpha cotangent
    flops = n * (15 * q if case["collision"] == "bgk" else 18 * q)
    passes = {"evaluate": (T, 0), "march": (T, 0), "steady": (T, case["adjoint_steps"]),
              "horizon": (T, T), "stage": (2 * T, T), "map": (0, 0)}[case["kind"]]
    bytes_ = passes[0] * forward + passes[1] * adjoint + 16 * n
    if case["kind"] == "evaluate":
        bytes_ += 40 * n
    if case["kind"] == "march":
        bytes_ += 16 * q * n
    if case["kind"] == "map":
        bytes_ += 32 * n
        flops = 0
    return {"bytes": bytes_, "flops": (passes[0] + passes[1]) * flops + 60 * n}


# ------------------------------------------------------------------ the same in 64 bits
class _Exact:
    """The solver restated in FP64 torch: f[q, cells] streamed states; one
    interval is collide, stream (halfway bounce-back), port reconstruction."""

    def __init__(self, case, problem):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.case, self.p = case, problem
        shape = _shape(case)
        self.shape, self.n, self.q = shape, math.prod(shape), case["lattice"]
        self.c, w = _lattice(self.q)
        self.w = self._t(w)
        self.opp = [0] + [self.q - k for k in range(1, self.q)]
        p = problem
        self.dx, self.dt, self.dens = p["spacing_m"], p["step_s"], p["density_kg_m3"]
        self.vel = self.dx / self.dt
        self.tau = 0.5 + 3.0 * p["kinematic_viscosity_m2_s"] * self.dt / self.dx**2
        self.om = 1.0 / self.tau
        self.omm = self.om if case["collision"] == "bgk" else 1.0 / (0.5 + (3.0 / 16.0) / (self.tau - 0.5))
        self.bulk = 1.2 - self.om if case["collision"] == "mrt" else 0.0
        self.a = [v * self.dt**2 / self.dx for v in p["acceleration_m_s2"]]
        self.solid_np = np.asarray(p["solid_mask"])
        self.solid = torch.from_numpy(self.solid_np.reshape(-1)).to(self.dev)
        self.fluid_count = int((~self.solid_np).sum())
        self._streaming()
        self.ports = [(torch.from_numpy(np.flatnonzero(pt["mask"])).to(self.dev), pt) for pt in p["ports"]]
        self.pulsatile = any(pt.get("frequency_hz", 0.0) for pt in p["ports"])
        self._maps = {}

    def _t(self, v):
        return torch.as_tensor(np.asarray(v, dtype=np.float64), device=self.dev)

    def _streaming(self):
        nx, ny, nz = self.shape
        cells = np.arange(self.n, dtype=np.int64)
        at = np.stack(np.unravel_index(cells, self.shape))
        src = np.empty((self.q, self.n), dtype=np.int64)
        solid = self.solid_np.reshape(-1)
        for k in range(self.q):
            s = at - self.c[k][:, None]
            outside = np.zeros(self.n, dtype=bool)
            for a in range(3):
                if not self.p["periodic_axes"][a]:
                    outside |= (s[a] < 0) | (s[a] >= self.shape[a])
                s[a] %= self.shape[a]
            y = (s[0] * ny + s[1]) * nz + s[2]
            src[k] = np.where(outside | solid[y], self.opp[k] * self.n + cells, k * self.n + y)
            src[k][solid] = (k * self.n + cells)[solid]
        back = np.empty(self.q * self.n, dtype=np.int64)
        back[src.reshape(-1)] = np.arange(self.q * self.n)
        self.src = torch.from_numpy(src.reshape(-1)).to(self.dev)
        self.back = torch.from_numpy(back).to(self.dev)

    # -- design map
    def design(self, raw):
        cls = torch.from_numpy(np.asarray(self.p["design_region"], dtype=np.float64)).to(self.dev)
        x = raw
        if self.case["filter"] != "none":
            r = 1 if self.case["filter"] == "box1" else 2
            g = np.indices((2 * r + 1,) * 3) - r
            k = np.ones(g.shape[1:]) if r == 1 else np.maximum(2.0 - np.sqrt((g**2).sum(0)), 0.0)
            num, den = torch.zeros_like(x), torch.zeros_like(x)
            for i, j, l in np.argwhere(k > 0):
                v, m = self._shift(x * cls, (i - r, j - r, l - r)), self._shift(cls, (i - r, j - r, l - r))
                num, den = num + k[i, j, l] * v, den + k[i, j, l] * m
            x = num / torch.where(den > 0, den, torch.ones_like(den))
        phi = torch.where(cls > 0, x, self._t(self.p["fixed_design"]))
        phi = torch.where(self.solid.view(self.shape), torch.zeros_like(phi), phi)
        qs = self.p["drag_shape"]
        alpha = self.dt * self.p["drag_max_per_s"] * qs * (1.0 - phi) / (qs + phi)
        return phi, alpha

    def _shift(self, x, by):
        for a in range(3):
            if by[a] == 0:
                continue
            x = torch.roll(x, -int(by[a]), a)
            if not self.p["periodic_axes"][a]:
                edge = [slice(None)] * 3
                edge[a] = slice(-int(by[a]), None) if by[a] > 0 else slice(0, -int(by[a]))
                x = x.clone()
                x[tuple(edge)] = 0.0
        return x

    # -- one interval
    def moments(self, f, alpha):
        rho = f.sum(0)
        u, F = [], []
        for d in range(3):
            j = sum(float(self.c[k][d]) * f[k] for k in range(self.q) if self.c[k][d])
            u.append((j / rho + 0.5 * self.a[d]) / (1.0 + 0.5 * alpha))
        F = [rho * (self.a[d] - alpha * u[d]) for d in range(3)]
        return rho, u, F

    def collide(self, f, alpha):
        rho, u, F = self.moments(f, alpha)
        usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        uf = u[0] * F[0] + u[1] * F[1] + u[2] * F[2]
        w = [float(v) for v in self.w]
        y0 = f[0] - rho * w[0] * (1.0 - 1.5 * usq) - 1.5 * w[0] * uf
        out = [None] * self.q
        out[0] = f[0] - self.om * y0 - 3.0 * w[0] * uf
        base, E = rho * (1.0 - 1.5 * usq), -y0
        for k in range(1, self.q // 2 + 1):
            o = self.opp[k]
            cu = sum(float(self.c[k][d]) * u[d] for d in range(3) if self.c[k][d])
            cf = sum(float(self.c[k][d]) * F[d] for d in range(3) if self.c[k][d])
            even, odd = 0.5 * (f[k] + f[o]), 0.5 * (f[k] - f[o])
            se, so = w[k] * (9.0 * cu * cf - 3.0 * uf), 3.0 * w[k] * cf
            ye = even - w[k] * (base + 4.5 * rho * cu * cu) + 0.5 * se
            yo = odd - 3.0 * w[k] * rho * cu + 0.5 * so
            pe, po = even - self.om * ye + se, odd - self.omm * yo + so
            out[k], out[o] = pe + po, pe - po
            if self.bulk:
                E = E + 2.0 * (int((self.c[k] ** 2).sum()) - 1) * ye
        if self.bulk:  # bulk moment b = |c|^2 - 1, |b|^2 = 2/3
            for k in range(self.q):
                b = int((self.c[k] ** 2).sum()) - 1
                if b:
                    out[k] = out[k] - (1.5 * self.bulk * w[k] * b) * E
        return torch.stack(out)

    def port_maps(self, t):
        """Affine map f -> J f + b of every port for the state at step t."""
        t = t if self.pulsatile else 0
        if t in self._maps:
            return self._maps[t]
        maps = []
        for cells, pt in self.ports:
            axis, sign = "xyz".index(pt["face"][0]), 1 if pt["face"].endswith("min") else -1
            v = np.array(pt["velocity_m_s"], dtype=np.float64) / self.vel
            if pt.get("frequency_hz", 0.0):
                wave = math.sin(2.0 * math.pi * pt["frequency_hz"] * t * self.dt + pt.get("phase_rad", 0.0))
                v = v + np.array(pt["amplitude_m_s"]) / self.vel * wave
            rho = 1.0 + 3.0 * pt.get("gauge_pressure_Pa", 0.0) / (self.dens * self.vel**2)
            rho = rho if pt["kind"] == "pressure" else None
            f0 = self._reconstruct(np.zeros(self.q), axis, sign, v, rho)
            J = np.stack([self._reconstruct(e, axis, sign, v, rho) - f0 for e in np.eye(self.q)], 1)
            maps.append((cells, self._t(J), self._t(f0)))
        if self.pulsatile and len(self._maps) > 4:
            self._maps.clear()
        self._maps[t] = maps
        return maps

    def _reconstruct(self, f, axis, sign, v, rho):
        c, w = self.c, self.w.cpu().numpy()
        v = v - 0.5 * np.array(self.a)
        into, out = c[:, axis] == sign, c[:, axis] == -sign
        compat = f[~into & ~out].sum() + 2.0 * f[out].sum()
        if rho is None:
            rho = compat / (1.0 - sign * v[axis])
        else:
            v = v.copy()
            v[axis] = (1.0 - compat / rho) * sign
        unknown = np.flatnonzero(into)
        prop = np.array([f[self.opp[k]] + 6.0 * w[k] * rho * (c[k] @ v) for k in unknown])
        t = [d for d in range(3) if d != axis]
        R = np.stack([np.ones(len(unknown)), c[unknown][:, t[0]], c[unknown][:, t[1]]])
        known = ~into
        target = np.array([rho - f[known].sum()] + [rho * v[d] - (f[known] * c[known][:, d]).sum() for d in t])
        g = f.copy()
        g[unknown] = prop + R.T @ np.linalg.solve(R @ R.T, target - R @ prop)
        return g

    def interval(self, f, alpha, t):
        g = self.collide(f, alpha).reshape(-1)[self.src].view(self.q, self.n)
        g[:, self.solid] = f[:, self.solid]
        for cells, J, b in self.port_maps(t + 1):
            g[:, cells] = J @ g[:, cells] + b[:, None]
        return g

    def initial(self):
        ca = self._t(self.c @ np.array(self.a))
        f = (self.w * (1.0 - 1.5 * ca))[:, None].repeat(1, self.n)
        f[:, self.solid] = self.w[:, None]
        return f

    def ports_back(self, lam, t):
        for cells, J, _ in self.port_maps(t):
            lam[:, cells] = J.T @ lam[:, cells]
        lam[:, self.solid] = 0.0
        return lam

    def pull_back(self, lam):
        return lam.reshape(-1)[self.back].view(self.q, self.n)

    # -- responses of one state
    def responses(self, f, alpha, phi):
        rho, u, F = self.moments(f, alpha)
        live = (~self.solid).to(torch.float64)
        U = [v * self.vel for v in u]
        usq = U[0] ** 2 + U[1] ** 2 + U[2] ** 2
        R, dv = rho * self.dens, self.dx**3
        r = [(v * live).sum() / self.fluid_count for v in U]
        r += [0.5 * (R * usq * live).sum() * dv, (R * alpha / self.dt * usq * live).sum() * dv, phi.sum() * dv]
        rp, drop = rho - 1.0, rho.new_zeros(())
        for cells, pt in self.ports:
            drop = drop + (1.0 if pt["kind"] == "velocity" else -1.0) * rp[cells].mean()
        r.append(drop * self.dens * self.vel**2 / 3.0)
        g, ss = f - self.w[:, None], 0.0
        for i in range(3):
            for j in range(i, 3):
                S = sum(float(self.c[k][i] * self.c[k][j]) * g[k] for k in range(self.q) if self.c[k][i] * self.c[k][j])
                sig = S - (rp / 3.0 if i == j else 0.0) - rho * u[i] * u[j] + 0.5 * (u[i] * F[j] + u[j] * F[i])
                ss = ss + (1.0 if i == j else 2.0) * ((1.0 - 0.5 * self.om) * sig) ** 2
        nu = (self.tau - 0.5) / 3.0
        r.append((ss / (2.0 * rho * nu) * live).sum() * self.dens * self.dx**5 / self.dt**3)
        return torch.stack(r)

    def seed(self, f, alpha, phi, w, scale=1.0):
        """Cotangents of f, alpha and phi of scale * w . responses."""
        f, a, p = f.detach().requires_grad_(True), alpha.detach().requires_grad_(True), phi.detach().requires_grad_(True)
        with torch.enable_grad():
            J = scale * (self.responses(f, a, p) * w).sum()
        fb, ab, pb = torch.autograd.grad(J, (f, a, p), allow_unused=True)
        return fb, ab, pb if pb is not None else torch.zeros_like(phi)


def _exact_cost(case):
    """Seconds of the restatement, roughly (2 ns per cell and forward step on a
    GPU, three times that per transposed step, and its launches)."""
    n = math.prod(_shape(case)) * case["lattice"] / 19
    T = case["steps"]
    fwd = {"map": 0, "horizon": 2 * T, "stage": 2 * T}.get(case["kind"], T)
    adj = {"steady": case["adjoint_steps"], "horizon": T, "stage": 2 * T}.get(case["kind"], 0)
    return fwd * (2e-9 * n + 1.5e-3) + adj * (6e-9 * n + 4e-3)


@torch.no_grad()
def exact(case, seed):
    if _exact_cost(case) > 17.0:
        return None
    p = _problem(case)
    E = _Exact(case, p)
    kind, T = case["kind"], case["steps"]
    raw = torch.from_numpy(_design(case, seed)).to(E.dev).requires_grad_(True)
    with torch.enable_grad():
        phi_g, alpha_g = E.design(raw)
    phi, alpha = phi_g.detach().reshape(-1), alpha_g.detach().reshape(-1)
    if kind == "map":
        n = math.prod(_shape(case))
        pb = np.random.default_rng(seed + 1).uniform(0.5, 1.5, _shape(case)) / (0.4 * n)
        g, = torch.autograd.grad(phi_g, raw, E._t(pb))
        return {"phi": phi_g.detach(), "alpha": alpha_g.detach(), "gradient": g}
    w = E._t(_weights(kind))
    live = ~E.solid
    top, low = 0.0, math.inf

    def watch(f):
        nonlocal top, low
        _, u, _ = E.moments(f, alpha)
        top = torch.clamp((u[0] ** 2 + u[1] ** 2 + u[2] ** 2)[live].max(), min=top)
        low = torch.clamp(f[:, live].min(), max=low)

    f = torch.from_numpy(_populations(case, seed).T.copy()).to(E.dev) if kind == "march" else E.initial()
    every = max(1, math.isqrt(T)) if kind in ("horizon", "stage") else 0
    kept, mean = [], 0.0
    for t in range(T):
        if every and t % every == 0:
            kept.append(f.clone())
        if kind in ("evaluate", "march"):
            watch(f)
        f = E.interval(f, alpha, t)
        if kind == "stage":
            mean = mean + E.responses(f, alpha, phi) / T
    if kind in ("evaluate", "march"):
        watch(f)
        mach, low = float(top.sqrt() * math.sqrt(3.0)), float(low)
        if kind == "march":
            return {"populations": f.T.contiguous(), "mach": mach, "minimum_population": low}
        rho, u, _ = E.moments(f, alpha)
        rho = torch.where(live, rho, torch.ones_like(rho))
        U = torch.stack([torch.where(live, v, torch.zeros_like(v)) * E.vel for v in u], 1)
        return {"responses": E.responses(f, alpha, phi), "velocity": U.view(*E.shape, 3),
                "pressure": ((rho - 1.0) * E.dens * E.vel**2 / 3.0).view(E.shape),
                "density": (rho * E.dens).view(E.shape), "mach": mach, "minimum_population": low}
    scale = 1.0 / T if kind == "stage" else 1.0
    lam, abar, pbar = E.seed(f, alpha, phi, w, scale)
    lam = E.ports_back(lam, T)

    def transposed(state, lam, retained=None):
        if retained is None:
            x, a = state.detach().requires_grad_(True), alpha.detach().requires_grad_(True)
            with torch.enable_grad():
                retained = (E.collide(x, a), x, a)
        back = torch.where(E.solid, torch.zeros_like(alpha), E.pull_back(lam))
        return torch.autograd.grad(retained[0], retained[1:], back, retain_graph=True), retained

    if kind == "steady":
        retained = None
        for _ in range(case["adjoint_steps"]):
            (lam, ab), retained = transposed(f, lam, retained)
            abar = abar + ab
            lam = E.ports_back(lam, T)
    else:
        for k in range(len(kept) - 1, -1, -1):
            states = [kept.pop()]
            for t in range(k * every, min((k + 1) * every, T) - 1):
                states.append(E.interval(states[-1], alpha, t))
            for t in range(k * every + len(states) - 1, k * every - 1, -1):
                state = states.pop()
                (lam, ab), _ = transposed(state, lam)
                abar = abar + ab
                if kind == "stage" and t >= 1:
                    fb, sb, _ = E.seed(state, alpha, phi, w, scale)
                    lam, abar = lam + fb, abar + sb
                lam = E.ports_back(lam, t)
    abar[E.solid] = 0.0
    g, = torch.autograd.grad([phi_g, alpha_g], raw, [pbar.view(E.shape), abar.view(E.shape)])
    if kind == "steady":
        return {"responses": E.responses(f, alpha, phi), "gradient": g, "iterations": None}
    if kind == "horizon":
        return {"gradient": g, "iterations": None}
    return {"responses": mean, "gradient": g, "iterations": None}
