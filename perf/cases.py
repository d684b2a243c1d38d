"""Performance cases of the framework: what its users run, through its public entry points.

Each case is a dict of plain values; `prepare` builds what a program has in
hand before the call (the operator, its vectors with the projected initial
data, a seeded phase or blob centre), `run` makes one pass, `exact` gives the
same outputs in plain float64 torch without the package, `work` the bytes and
operations of a pass.

Kinds
-----
steps        `lsrk_steps`: n LSRK steps on the device (the time loop between two outputs)
integrator   `LowStorageRungeKuttaIntegrator.perform_time_step`, one step per call
host_steps   `lsrk_steps_host`: the same loop with the solution in pinned host memory
stages       a caller's own LSRK loop over `perform_stage`, with the reference's aliasing
apply        one operator application `apply` (a caller's own integrator)
bdf2         two implicit steps (implicit Euler, then BDF2) with FGMRES and the FDM preconditioner
output       the diagnostics of an output time: projection, L2 error, mass and energy
serving      a burst of requests of the serving mix through `Server`, drained
"""
import math

import numpy as np
import torch

import advection_miniapp_gb300 as adv
from advection_miniapp_gb300 import serving

SCHEMES = {"3_3": adv.LSRK_3_3, "5_4": adv.LSRK_5_4, "7_4": adv.LSRK_7_4, "9_5": adv.LSRK_9_5}
PRECISIONS = {"fp64": adv.PRECISION_FP64, "fp32_operator": adv.PRECISION_FP32_OPERATOR,
              "fp32_increment": adv.PRECISION_FP32_INCREMENT}


def _case(name, kind, degree, nx, ny, nz, **kw):
    base = dict(name=name, kind=kind, degree=degree, nx=nx, ny=ny, nz=nz, curved=False, physics="advection",
                precision="fp64", scheme="5_4", steps=1, courant=0.5)
    base.update(kw)
    return base


def listed():
    return [
        # the configuration a CPU can run, stepped by the integrator class one
        # step per call: the smallest calls, latency and launches
        _case("integrator-affine-k3-8", "integrator", 3, 8, 8, 8),
        # the plain method at GPU scale, between two outputs of its time loop
        _case("steps-curved-k4-64", "steps", 4, 64, 64, 64, curved=True, steps=4),
        # the same problem class with the binary32 operator
        _case("steps-curved-k4-48-fp32op", "steps", 4, 48, 48, 48, curved=True, steps=4,
              precision="fp32_operator"),
        # and with binary32 increments: one anchor block of four steps
        _case("steps-curved-k4-48-fp32inc", "steps", 4, 48, 48, 48, curved=True, steps=4,
              precision="fp32_increment"),
        # variable-coefficient advection-diffusion with Dirichlet data (explicit SIPG)
        _case("steps-sipg-k5-32", "steps", 5, 32, 32, 32, physics="rotating_diffusion"),
        # affine box of odd extents at low order, a seven-stage scheme
        _case("steps-affine-k2-odd", "steps", 2, 37, 23, 29, scheme="7_4", steps=4),
        # the solution lives in the caller's host memory: copy in, step, copy out
        _case("host-curved-k4-48", "host_steps", 4, 48, 48, 48, curved=True, steps=1),
        # a caller's own Runge-Kutta loop over perform_stage
        _case("stages-curved-k4-32", "stages", 4, 32, 32, 32, curved=True),
        # a caller's own integrator at the highest degree, ragged mesh, inflow data
        _case("apply-dirichlet-k6-ragged", "apply", 6, 17, 13, 11, curved=True, physics="dirichlet"),
        # implicit steps at a Courant number of 8
        _case("bdf2-curved-k4-32", "bdf2", 4, 32, 32, 32, curved=True, courant=8.0),
        # an output time: project the exact solution, L2 error, mass and energy
        _case("output-curved-k4-32", "output", 4, 32, 32, 32, curved=True),
        # a burst of small and middle solves of mixed degree and precision
        _case("serving-burst-16", "serving", 4, 16, 16, 16, requests=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "integrator", "host_steps", "stages", "apply", "bdf2", "output",
                       "serving"])
    degree = rng.randint(1, 6)
    # degrees of freedom over the range of the listed cases, at most the largest's
    top = 4e6 if kind in ("bdf2", "output") else 3.2e5 if kind == "serving" else 1.6e7
    dofs = math.exp(rng.uniform(math.log(8e3), math.log(top)))
    edge = (dofs / (degree + 1) ** 3) ** (1.0 / 3.0)
    # unequal, often odd extents around the cubic mesh of that size
    nx, ny = (max(2, int(round(edge * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(2))
    nz = max(2, int(dofs / (degree + 1) ** 3 / (nx * ny)))
    curved = rng.random() < 0.6
    physics = "advection"
    if kind in ("steps", "integrator", "host_steps", "stages", "apply"):
        physics = rng.choice(["advection", "advection", "rotating", "rotating_diffusion", "dirichlet"])
    if physics == "rotating_diffusion":
        curved = False
    precision = "fp64"
    if kind in ("steps", "host_steps"):
        precision = rng.choice(["fp64", "fp64", "fp32_operator", "fp32_increment"])
    elif kind in ("integrator", "stages", "apply"):
        precision = rng.choice(["fp64", "fp64", "fp32_operator"])
    c = _case("", kind, degree, nx, ny, nz, curved=curved, physics=physics, precision=precision)
    del c["name"]
    if kind in ("steps", "host_steps", "integrator", "stages"):
        c["scheme"] = rng.choice(list(SCHEMES))
    if kind in ("steps", "host_steps"):
        c["steps"] = rng.randint(1, 4)
    if kind == "bdf2":
        c["courant"] = rng.choice([2.0, 4.0, 8.0])
    if kind == "serving":
        c["requests"] = rng.randint(2, 16)
    return c


# ------------------------------------------------------------ configurations


def _config(case, seed):
    """adv_config fields of a case; the seed places the initial data."""
    g = np.random.default_rng([seed, 17])
    c = dict(degree=case["degree"], n_cells=(case["nx"], case["ny"], case["nz"]),
             mesh_type=adv.MESH_DEFORMED if case["curved"] else adv.MESH_CARTESIAN,
             deformation=0.08 if case["curved"] else 0.0, velocity=(1.0, 0.15, -0.05), flux_alpha=1.0, periodic=1,
             precision=PRECISIONS[case["precision"]], initial_condition=adv.IC_SINE_GAUSS,
             ic_params=tuple(float(x) for x in g.uniform(0.0, 1.0, 3)) + (0.0,) * 5)
    if case["physics"] in ("rotating", "rotating_diffusion"):
        centre = np.array([0.3, 0.5, 0.5]) + g.uniform(-0.05, 0.05, 3)
        c.update(periodic=0, velocity_type=adv.VELOCITY_ROTATING, velocity=(1.0, 1.0, 0.3), velocity_period=0.5,
                 initial_condition=adv.IC_BLOB, ic_params=tuple(float(x) for x in centre) + (0.1,) + (0.0,) * 4,
                 boundary_value=adv.BOUNDARY_ZERO)
        if case["physics"] == "rotating_diffusion":
            c.update(diffusion=1e-3, penalty_factor=1.0)
    elif case["physics"] == "dirichlet":
        c.update(periodic=0, boundary_value=adv.BOUNDARY_EXACT)
    return c


def _time_step(case, cfg):
    """Courant times the smallest cell width over |velocity| and k^1.5, with an
    explicit diffusion's limit; the deformation shortens edges to about 0.6."""
    h = min(1.0 / c for c in cfg["n_cells"]) * (0.6 if case["curved"] else 1.0)
    dt = case["courant"] * h / math.sqrt(sum(x * x for x in cfg["velocity"])) / case["degree"] ** 1.5
    nu = cfg.get("diffusion", 0.0)
    if nu:
        dt = 1.0 / (1.0 / dt + nu * (case["degree"] + 1) ** 4 / (0.3 * h * h))
    return dt


def _requests(case, seed):
    """Short solves of the serving mix with at most the case's edge: meshes,
    degrees, precisions and end times belong to the case, velocity directions
    and phases to the seed."""
    sizes = tuple(n for n in serving.SIZES if n <= max(4, case["nx"]))
    requests = serving.request_mix(case["requests"], seed=case["degree"], sizes=sizes, t_range=(0.1, 0.3))
    for r in requests:
        g = np.random.default_rng([seed, r.index])
        v = g.uniform(0.1, 1.0, 3) * g.choice([-1.0, 1.0], 3)
        r.velocity = tuple(float(x) for x in v / np.linalg.norm(v))
        r.phase = tuple(float(x) for x in g.uniform(0.0, 1.0, 3))
    return requests


def prepare(case, seed):
    if case["kind"] == "serving":
        return dict(kind="serving", requests=_requests(case, seed))
    cfg = _config(case, seed)
    op = adv.AdvectionOperation(**cfg)
    s = dict(kind=case["kind"], op=op, scheme=SCHEMES[case["scheme"]], steps=case["steps"], t=0.0,
             dt=_time_step(case, cfg))
    s["u"] = op.initialize_dof_vector()
    op.project_initial(s["u"])
    if case["kind"] == "bdf2":
        s["solver"] = adv.ImplicitSolver(op)
        s["u1"], s["u2"] = op.initialize_dof_vector(), op.initialize_dof_vector()
        return s
    if case["kind"] == "apply":
        s["dst"] = op.initialize_dof_vector()
        return s
    if case["kind"] == "output":
        s["projected"] = op.initialize_dof_vector()
        return s
    s["r"], s["k"] = op.initialize_dof_vector(), op.initialize_dof_vector()
    s["rk"] = adv.LowStorageRungeKuttaIntegrator(s["scheme"])
    if case["kind"] == "host_steps":
        s["host"] = s["u"].cpu().pin_memory()
    return s


def run(s):
    kind = s["kind"]
    if kind == "serving":
        results, _, solutions = serving.run_mix(s["requests"], rate_clock=False, keep_solutions=True)
        order = [r.index for r in s["requests"]]
        return {"solutions": [solutions[i] for i in order], "steps": [results[i]["steps"] for i in order],
                "errors": np.array([results[i]["rel_l2_error"] for i in order])}
    op, u = s["op"], s["u"]
    if kind == "steps":
        op.lsrk_steps(s["scheme"], s["t"], s["dt"], s["steps"], u, s["r"], s["k"])
        s["t"] += s["steps"] * s["dt"]
        return u
    if kind == "integrator":
        s["rk"].perform_time_step(op, s["t"], s["dt"], u, s["r"], s["k"])
        s["t"] += s["dt"]
        return u
    if kind == "host_steps":
        op.lsrk_steps_host(s["scheme"], s["t"], s["dt"], s["steps"], s["host"], u, s["r"], s["k"])
        s["t"] += s["steps"] * s["dt"]
        return s["host"]
    if kind == "stages":
        a, b, dt, r, k, t = s["rk"].ai, s["rk"].bi, s["dt"], s["r"], s["k"], s["t"]
        op.perform_stage(t, b[0] * dt, a[0] * dt, u, r, u, r)
        done = 0.0
        for i in range(1, len(b)):
            op.perform_stage(t + (done + a[i - 1]) * dt, b[i] * dt, 0.0 if i == len(b) - 1 else a[i] * dt, r, k, u, r)
            done += b[i - 1]
        s["t"] += dt
        return u
    if kind == "apply":
        op.apply(u, s["dst"], s["t"])
        return s["dst"]
    if kind == "bdf2":
        s["solver"].bdf2_step(s["dt"], s["dt"], True, u, None, s["u1"])
        s["solver"].bdf2_step(2.0 * s["dt"], s["dt"], False, s["u1"], u, s["u2"])
        return {"first": s["u1"], "second": s["u2"]}
    op.project_initial(s["projected"], 0.05)
    error, norm = op.l2_error(u, 0.05)
    return {"projected": s["projected"], "l2": np.array([error, norm]), "mass_energy": op.compute_mass_and_energy(u)}


# --------------------------------------------------------------------- work


def work(case):
    """Bytes: per stage every vector the scheme reads and writes (input
    register, solution in and out, next register) and the geometry of curved
    or variable cells (four values per point and 1.2 n per face point) once.
    Operations: per point and stage three n-point derivative contractions,
    three products with the metric, the face traces and lifts of three
    directions and the update; with diffusion a second set of contractions."""
    if case["kind"] == "serving":
        total = 0.0
        for r in _requests(case, 0):
            total += 5.0 * r.steps() * r.n_dofs
        return {"bytes": 28.8 * total, "flops": 2.0 * 30.0 * total}
    n = case["degree"] + 1
    dofs = case["nx"] * case["ny"] * case["nz"] * n ** 3
    field = case["curved"] or case["physics"] != "advection" and case["physics"] != "dirichlet"
    size = 8.0 if case["precision"] == "fp64" else 4.0
    geometry = (4.0 + 6.0 / n) * size if field else 0.0
    flops = 2.0 * (3.0 * n + 3.0 + 12.0 + 3.0)
    if case["physics"] == "rotating_diffusion":
        flops *= 2.0
    if case["kind"] == "apply":
        return {"bytes": dofs * (16.0 + geometry), "flops": dofs * flops}
    if case["kind"] == "bdf2":
        # two solves: right-hand side, solution, and per iteration one operator
        # with its geometry and one preconditioner application; the iterations
        # (about 21) grow with the Courant number
        its = 2.0 * 2.6 * case["courant"]
        return {"bytes": dofs * (48.0 + its * (32.0 + geometry)), "flops": dofs * its * (flops + 2.0 * 14.0 * n)}
    if case["kind"] == "output":
        # solution in, projection out; the exact solution at n^3 + (n+1)^3
        # points per cell, the interpolations to both rules and the gradient
        return {"bytes": dofs * 24.0, "flops": dofs * (2.0 * 9.0 * n + 2.0 * (1.0 + (1.0 + 1.0 / n) ** 3) * 40.0)}
    stages = {"3_3": 3, "5_4": 5, "7_4": 7, "9_5": 9}[case["scheme"]] * case["steps"]
    copies = 0.0
    if case["kind"] == "host_steps":
        copies = 16.0  # the solution in and out of host memory
    per_stage = (24.0 + 32.0 * (stages / case["steps"] - 2.0) + 24.0) / (stages / case["steps"])
    return {"bytes": dofs * (copies + stages * (per_stage + geometry)), "flops": dofs * stages * flops}


# -------------------------------------------------------------------- exact
#
# The same method written as whole-mesh float64 tensor contractions: vectors
# as [z cells, y cells, x cells, z node, y node, x node].


def _lagrange(nodes, x):
    """Values and derivatives of the Lagrange basis: [len(x), len(nodes)] each."""
    n = len(nodes)
    v, d = np.ones((len(x), n)), np.zeros((len(x), n))
    for i in range(n):
        for j in range(n):
            if j != i:
                v[:, i] *= (x - nodes[j]) / (nodes[i] - nodes[j])
        for m in range(n):
            if m == i:
                continue
            p = np.full(len(x), 1.0 / (nodes[i] - nodes[m]))
            for j in range(n):
                if j not in (i, m):
                    p *= (x - nodes[j]) / (nodes[i] - nodes[j])
            d[:, i] += p
    return v, d


def _gauss_lobatto(n):
    if n == 2:
        return np.array([0.0, 1.0])
    p = np.polynomial.legendre.Legendre.basis(n - 1).deriv()
    x = np.sort(p.roots().real)
    for _ in range(3):
        x = x - p(x) / p.deriv()(x)
    return 0.5 + 0.5 * np.concatenate([[-1.0], x, [1.0]])


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 + 0.5 * x, 0.5 * w


class _Reference:
    """Operator, integrator and diagnostics of one configuration."""

    AXIS = (5, 4, 3)  # tensor axis of the points along x, y, z

    def __init__(self, cfg):
        self.cfg = cfg
        self.n = n = cfg["degree"] + 1
        self.nc = cfg["n_cells"]
        self.h = [1.0 / c for c in self.nc]
        self.gl, (self.gp, self.gw) = _gauss_lobatto(n), _gauss(n)
        T = self.tensor
        self.S = T(_lagrange(self.gl, self.gp)[0])
        self.Si = T(np.linalg.inv(_lagrange(self.gl, self.gp)[0]))
        D = _lagrange(self.gp, self.gp)[1]
        self.D = T(D)
        self.Dw = T(D.T * self.gw[None, :] / self.gw[:, None])
        ends, dends = _lagrange(self.gp, np.array([0.0, 1.0]))
        self.l, self.dl = T(ends), T(dends)
        self.lw, self.dlw = T(ends / self.gw), T(dends / self.gw)
        self.w3 = T(self.gw)[:, None, None] * T(self.gw)[:, None] * T(self.gw)
        self.diffusion = cfg.get("diffusion", 0.0)
        self.rotating = cfg.get("velocity_type", adv.VELOCITY_CONSTANT) == adv.VELOCITY_ROTATING
        gp = self.gp
        cof, self.det, _ = self.metric(gp, gp, gp)
        a = self.speed(self.positions(gp, gp, gp))
        self.vt = [sum(cof[d][i] * a[i] for i in range(3)) for d in range(3)]
        del cof
        # normal velocity c and position at the low and high faces of every cell
        self.c, self.fx = [], []
        for d in range(3):
            for end in (0.0, 1.0):
                pts = [gp, gp, gp]
                pts[d] = np.array([end])
                fc, _, _ = self.metric(*pts)
                x = self.positions(*pts)
                v = self.speed(x)
                self.c.append(sum(fc[d][i] * v[i] for i in range(3)))
                self.fx.append(x)

    @staticmethod
    def tensor(a):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")

    def along(self, M, u, d):
        """M applied along direction d of the points."""
        ax = self.AXIS[d]
        return torch.movedim(torch.tensordot(u, M, dims=([ax], [1])), -1, ax)

    def every(self, M, u):
        for d in range(3):
            u = self.along(M, u, d)
        return u

    def support(self):
        """Support points of the degree-k mapping relative to each cell's corner,
        and the corners."""
        s = []
        for d in range(3):
            shape, cells = [1] * 6, [1] * 6
            shape[self.AXIS[d]], cells[2 - d] = self.n, self.nc[d]
            corner = self.tensor(np.arange(self.nc[d]) * self.h[d]).reshape(cells)
            s.append((corner, self.tensor(self.gl * self.h[d]).reshape(shape)))
        if self.cfg["mesh_type"] != adv.MESH_DEFORMED:
            return None, s
        A, full = self.cfg["deformation"], []
        sn = [torch.sin(2.0 * math.pi * (c + r)) for c, r in s]
        sn0 = [torch.sin(2.0 * math.pi * c) for c, _ in s]
        for d in range(3):
            p, q = (d + 1) % 3, (d + 2) % 3
            full.append(s[d][1] + A * (sn[p] * sn[q] - sn0[p] * sn0[q]))
        base = [s[d][0] + A * sn0[(d + 1) % 3] * sn0[(d + 2) % 3] for d in range(3)]
        return (full, base), s

    def positions(self, px, py, pz):
        pts, (curved, s) = (px, py, pz), self.support()
        if curved is None:
            out = []
            for d in range(3):
                shape = [1] * 6
                shape[self.AXIS[d]] = len(pts[d])
                out.append(s[d][0] + self.h[d] * self.tensor(pts[d]).reshape(shape))
            return out
        full, base = curved
        M = [self.tensor(_lagrange(self.gl, p)[0]) for p in pts]
        out = []
        for d in range(3):
            x = full[d].expand(*self.nc[::-1], self.n, self.n, self.n)
            for e in range(3):
                x = self.along(M[e], x, e)
            out.append(x + base[d])
        return out

    def metric(self, px, py, pz):
        """Cofactors det J J^{-1} as [d][i], det J at the tensor points."""
        pts, (curved, _) = (px, py, pz), self.support()
        if curved is None:
            h = self.h
            one = torch.ones((1,) * 6, dtype=torch.float64, device="cuda")
            cof = [[one * (h[0] * h[1] * h[2] / h[d] if d == i else 0.0) for i in range(3)] for d in range(3)]
            return cof, one * (h[0] * h[1] * h[2]), None
        full, _ = curved
        V = [_lagrange(self.gl, p) for p in pts]
        J = [[None] * 3 for _ in range(3)]
        for i in range(3):
            x0 = full[i].expand(*self.nc[::-1], self.n, self.n, self.n)
            for d in range(3):
                x = x0
                for e in range(3):
                    x = self.along(self.tensor(V[e][1 if e == d else 0]), x, e)
                J[i][d] = x
        cof = [[None] * 3 for _ in range(3)]
        for d in range(3):
            for i in range(3):
                i1, i2, d1, d2 = (i + 1) % 3, (i + 2) % 3, (d + 1) % 3, (d + 2) % 3
                cof[d][i] = J[i1][d1] * J[i2][d2] - J[i1][d2] * J[i2][d1]
        det = sum(J[0][d] * cof[d][0] for d in range(3))
        return cof, det, J

    def speed(self, x):
        v = self.cfg["velocity"]
        if not self.rotating:
            return v
        sx, sy = torch.sin(math.pi * x[0]), torch.sin(math.pi * x[1])
        return [v[0] * sx * sx * torch.sin(2.0 * math.pi * x[1]),
                -v[1] * sy * sy * torch.sin(2.0 * math.pi * x[0]), v[2]]

    def factor(self, t):
        return math.cos(math.pi * t / self.cfg["velocity_period"]) if self.rotating else 1.0

    def solution(self, x, t):
        p, v = self.cfg["ic_params"], self.cfg["velocity"]
        if self.cfg["initial_condition"] == adv.IC_BLOB:
            return torch.exp(-sum((x[d] - p[d]) ** 2 for d in range(3)) / p[3] ** 2)
        y = [x[d] - v[d] * t - p[d] for d in range(3)]
        y = [q - torch.floor(q) for q in y]
        return (torch.sin(2.0 * math.pi * y[0]) * torch.sin(2.0 * math.pi * y[1]) * torch.sin(2.0 * math.pi * y[2])
                + torch.exp(-50.0 * sum((q - 0.5) ** 2 for q in y)))

    def operator(self, U, t):
        """M^{-1} L(t) on Gauss-point values."""
        f, nu = self.factor(t), self.diffusion
        exact_data = self.cfg.get("boundary_value") == adv.BOUNDARY_EXACT
        Z = torch.zeros_like(U)
        V = self.h[0] * self.h[1] * self.h[2]
        for d in range(3):
            ax, cax = self.AXIS[d], 2 - d
            flux = f * self.vt[d] * U
            if nu:
                flux = flux - nu * V / self.h[d] ** 2 * self.along(self.D, U, d)
            Z += self.along(self.Dw, flux, d)
            own = [self.along(self.l[e:e + 1], U, d) for e in (0, 1)]
            der = [self.along(self.dl[e:e + 1], U, d) for e in (0, 1)] if nu else None
            for e in (0, 1):
                shift, sign = (1, 1.0) if e == 0 else (-1, -1.0)
                other = torch.roll(own[1 - e], shift, cax)
                dother = torch.roll(der[1 - e], shift, cax) if nu else None
                if not self.cfg["periodic"]:
                    at = [slice(None)] * 6
                    at[cax] = slice(0, 1) if e == 0 else slice(-1, None)
                    at = tuple(at)
                    g = torch.zeros_like(own[e])
                    if exact_data:
                        g = self.solution(self.fx[2 * d + e], t).expand_as(own[e])
                    vis = other.clone()
                    vis[at] = 2.0 * g[at] - own[e][at]
                    other = other.clone()
                    other[at] = g[at]
                    if nu:
                        dother = dother.clone()
                        dother[at] = der[e][at]
                else:
                    vis = other
                c = f * self.c[2 * d + e]
                a = self.cfg["flux_alpha"]
                P, M = 0.5 * (c + a * c.abs()), 0.5 * (c - a * c.abs())
                phi = M * own[0] + P * other if e == 0 else -(P * own[1] + M * other)
                if nu:
                    n = self.n
                    K1 = nu * (self.cfg["penalty_factor"] * n * n / self.h[d]) * V / self.h[d]
                    K2 = nu * V / (2.0 * self.h[d] ** 2)
                    jump = (vis - own[0]) if e == 0 else (own[1] - vis)
                    phi = phi + sign * (K1 * jump - K2 * (dother + der[e]))
                    Z += self.along(self.dlw[e][:, None], K2 * jump, d)
                Z += self.along(self.lw[e][:, None], phi, d)
        return Z / self.det

    def shape(self):
        return (*self.nc[::-1], self.n, self.n, self.n)

    def project(self, t):
        gp = self.gp
        x = self.solution(self.positions(gp, gp, gp), t)
        return x.expand(self.shape()).contiguous()

    def steps(self, U, scheme, t, dt, count):
        a, b = _coefficients(scheme)
        for _ in range(count):
            r, done = U, 0.0
            for i in range(len(b)):
                ti = t if i == 0 else t + (done + a[i - 1]) * dt
                k = self.operator(r, ti)
                if i < len(b) - 1:
                    r = U + a[i] * dt * k
                U = U + b[i] * dt * k
                if i > 0:
                    done += b[i - 1]
            t += dt
        return U

    def nodal(self, U):
        return self.every(self.Si, U).reshape(-1)

    def solve(self, rhs, mass, t, x, tol=1e-13, most=220):
        """(mass - M^{-1}L) x = rhs by full GMRES on Gauss-point values."""
        r = rhs - (mass * x - self.operator(x, t))
        size = float(torch.linalg.vector_norm(rhs))
        beta = torch.linalg.vector_norm(r)
        Q, H = [r / beta], np.zeros((most + 1, most))
        for j in range(most):
            w = mass * Q[j] - self.operator(Q[j], t)
            for _ in range(2):
                for i in range(j + 1):
                    hij = torch.dot(Q[i].reshape(-1), w.reshape(-1))
                    w = w - hij * Q[i]
                    H[i, j] += float(hij)
            H[j + 1, j] = float(torch.linalg.vector_norm(w))
            Q.append(w / H[j + 1, j])
            e = np.zeros(j + 2)
            e[0] = float(beta)
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[0]
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) <= tol * size:
                break
        for i, yi in enumerate(y):
            x = x + float(yi) * Q[i]
        return x

    def diagnostics(self, U, t):
        """[L2 error, norm of the exact solution], [mass, energy, gradient energy]."""
        n = self.n
        ep, ew = _gauss(n + 1)
        E = self.tensor(_lagrange(self.gp, ep)[0])
        _, det, _ = self.metric(ep, ep, ep)
        w = self.tensor(ew)
        w3 = w[:, None, None] * w[:, None] * w
        diff = self.every(E, U) - self.solution(self.positions(ep, ep, ep), t)
        error = math.sqrt(float((det * w3 * diff * diff).sum()))
        gp = self.gp
        cof, det, _ = self.metric(gp, gp, gp)
        jxw = (det * self.w3).expand_as(U)
        ex = self.solution(self.positions(gp, gp, gp), t)
        norm = math.sqrt(float((jxw * ex * ex).sum()))
        du = [self.along(self.D, U, d) for d in range(3)]
        grad = sum(((sum(cof[d][i] * du[d] for d in range(3)) / det) ** 2 for i in range(3)))
        out = [float((jxw * U).sum()), float((jxw * U * U).sum()), float((jxw * grad).sum())]
        return np.array([error, norm]), np.array(out)


def _coefficients(scheme):
    """(a, b) of the published low-storage schemes: Kennedy, Carpenter and
    Lewis 2000 (5_4, 9_5), Tselios and Simos 2007 (3_3, 7_4)."""
    if scheme == "3_3":
        return [0.755726351946097, 0.386954477304099], [0.245170287303492, 0.184896052186740, 0.569933660509768]
    if scheme == "5_4":
        return ([970286171893 / 4311952581923, 6584761158862 / 12103376702013, 2251764453980 / 15575788980749,
                 26877169314380 / 34165994151039],
                [1153189308089 / 22510343858157, 1772645290293 / 4653164025191, -1672844663538 / 4480602732383,
                 2114624349019 / 3568978502595, 5198255086312 / 14908931495163])
    if scheme == "7_4":
        b = [0.0941840925477795334, 0.149683694803496998, 0.285204742060440058, -0.122201846148053668,
             0.0605151571191401122, 0.345986987898399296, 0.186627171718797670]
        g = [0.241566650129646868, 0.0423866513027719953, 0.215602732678803776, 0.232328007537583987,
             0.256223412574146438, 0.0978694102142697230]
        return [x + y for x, y in zip(g, b)], b
    return ([1107026461565 / 5417078080134, 38141181049399 / 41724347789894, 493273079041 / 11940823631197,
             1851571280403 / 6147804934346, 11782306865191 / 62590030070788, 9452544825720 / 13648368537481,
             4435885630781 / 26285702406235, 2357909744247 / 11371140753790],
            [2274579626619 / 23610510767302, 693987741272 / 12394497460941, -347131529483 / 15096185902911,
             1144057200723 / 32081666971178, 1562491064753 / 11797114684756, 13113619727965 / 44346030145118,
             393957816125 / 7825732611452, 720647959663 / 6565743875477, 3559252274877 / 14424734981077])


def exact(case, seed):
    if case["kind"] == "serving":
        requests = _requests(case, seed)
        # whole-mesh tensor steps take about 3 ms each on these meshes
        if sum(r.steps() for r in requests) * 5 * 3e-3 > 18.0:
            return None
        solutions = []
        for r in requests:
            cfg = dict(degree=r.degree, n_cells=(r.n,) * 3, mesh_type=adv.MESH_CARTESIAN, deformation=0.0, periodic=1,
                       velocity=r.velocity, flux_alpha=1.0, initial_condition=adv.IC_SINE_GAUSS,
                       ic_params=tuple(r.phase) + (0.0,) * 5)
            ref = _Reference(cfg)
            U = ref.steps(ref.project(0.0), "5_4", 0.0, r.t_end / r.steps(), r.steps())
            solutions.append(ref.nodal(U).cpu().numpy())
        return {"solutions": solutions, "steps": [None] * len(requests), "errors": None}
    cfg = _config(case, seed)
    dt = _time_step(case, cfg)
    ref = _Reference(cfg)
    U = ref.project(0.0)
    if case["kind"] == "apply":
        return ref.nodal(ref.operator(U, 0.0))
    if case["kind"] == "bdf2":
        first = ref.solve(U / dt, 1.0 / dt, dt, U)
        second = ref.solve((2.0 * first - 0.5 * U) / dt, 1.5 / dt, 2.0 * dt, 2.0 * first - U)
        return {"first": ref.nodal(first), "second": ref.nodal(second)}
    if case["kind"] == "output":
        l2, me = ref.diagnostics(U, 0.05)
        return {"projected": ref.nodal(ref.project(0.05)), "l2": l2, "mass_energy": me}
    count = case["steps"] if case["kind"] in ("steps", "host_steps") else 1
    return ref.nodal(ref.steps(U, case["scheme"], 0.0, dt, count))
