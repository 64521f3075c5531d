"""The work that programs built on this solver have it do, as measurable cases.

A case is one run of the time loop through the package's `Solver`: the state
goes in from (pinned) host memory, some steps are integrated, and the fields
and the turbine loads come back, as in a restart, a coupled program or a
parameter study; one case runs the discrete adjoint instead.  Meshes, inflow,
turbines and solvers are the ones of `casegen.config`: wall-stretched 20 x 5 x 5
domains, 5-8 % seeded noise, up to three rotors in a row.

BiCGStab solves run to the case's iteration cap.  Every iteration amplifies the
rounding of the sums before it (measured against another summation order: p
moves by 1e-11 after 20 iterations with the Jacobi preconditioner, by 4e-8
after 16 with SOR, and by 1e-4 after 40), so a small fixed count is where two
builds have the same result; a developed flow on the largest grid takes 26.
Mixed-precision results are taken in single precision, the precision that form
stores its fields in.
"""
import importlib
import math
import os
import tempfile

import numpy as np
import torch

dalm = importlib.import_module("3dalm_b200")
casegen = importlib.import_module("3dalm_b200.casegen")

GC = 2
CAP, CAP_SOR_PC = 16, 8  # BiCGStab iterations per solve, FP64 form
HUBS = (4.0, 9.0, 14.0)
YAWS = (0.0, 10.0, 0.0)
EXACT_CELL_ITERATIONS = 3.0e9  # exact() below this many cell updates only


def _case(name, nx, ny, nz, solver, steps, **over):
    c = dict(name=name, kind="steps", nx=nx, ny=ny, nz=nz, solver=solver, pc="Jacobi",
             precision="fp64", max_it=CAP, tol=1e-8, steps=steps, dt=5e-4, turbines=0,
             loglaw=False, points=32, van_albada=False, average=False)
    c.update(over)
    return c


def listed():
    return [
        # the smallest calls: one step of a 3.5k-cell box, red-black SOR (latency and launches)
        _case("sor_24x12x12", 24, 12, 12, "SOR", 1, max_it=200, tol=1e-6, dt=1e-3),
        # a small rotor study, one turbine
        _case("bicg_40x20x20_rotor", 40, 20, 20, "BiCG", 2, turbines=1, points=8, dt=1e-3),
        # the 128x64x64 configuration: red-black SOR at its 1000-iteration cap
        _case("sor_128x64x64", 128, 64, 64, "SOR", 1, max_it=1000, tol=1e-6),
        # point-Jacobi pressure solver on several partial tiles
        _case("jacobi_72x20x100", 72, 20, 100, "Jacobi", 1, max_it=200, tol=1e-6),
        # SOR-preconditioned BiCGStab, odd sizes
        _case("bicg_sorpc_101x45x67", 101, 45, 67, "BiCG", 2, pc="SOR", max_it=CAP_SOR_PC),
        # Jacobi-preconditioned BiCGStab on a ragged grid with a rotor
        _case("bicg_131x75x53_rotor", 131, 75, 53, "BiCG", 3, turbines=1),
        # three rotors in a log-law inflow, smooth limiter, running time average
        _case("bicg_256x128x64_rotors", 256, 128, 64, "BiCG", 3, turbines=3, loglaw=True,
              van_albada=True, average=True),
        # the largest configuration in FP64: three rotors, 16.8 M cells
        _case("bicg_512x256x128_rotors", 512, 256, 128, "BiCG", 4, turbines=3, loglaw=True),
        # mixed precision (FP32 fields, FP64 refinement): small, ragged in z, and the largest
        _case("mixed_64x32x40_rotor", 64, 32, 40, "BiCG", 5, precision="mixed", turbines=1,
              loglaw=True, max_it=2000),
        _case("mixed_160x96x72_rotors", 160, 96, 72, "BiCG", 5, precision="mixed", turbines=3,
              loglaw=True, max_it=2000),
        _case("mixed_512x256x128_rotors", 512, 256, 128, "BiCG", 24, precision="mixed", turbines=3,
              loglaw=True, max_it=2000),
        # backward: gradient of the turbines' power over 8 steps (yaw, pitch, rotor speed)
        _case("gradient_64x32x32_rotors", 64, 32, 32, "BiCG", 8, kind="gradient", turbines=3,
              loglaw=True, van_albada=True),
    ]


def _coarsest(nx, ny, nz):
    """Cells of the coarsest multigrid level (pairs merge along x and y while
    even and at least 4, along z after that, down to 512 cells)."""
    while nx * ny * nz > 512:
        mx, my = nx % 2 == 0 and nx >= 4, ny % 2 == 0 and ny >= 4
        if mx or my:
            nx, ny = nx // 2 if mx else nx, ny // 2 if my else ny
        elif nz % 2 == 0 and nz >= 4:
            nz //= 2
        else:
            break
    return nx * ny * nz


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["bicg", "bicg", "bicg", "bicg", "sor", "sor", "jacobi", "sorpc", "mixed",
                       "mixed", "gradient"])
    while True:
        nx, ny, nz = size(16, 512), size(10, 256), size(8, 128)
        cells = nx * ny * nz
        if kind == "mixed":
            nx, ny = max(16, nx // 16 * 16), max(8, ny // 8 * 8)
            nz = max(8, nz // 4 * 4)
            if 15_000 <= cells <= 8_000_000 and _coarsest(nx, ny, nz) <= 512:
                break
        elif kind == "gradient":
            nx, ny, nz = max(32, nx // 32 * 32), max(16, ny // 16 * 16), max(8, nz // 8 * 8)
            if 15_000 <= nx * ny * nz <= 300_000 and _coarsest(nx, ny, nz) <= 512:
                break
        elif kind == "bicg":
            if 3_000 <= cells <= 12_000_000:
                break
        elif 3_000 <= cells <= 800_000:
            break
    turbines = rng.choice([0, 1, 2, 3]) if kind in ("bicg", "mixed") else 3 if kind == "gradient" else 0
    common = dict(turbines=turbines, loglaw=kind == "gradient" or (turbines > 0 and rng.random() < 0.7),
                  points=rng.choice([8, 16, 32]), van_albada=kind == "gradient" or rng.random() < 0.3,
                  average=kind == "bicg" and rng.random() < 0.3,
                  dt=rng.choice([1e-3, 5e-4, 2e-4]) if nz <= 64 else 5e-4 if nz <= 100 else 1e-4)
    steps = rng.choice([1, 2, 3, 4])
    if kind == "sor":
        c = _case("", nx, ny, nz, "SOR", 1, max_it=rng.choice([100, 300, 1000]), tol=1e-6, **common)
    elif kind == "jacobi":
        c = _case("", nx, ny, nz, "Jacobi", 1, max_it=rng.choice([100, 300]), tol=1e-6, **common)
    elif kind == "sorpc":
        c = _case("", nx, ny, nz, "BiCG", steps, pc="SOR", max_it=CAP_SOR_PC, **common)
    elif kind == "mixed":
        c = _case("", nx, ny, nz, "BiCG", steps, precision="mixed", max_it=2000, **common)
    elif kind == "gradient":
        c = _case("", nx, ny, nz, "BiCG", 2 + steps, kind="gradient", **common)
    else:
        c = _case("", nx, ny, nz, "BiCG", steps, **common)
    del c["name"]
    return c


def _spec(case):
    t = [casegen.Turbine(base=(x, 2.5, 0.0), yaw_deg=y, omega=12.0)
         for x, y in zip(HUBS[:case["turbines"]], YAWS)]
    return casegen.CaseSpec(
        "case", (case["nx"], case["ny"], case["nz"]), dt=case["dt"], steps=1_000_000,
        solver=case["solver"], pc=case["pc"], tol=case["tol"], max_it=case["max_it"], turbines=t,
        points_per_blade=case["points"], intensity=0.08 if case["loglaw"] else 0.05,
        loglaw=(0.05, 1e-3) if case["loglaw"] else None,
        tavg_start_time=0.0 if case["average"] else 1e30)


def _initial(case, spec, mesh, seed):
    """Mean inflow plus seeded Gaussian noise on the interior, [NX][NY][NZ][3], on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    prof = casegen.inflow_profile(spec, mesh)
    if prof is None:
        mean = torch.tensor(spec.uin, dtype=torch.float64, device="cuda").expand(*mesh.size, 3)
    else:
        mean = torch.as_tensor(prof, device="cuda")[None].expand(*mesh.size, 3)
    U = mean.clone()
    noise = torch.randn(*spec.n, 3, generator=g, dtype=torch.float64, device="cuda")
    U[GC:-GC, GC:-GC, GC:-GC] += spec.intensity * noise
    return U, prof


def prepare(case, seed):
    spec = _spec(case)
    mixed = case["precision"] == "mixed"
    with tempfile.TemporaryDirectory() as d:
        mesh = casegen.write_case(spec, d)
        solver = dalm.Solver(d, device=0, precision=dalm.MIXED if mixed else dalm.FP64,
                             limiter=dalm.VAN_ALBADA if case["van_albada"] else dalm.MINMOD)
    U, prof = _initial(case, spec, mesh, seed)
    if prof is not None:
        solver.set_inflow_profile(prof)
    solver.advance_clock()  # step 0 integrates nothing
    s = dict(case=case, solver=solver, mixed=mixed,
             U=torch.empty(U.shape, dtype=torch.float64, pin_memory=True),
             p=torch.zeros(U.shape[:3], dtype=torch.float64, pin_memory=True))
    s["U"].copy_(U)
    for name in ("U", "p") + (("Utavg",) if case["average"] else ()):
        s["out_" + name] = torch.empty_like(s["p" if name == "p" else "U"], pin_memory=True)
        if mixed:
            s["single_" + name] = torch.empty(s["out_" + name].shape, dtype=torch.float32)
    return s


def run(s):
    case, solver = s["case"], s["solver"]
    solver.set_state(s["U"].numpy(), p=s["p"].numpy())
    if case["kind"] == "gradient":
        t0 = solver.stats()["step"]
        J, grad = solver.power_gradient(t0 + case["steps"] // 2, t0 + case["steps"] - 1,
                                        ckpt_every=max(1, case["steps"] // 2))
        return {"J": J, "grad": grad}
    solver.step(case["steps"])
    out = {}
    for name in ("U", "p") + (("Utavg",) if case["average"] else ()):
        solver.field(name, out=s["out_" + name].numpy())
        if s["mixed"]:
            s["single_" + name].copy_(s["out_" + name])
            out[name] = s["single_" + name]
        else:
            out[name] = s["out_" + name]
    if case["turbines"]:
        thrust, torque, power = solver.turbines()
        kind = np.float32 if s["mixed"] else np.float64
        out.update(thrust=thrust.astype(kind), torque=torque.astype(kind), power=power.astype(kind))
    if not s["mixed"]:
        out["iterations"] = solver.stats()["it"]
    return out


def work(case):
    """The state in and out of every step once (U, JU, f, p; 4-byte U, JU, f in
    the mixed form), and per solver iteration the vectors it cannot keep
    anywhere but in memory on large grids, each read and written once."""
    n = case["nx"] * case["ny"] * case["nz"]
    e = 4 if case["precision"] == "mixed" else 8
    step_bytes = n * (e * 15 + 16)
    step_flops = n * 500
    if case["precision"] == "mixed":
        it, it_bytes, it_flops = 3, 36, 200  # e, p, r, q, b in single precision
    elif case["solver"] == "BiCG":
        it, it_bytes, it_flops = case["max_it"], 72, 130  # x, r, r0, p, q read; x, r, p, q written
    else:
        it, it_bytes, it_flops = case["max_it"], 24, 35  # x, b read; x written
    steps = case["steps"] * (3 if case["kind"] == "gradient" else 1)
    return {"bytes": float(steps * (step_bytes + it * n * it_bytes) + n * 8 * 8),
            "flops": float(steps * (step_flops + it * n * it_flops))}


# ---- the same steps in plain torch, 64 bits -------------------------------------


class _Plain:
    """One case's time step (explicit predictor, pressure solve, projection,
    boundary conditions, actuator line) as whole-array torch expressions."""

    def __init__(self, case, device):
        self.case, self.dev = case, device
        self.spec = _spec(case)
        self.mesh = casegen.make_mesh(*self.spec.n)
        self.prof = casegen.inflow_profile(self.spec, self.mesh)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)  # noqa: E731
        ax = (self.mesh.x, self.mesh.y, self.mesh.z)
        shp = ((-1, 1, 1), (1, -1, 1), (1, 1, -1))
        self.c = [t(a).reshape(s) for a, s in zip(ax, shp)]
        self.d = [t(casegen.spacing(a)).reshape(s) for a, s in zip(ax, shp)]
        self.c1 = [t(a) for a in ax]
        if self.prof is None:
            self.inflow = t(self.spec.uin).expand(len(ax[1]), len(ax[2]), 3)
        else:
            self.inflow = t(self.prof)
        self.I = (slice(GC, -GC),) * 3
        # coefficients per axis on the interior: upper, lower neighbour
        self.co = []
        diag = 0
        for a in range(3):
            x, dx = self.c[a], self.d[a]
            i = self._ax(a, 0)
            up = 1 / (dx[i] * (x[self._ax(a, 1)] - x[i]))
            lo = 1 / (dx[i] * (x[i] - x[self._ax(a, -1)]))
            first, last = torch.zeros_like(up), torch.zeros_like(up)
            first.reshape(-1)[0] = 1
            last.reshape(-1)[-1] = 1
            lo, up = lo * (1 - first), up * (1 - last)
            extra = last * 2 / (dx[i] * dx[i]) if a == 0 else 0  # p = 0 at the outlet
            diag = diag - up - lo - extra
            self.co.append((up, lo))
        self.md = float(diag.abs().max())
        self.co = [(u / self.md, l / self.md) for u, l in self.co]
        self.ac = diag / self.md
        n = self.spec.n
        par = sum(torch.arange(GC, GC + m, device=device).reshape(s) for m, s in zip(n, shp)) % 2
        self.color = [(par == q) for q in (0, 1)]

    def _ax(self, a, o):
        """Index of the interior shifted by o along axis a only, for a per-axis array."""
        s = [slice(None)] * 3
        n = self.mesh.size[a]
        s[a] = slice(GC + o, n - GC + o)
        return tuple(s)

    def sh(self, f, a, o):
        """Interior cells of f shifted by o along axis a."""
        s = [slice(GC, n - GC) for n in f.shape[:3]]
        s[a] = slice(GC + o, f.shape[a] - GC + o)
        return f[tuple(s)]

    # -- pressure solve
    def apply(self, x):
        v = self.ac * x
        for a in range(3):
            up, lo = self.co[a]
            n = x.shape[a]
            v.narrow(a, 0, n - 1).add_(up.narrow(a, 0, n - 1) * x.narrow(a, 1, n - 1))
            v.narrow(a, 1, n - 1).add_(lo.narrow(a, 1, n - 1) * x.narrow(a, 0, n - 1))
        return v

    def sor(self, x, b, w):
        for q in (0, 1):
            x = torch.where(self.color[q], x + w * (b - self.apply(x)) / self.ac, x)
        return x

    def rms(self, r):
        return math.sqrt(float((r * r).sum())) / math.sqrt(r.numel())

    def precondition(self, p):
        spec = self.spec
        x = p / self.ac if spec.pc == "Jacobi" else torch.zeros_like(p)
        for _ in range(spec.pc_max_it - 1 if spec.pc == "Jacobi" else spec.pc_max_it):
            x = x + (p - self.apply(x)) / self.ac if spec.pc == "Jacobi" else self.sor(x, p, spec.pc_relax)
        return x

    def solve(self, x, b):
        spec, it = self.spec, 0
        if spec.solver != "BiCG":
            while True:
                x = self.sor(x, b, spec.relax) if spec.solver == "SOR" else x + (b - self.apply(x)) / self.ac
                it += 1
                if not (it < spec.max_it and self.rms(b - self.apply(x)) > spec.tol):
                    return x, it
        r = b - self.apply(x)
        r0, p, q = r.clone(), r, torch.zeros_like(r)
        rho, alpha, omega = float((r0 * r).sum()), 1.0, 1.0
        while True:
            if it:
                beta = (rho / old) * (alpha / omega)
                p = r + beta * (p - omega * q)
            pp = self.precondition(p)
            q = self.apply(pp)
            alpha = rho / float((r0 * q).sum())
            s = r - alpha * q
            ss = self.precondition(s)
            t = self.apply(ss)
            omega = float((t * s).sum()) / float((t * t).sum())
            x = x + alpha * pp + omega * ss
            r = s - omega * t
            it += 1
            if not (it < spec.max_it and self.rms(r) > spec.tol):
                return x, it
            old, rho = rho, float((r0 * r).sum())

    # -- flow
    def flux_pair(self, v, a, J):
        """Upwind fluxes through the upper faces of the interior cells and of
        the layer below along axis a: (upper, lower) per interior cell."""
        kap = 1 / 3
        f = [self.sh(v, a, o) for o in (-2, -1, 0, 1, 2)]

        def states(fm, fc, fp, fpp):
            d1, d2, d3 = fc - fm, fp - fc, fpp - fp
            if self.case["van_albada"]:
                sw = lambda x, y: (2 * x * y + 1e-12) / (x * x + y * y + 1e-12)  # noqa: E731
                sl, sr = sw(d2, d1), sw(d3, d2)
                left = fc + sl / 4 * ((1 - kap * sl) * d1 + (1 + kap * sl) * d2)
                right = fp - sr / 4 * ((1 - kap * sr) * d3 + (1 + kap * sr) * d2)
                return left, right
            b = (3 - kap) / (1 - kap)
            mm = lambda x, y: torch.sign(x) * torch.clamp(  # noqa: E731
                torch.minimum(x.abs(), torch.sign(x) * b * y), min=0)
            left = fc + 0.25 * ((1 - kap) * mm(d1, d2) + (1 + kap) * mm(d2, d1))
            right = fp - 0.25 * ((1 - kap) * mm(d3, d2) + (1 + kap) * mm(d2, d3))
            return left, right

        out = []
        for o in (0, -1):
            left, right = states(*f[1 + o:5 + o])
            Jf = self.sh(J, a, o)
            out.append(0.5 * (Jf * (right + left) - Jf.abs() * (right - left)))
        return out

    def predict(self, U, JU, F):
        I, vol = self.I, self.d[0][self._ax(0, 0)] * self.d[1][self._ax(1, 0)] * self.d[2][self._ax(2, 0)]
        G = [[(self.sh(U[m], a, 1) - self.sh(U[m], a, -1)) /
              (self.c[a][self._ax(a, 1)] - self.c[a][self._ax(a, -1)]) for a in range(3)] for m in range(3)]
        shear = torch.sqrt(2 * (G[0][0] ** 2 + G[1][1] ** 2 + G[2][2] ** 2) + (G[0][1] + G[1][0]) ** 2 +
                           (G[0][2] + G[2][0]) ** 2 + (G[1][2] + G[2][1]) ** 2)
        del G
        visc = 1 / self.spec.re + (self.spec.cs * vol ** (1 / 3)) ** 2 * shear
        new = [u.clone() for u in U]
        for m in range(3):
            u = U[m]
            conv = diff = 0
            for a in range(3):
                up, lo = self.flux_pair(u, a, JU[a])
                conv = conv + up - lo
                x = self.c[a]
                i, e, w = self._ax(a, 0), self._ax(a, 1), self._ax(a, -1)
                diff = diff + ((self.sh(u, a, 1) - u[I]) / (x[e] - x[i]) -
                               (u[I] - self.sh(u, a, -1)) / (x[i] - x[w])) / self.d[a][i]
            new[m][I] = u[I] + self.spec.dt * (-conv / vol + visc * diff + F[m])
        return new

    def face_bc(self, JU):
        j = self.I[1], self.I[2]
        yz = self.d[1][:, GC:-GC] * self.d[2][:, :, GC:-GC]
        JU[0][GC - 1, j[0], j[1]] = (yz[0] * self.inflow[GC:-GC, GC:-GC, 0])
        JU[1][GC:-GC, GC - 1, GC:-GC] = 0
        JU[1][GC:-GC, -GC - 1, GC:-GC] = 0
        JU[2][GC:-GC, GC:-GC, GC - 1] = 0
        JU[2][GC:-GC, GC:-GC, -GC - 1] = 0

    def area(self, a):
        b = [self.d[q] for q in range(3) if q != a]
        return b[0] * b[1]

    def faces(self, U):
        JU = [torch.zeros_like(u) for u in U]
        for a in range(3):
            n = U[a].shape[a]
            s = U[a] * self.area(a)
            JU[a].narrow(a, 0, n - 1).copy_(0.5 * (s.narrow(a, 0, n - 1) + U[a].narrow(a, 1, n - 1) * self.area(a)))
        self.face_bc(JU)
        return JU

    def divergence(self, JU):
        vol = self.d[0][self._ax(0, 0)] * self.d[1][self._ax(1, 0)] * self.d[2][self._ax(2, 0)]
        return sum(JU[a][self.I] - self.sh(JU[a], a, -1) for a in range(3)) / vol

    def pressure_bc(self, p):
        h = self.d[0].reshape(-1)
        p[GC - 1, GC:-GC, GC:-GC] = p[GC, GC:-GC, GC:-GC]
        p[-GC, GC:-GC, GC:-GC] = -p[-GC - 1, GC:-GC, GC:-GC] * (0.5 * h[-GC] / (0.5 * h[-GC - 1]))
        p[GC:-GC, GC - 1, GC:-GC] = p[GC:-GC, GC, GC:-GC]
        p[GC:-GC, -GC, GC:-GC] = p[GC:-GC, -GC - 1, GC:-GC]
        p[GC:-GC, GC:-GC, GC - 1] = p[GC:-GC, GC:-GC, GC]
        p[GC:-GC, GC:-GC, -GC] = p[GC:-GC, GC:-GC, -GC - 1]

    def project(self, U, JU, p):
        dt = self.spec.dt
        for a in range(3):
            n = p.shape[a]
            x = self.c[a]
            g = (p.narrow(a, 1, n - 1) - p.narrow(a, 0, n - 1)) / (x.narrow(a, 1, n - 1) - x.narrow(a, 0, n - 1))
            JU[a].narrow(a, 0, n - 1).sub_(dt * self.area(a) * g)
            U[a][self.I] -= dt * (self.sh(p, a, 1) - self.sh(p, a, -1)) / (x[self._ax(a, 1)] - x[self._ax(a, -1)])
        self.face_bc(JU)

    def velocity_bc(self, U, V):
        dt, R = self.spec.dt, slice(GC, -GC)
        h = self.d[0].reshape(-1)
        for m in range(3):
            U[m][:GC, R, R] = self.inflow[R, R, m]
        for i in range(U[0].shape[0] - GC, U[0].shape[0]):  # convective outflow
            uout = U[0][i, R, R].clone()
            for m in range(3):
                f0, f1, f2 = (V[m][i - o, R, R] for o in (0, 1, 2))
                U[m][i, R, R] = f0 - uout * dt * ((3 * f0 - 4 * f1 + f2) / 2) / h[i]

        def quad(x0, x1, x2, f0, f1, f2, x3):
            return (f0 * (((x3 - x1) * (x3 - x2)) / ((x0 - x1) * (x0 - x2))) +
                    f1 * (((x3 - x0) * (x3 - x2)) / ((x1 - x0) * (x1 - x2))) +
                    f2 * (((x3 - x0) * (x3 - x1)) / ((x2 - x0) * (x2 - x1))))

        for a in (1, 2):
            x, d = self.c1[a], self.d[a].reshape(-1)
            n = len(x)
            for side in (0, 1):
                j0, j1, out = ((n - GC - 2, n - GC - 1, (n - GC, n - GC + 1)) if side
                               else (GC + 1, GC, (GC - 1, GC - 2)))
                wall = x[j1] + 0.5 * d[j1] if side else x[j1] - 0.5 * d[j1]
                for m in range(3):
                    at = lambda j: (R, j, R) if a == 1 else (R, R, j)  # noqa: E731
                    f0, f1 = U[m][at(j0)], U[m][at(j1)]
                    slip = m != a and (a == 1 or side)
                    f2 = f1 if slip else torch.zeros_like(f1)
                    for j in out:
                        U[m][at(j)] = quad(x[j0], x[j1], wall, f0, f1, f2, x[j])

    # -- actuator line: per turbine and blade point
    def blades(self, U, t):
        spec, I = self.spec, self.I
        F = [torch.zeros(spec.n, dtype=torch.float64, device=self.dev) for _ in range(3)]
        if not spec.turbines:
            return F, None, None
        js = casegen.windturbine_json(spec)
        foil = js["blade"]["airfoil"]
        r_st = np.array([f["r/R"] for f in foil])
        dr = (spec.rotor_r - spec.hub_r) / spec.points_per_blade
        width = casegen.projection_width(self.mesh, spec)
        ax = (self.mesh.x, self.mesh.y, self.mesh.z)
        Uh = [u.cpu().numpy() for u in U] if U[0].numel() < 3e6 else None
        thrust, torque = np.zeros(len(spec.turbines)), np.zeros(len(spec.turbines))
        atk_list = np.array(js["blade"]["attack angle"])
        for w, tb in enumerate(spec.turbines):
            yaw = math.radians(tb.yaw_deg)
            cy, sy = math.cos(-yaw), math.sin(-yaw)

            def rot(v):
                return np.array([cy * v[0] + sy * v[1], -sy * v[0] + cy * v[1], v[2]])

            for bl in range(spec.blades):
                th = bl * (2 * math.pi / spec.blades) + t * tb.omega
                for q in range(spec.points_per_blade):
                    r = spec.hub_r + (q + 0.5) * dr
                    at = rot([-spec.overhang, r * math.cos(th), spec.tower + r * math.sin(th)])
                    pos = at + np.array(tb.base)
                    idx = [int(np.searchsorted(c, v, side="right")) - 1 for c, v in zip(ax, pos)]
                    if any(not GC <= i < len(c) - GC for i, c in zip(idx, ax)):
                        continue
                    fr = [(v - c[i]) / (c[i + 1] - c[i]) for c, i, v in zip(ax, idx, pos)]
                    u = []
                    for m in range(3):
                        src = Uh[m] if Uh is not None else U[m]
                        v8 = src[idx[0]:idx[0] + 2, idx[1]:idx[1] + 2, idx[2]:idx[2] + 2]
                        v8 = v8 if Uh is not None else v8.cpu().numpy()
                        vx = v8[0] * (1 - fr[0]) + v8[1] * fr[0]
                        vy = vx[0] * (1 - fr[1]) + vx[1] * fr[1]
                        u.append(vy[0] * (1 - fr[2]) + vy[1] * fr[2])
                    c, s = math.cos(yaw), math.sin(yaw)
                    ur = (c * u[0] + s * u[1], -s * u[0] + c * u[1], u[2])
                    ut = r * tb.omega + ur[1] * math.sin(th) - ur[2] * math.cos(th)
                    u2 = ur[0] ** 2 + ut ** 2
                    phi = math.atan(ur[0] / ut)
                    st = min(int(np.searchsorted(r_st, r, side="right")) - 1, len(r_st) - 2)
                    a1 = (r - r_st[st]) / (r_st[st + 1] - r_st[st])
                    mix = lambda key: (1 - a1) * np.asarray(foil[st][key]) + a1 * np.asarray(foil[st + 1][key])  # noqa: E731
                    atk = phi * 180 / math.pi - float(mix("twist[deg]"))
                    cd, cl = np.interp(atk, atk_list, mix("Cd")), np.interp(atk, atk_list, mix("Cl"))
                    fd, fl = (0.5 * k * u2 * float(mix("chord/R")) * dr for k in (cd, cl))
                    fx = fl * math.cos(phi) + fd * math.sin(phi)
                    ft = (fl * math.sin(phi) - fd * math.cos(phi)) * np.sign(tb.omega)
                    force = rot([-fx, ft * math.sin(th), -ft * math.cos(th)])
                    torque[w] += abs(ft) * r
                    thrust[w] += fx
                    e = [torch.exp(-((self.c[a][self._ax(a, 0)] - pos[a]) / width) ** 2) for a in range(3)]
                    lo = [int((e[a] > 1e-20).nonzero()[:, a].min()) if bool((e[a] > 1e-20).any()) else 0 for a in range(3)]
                    hi = [int((e[a] > 1e-20).nonzero()[:, a].max()) + 1 if bool((e[a] > 1e-20).any()) else 0 for a in range(3)]
                    box = tuple(slice(l, h) for l, h in zip(lo, hi))
                    g = 1 / (width * math.sqrt(math.pi)) ** 3
                    for a in range(3):
                        g = g * e[a].narrow(a, lo[a], hi[a] - lo[a])
                    for m in range(3):
                        F[m][box] += force[m] * g
        return F, thrust, torque

    def steps(self, U0, p0, n, first):
        spec = self.spec
        U = [U0[..., m].clone() for m in range(3)]
        p = p0.clone()
        self.velocity_bc(U, [u.clone() for u in U])
        JU = self.faces(U)
        F, thrust, torque = self.blades(U, spec.dt * first)
        avg = [torch.zeros_like(u) for u in U]
        it = 0
        for k in range(n):
            V = U
            U = self.predict(V, JU, F)
            JU = self.faces(U)
            b = self.divergence(JU) / (spec.dt * self.md)
            p[self.I], it = self.solve(p[self.I].clone(), b)
            self.pressure_bc(p)
            self.project(U, JU, p)
            self.velocity_bc(U, V)
            F, thrust, torque = self.blades(U, spec.dt * (first + k))
            avg = [(1 - 1 / (k + 1)) * a + u / (k + 1) for a, u in zip(avg, U)]
        return torch.stack(U, -1), p, torch.stack(avg, -1), thrust, torque, it


def exact(case, seed):
    """None for the gradient (it differentiates a solve run to convergence),
    for the pressure of the mixed form (determined to the solver's tolerance
    only) and for runs beyond some seconds."""
    n = case["nx"] * case["ny"] * case["nz"]
    mixed = case["precision"] == "mixed"
    cost = n * case["steps"] * (300 if mixed else case["max_it"])
    if case["kind"] == "gradient" or cost > EXACT_CELL_ITERATIONS:
        return None
    plain = _Plain(case, "cuda")
    U0, _ = _initial(case, plain.spec, plain.mesh, seed)
    p0 = torch.zeros(U0.shape[:3], dtype=torch.float64, device="cuda")
    U, p, avg, thrust, torque, it = plain.steps(U0, p0, case["steps"], 1)
    out = {"U": U, "p": None if mixed else p}
    if case["average"]:
        out["Utavg"] = avg
    if case["turbines"]:
        omega = np.array([abs(t.omega) for t in plain.spec.turbines])
        out.update(thrust=thrust, torque=torque, power=torque * omega)
    if not mixed:
        out["iterations"] = it
    return out
