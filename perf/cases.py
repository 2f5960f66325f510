"""The work that programs have this framework do, as cases that can be timed.

A program builds a context for a mesh, sets a time step, loads populations and
steps; between diagnostics it stays on the device (Scheme::step,
schemes.h:92-98,118-124). A program that keeps the scheme's loop to itself calls
the operators on its own device vectors instead (advection.h:49-58,
mass.h:185-213, collision.h:105-168). Parameter sweeps step many instances as
one batch. The cases cover these three uses over the meshes, degrees, schemes,
mass solves, streaming variants and precisions of the tests and the benchmark.

A case is a dict of plain values:
  kind       "step", "batch" or "operators"
  flow       "tgv" (doubly periodic), "couette" (periodic in x, walls in y) or
             "cavity" (walls all round, tanh-clustered mesh)
  nx, ny, p  cells per axis and polynomial degree
  scheme     "leelin" or "bardow"; mass "cg", "lumped" or "richardson";
             streaming "tg2", "tg3" or "tg3-split"; precision "fp64" or "mixed"
  tol        relative CG tolerance
  cfl, re, u0, steps
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "lbm-fem_b200"))

CS2 = 1.0 / 3.0
E = [(0, 0), (1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (-1, -1), (0, -1), (1, -1)]
W = [4 / 9, 1 / 9, 1 / 36, 1 / 9, 1 / 36, 1 / 9, 1 / 36, 1 / 9, 1 / 36]
STRETCH = 1.2


def _step(name, flow, nx, ny, p, scheme, mass, precision, cfl, re, u0, steps, tol=1e-8, streaming="tg2"):
    return {"name": name, "kind": "step", "flow": flow, "nx": nx, "ny": ny, "p": p, "scheme": scheme, "mass": mass,
            "precision": precision, "streaming": streaming, "tol": tol, "cfl": cfl, "re": re, "u0": u0, "steps": steps}


def listed():
    return [
        # The smallest calls, where launches and the solver's latency count: the plain
        # FP64 vortex on 64^2 Q1 with a tight CG tolerance, and the start-up Couette
        # flow on a rectangular mesh in mixed precision.
        _step("tgv_q1_64_fp64", "tgv", 64, 64, 1, "bardow", "cg", "fp64", 0.5, 100.0, 0.05, 10, tol=1e-12),
        _step("couette_q1_32x256_mixed", "couette", 32, 256, 1, "leelin", "cg", "mixed", 0.25, 50.0, 0.05, 20),
        # The lid-driven cavity on 128^2 Q2: consistent mass in mixed precision, and the
        # lumped FP64 form that is run to a steady state.
        _step("cavity_q2_128_mixed", "cavity", 128, 128, 2, "bardow", "cg", "mixed", 0.4, 400.0, 0.1, 20),
        _step("cavity_q2_128_lumped_fp64", "cavity", 128, 128, 2, "bardow", "lumped", "fp64", 0.4, 400.0, 0.1, 20),
        # An ordinary mesh of odd size at the highest degree, in FP64 with the default tolerance.
        _step("cavity_q4_101x77_fp64", "cavity", 101, 77, 4, "leelin", "cg", "fp64", 0.25, 400.0, 0.1, 5),
        # Split TG3 streaming (two sweeps of direction-dependent solves per step), odd size.
        _step("tgv_q2_191_tg3split_fp64", "tgv", 191, 191, 2, "bardow", "cg", "fp64", 0.8, 400.0, 0.05, 5,
              streaming="tg3-split"),
        # The largest mesh, in both precisions: the throughput workload.
        _step("tgv_q3_1024_mixed", "tgv", 1024, 1024, 3, "leelin", "cg", "mixed", 0.5, 100.0, 0.05, 10),
        _step("tgv_q3_1024_fp64", "tgv", 1024, 1024, 3, "leelin", "cg", "fp64", 0.5, 100.0, 0.05, 5),
        # A parameter sweep: 64 instances of uneven size, half cavities, half vortices.
        {"name": "batch_64_mixed", "kind": "batch", "n": 64, "table": 20261203, "cfl": 0.4, "steps": 10},
        # A program that keeps the scheme's loop and calls the operators on its own
        # device vectors: one Lee-Lin step of equilibrium, advection, 8 mass solves and
        # the predictor-corrector.
        {"name": "operators_q2_256_fp64", "kind": "operators", "flow": "cavity", "nx": 256, "ny": 256, "p": 2,
         "scheme": "leelin", "mass": "cg", "precision": "fp64", "streaming": "tg2", "tol": 1e-8, "cfl": 0.25,
         "re": 400.0, "u0": 0.1},
    ]


def _log(rng, a, b):
    return a * (b / a) ** rng.random()


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["batch"] + ["operators"] * 2)
    if kind == "batch":
        return {"kind": "batch", "n": int(round(_log(rng, 4, 64))), "table": rng.randrange(1 << 30), "cfl": 0.4,
                "steps": rng.randrange(4, 11)}
    flow = rng.choice(["tgv", "couette", "cavity"])
    p = rng.randrange(1, 5)
    # nodes over the range of the listed meshes, the aspect up to 8 either way where the mesh is uniform
    nodes = _log(rng, 4e3, 4e6) if kind == "step" else _log(rng, 4e3, 5e5)
    aspect = _log(rng, 0.125, 8.0) if flow == "couette" else _log(rng, 0.7, 1.4)
    edge = math.sqrt(nodes) / p
    nx, ny = max(8, int(edge * math.sqrt(aspect))), max(8, int(edge / math.sqrt(aspect)))
    case = {"kind": kind, "flow": flow, "nx": nx, "ny": ny, "p": p, "scheme": rng.choice(["leelin", "bardow"]),
            "mass": rng.choice(["cg", "cg", "cg", "lumped", "richardson"]), "precision": rng.choice(["fp64", "mixed"]),
            "streaming": "tg2", "tol": rng.choice([1e-8, 1e-8, 1e-10]), "cfl": 0.25,
            "re": _log(rng, 100.0, 1000.0), "u0": 0.05 + 0.05 * rng.random()}
    if kind == "operators":
        case.update(scheme="leelin", precision="fp64", mass=rng.choice(["cg", "cg", "lumped"]))
    else:
        case["steps"] = rng.randrange(4, 11)
        if case["scheme"] == "bardow" and case["mass"] == "cg" and case["precision"] == "fp64" and rng.random() < 0.3:
            case.update(streaming=rng.choice(["tg3", "tg3-split"]), flow="tgv")
    return case


# ------------------------------------------------------------------ the meshes
def _batch_cases(case):
    """The instances of a batch: uneven edges, degrees 1 and 2, Re log-uniform in
    [100, 1000], U0 in [0.05, 0.1]; cavities with Bardow, vortices with Lee-Lin."""
    rng = np.random.RandomState(case["table"] % (1 << 31))
    out = []
    for k in range(case["n"]):
        flow = "cavity" if k % 2 == 0 else "tgv"
        edge, p = int(rng.choice([32, 48, 64, 96, 128, 192, 256])), int(rng.choice([1, 2]))
        out.append({"kind": "step", "flow": flow, "nx": edge, "ny": edge, "p": p,
                    "scheme": "bardow" if flow == "cavity" else "leelin", "mass": "cg", "precision": "mixed",
                    "streaming": "tg2", "tol": 1e-8, "cfl": case["cfl"], "re": float(100.0 * 10 ** rng.rand()),
                    "u0": float(0.05 + 0.05 * rng.rand()), "steps": case["steps"]})
    return out


def _flow(case):
    """The test case of the package for a case."""
    from lbfem_gpu import cases

    mach = case["u0"] / math.sqrt(CS2)
    if case["flow"] == "tgv":
        tc = cases.TaylorGreenVortex(mach, 1, 1, shift=(0.25, 0.25), chapman_enskog=False)
    elif case["flow"] == "couette":
        tc = cases.CouetteFlow(mach)
    else:
        tc = cases.LidDrivenCavity(mach, STRETCH)
    tc.set_reynolds(case["re"])
    return tc


def _cluster(x):
    return 0.5 * (1.0 + np.tanh(STRETCH * (2.0 * x - 1.0)) / math.tanh(STRETCH))


def _vertices(case):
    v = [np.linspace(0.0, 1.0, n + 1) for n in (case["nx"], case["ny"])]
    return [_cluster(a) for a in v] if case["flow"] == "cavity" else v


def _times(case):
    """The time step and the relaxation time."""
    h = min(1.0 / case["nx"], 1.0 / case["ny"])
    if case["flow"] == "cavity":
        h = float(_cluster(np.float64(h)))
    return case["cfl"] * h / case["p"] ** 2, case["u0"] / case["re"] / CS2


def _points(p):
    if p == 1:
        return np.array([0.0, 1.0])
    inner = np.sort(np.polynomial.legendre.Legendre.basis(p).deriv().roots().real)
    return (np.concatenate([[-1.0], inner, [1.0]]) + 1.0) / 2.0


def _axis_nodes(v, p):
    return np.concatenate([(v[:-1, None] + np.diff(v)[:, None] * _points(p)[None, :-1]).ravel(), v[-1:]])


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _equilibrium(rho, ux, uy):
    uu = ux * ux + uy * uy
    out = torch.empty((9,) + tuple(rho.shape), dtype=rho.dtype, device=rho.device)
    for a, (ex, ey) in enumerate(E):
        eu = ex * ux + ey * uy
        out[a] = W[a] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu)
    return out


def _populations(case, seed):
    """Populations of a flow under way, on the GPU: the case's base flow plus a few
    smooth modes drawn from the seed (5% of U0), at equilibrium."""
    rng = np.random.RandomState(seed % (1 << 31))
    dev = _device()
    vx, vy = _vertices(case)
    x = torch.from_numpy(_axis_nodes(vx, case["p"])).to(dev)[None, :]
    y = torch.from_numpy(_axis_nodes(vy, case["p"])).to(dev)[:, None]
    u0, two_pi = case["u0"], 2.0 * math.pi
    flow = case["flow"]
    if flow == "tgv":
        sx, sy = rng.rand(2)
        ux = u0 * torch.sin(two_pi * (x + sx)) * torch.cos(two_pi * (y + sy))
        uy = -u0 * torch.cos(two_pi * (x + sx)) * torch.sin(two_pi * (y + sy))
    elif flow == "couette":
        ux = u0 * y * torch.ones_like(x)
        uy = torch.zeros_like(x * y)
    else:
        g = 16.0 * x * x * (1 - x) * (1 - x)
        ux = 0.3 * u0 * g * (2 * y * (1 - y) * (1 - y) - 2 * y * y * (1 - y)) * 4
        uy = -0.3 * u0 * 16.0 * (2 * x * (1 - x) * (1 - x) - 2 * x * x * (1 - x)) * 4 * y * y * (1 - y) * (1 - y)
    rho = torch.ones_like(x * y)
    for _ in range(3):
        kx, ky = rng.randint(1, 4, size=2)
        a, b, c = (0.05 * u0 * (2 * rng.rand(3) - 1)).tolist()
        px, py = (two_pi * rng.rand(2)).tolist()
        wx = torch.sin(two_pi * kx * x + px) if flow != "cavity" else torch.sin(math.pi * kx * x)
        wy = torch.sin(two_pi * ky * y + py) if flow == "tgv" else torch.sin(math.pi * ky * y)
        ux = ux + a * wx * wy
        uy = uy + b * wx * wy
        rho = rho + c * u0 * wx * wy
    return _equilibrium(rho, ux, uy).reshape(9, -1).contiguous()


# ------------------------------------------------------------- prepare and run
def _solver(case):
    import lbfem_gpu
    from lbfem_gpu import cases, make_params

    mesh = cases.build_mesh(_flow(case), case["nx"], case["p"], case["ny"])
    s = lbfem_gpu.Solver(mesh, make_params(case["scheme"], case["mass"], cg_tolerance=case["tol"],
                                           precision=case["precision"], streaming=case["streaming"]))
    s.set_time_step(*_times(case))
    return s


def prepare(case, seed):
    if case["kind"] == "batch":
        import lbfem_gpu

        inst = _batch_cases(case)
        solvers = [_solver(c) for c in inst]
        f = [_populations(c, seed + 7 * k) for k, c in enumerate(inst)]
        return {"kind": "batch", "steps": case["steps"], "solvers": solvers, "f": f,
                "out": [torch.empty_like(a) for a in f], "batch": lbfem_gpu.Batch(solvers)}
    f = _populations(case, seed)
    state = {"kind": case["kind"], "solver": _solver(case), "f": f, "out": torch.empty_like(f)}
    if case["kind"] == "step":
        state["steps"] = case["steps"]
    else:
        state["dt"], state["lam"] = _times(case)
        state["e"] = np.array(E, dtype=np.float64)
        state["feq"] = torch.empty_like(f)
        state["rhs"], state["x"] = torch.empty_like(f[:8]), torch.empty_like(f[:8])
    return state


def run(state):
    stream = torch.cuda.current_stream().cuda_stream
    if state["kind"] == "step":
        s = state["solver"]
        s.set_populations_dev(state["f"].data_ptr(), stream)
        s.step_stream(state["steps"], stream)
        s.get_populations_dev(state["out"].data_ptr(), stream)
        return state["out"]
    if state["kind"] == "batch":
        for s, f in zip(state["solvers"], state["f"]):
            s.set_populations_dev(f.data_ptr(), stream)
        torch.cuda.current_stream().synchronize()  # the batch runs on a stream of its own
        state["batch"].step(state["steps"])
        for s, out in zip(state["solvers"], state["out"]):
            s.get_populations_dev(out.data_ptr(), stream)
        return state["out"]
    s, f, feq, rhs, x, out = (state[k] for k in ("solver", "f", "feq", "rhs", "x", "out"))
    dt, lam = state["dt"], state["lam"]
    s.compute_equilibrium_dev(f.data_ptr(), feq.data_ptr(), stream)
    s.advection_dev(f.data_ptr(), state["e"], dt, lam, rhs.data_ptr(), kind="leelin", feq=feq.data_ptr(), stream=stream)
    x.zero_()
    for a in range(8):
        s.mass_solve_dev(x[a].data_ptr(), rhs[a].data_ptr(), stream=stream)
    out.copy_(f)
    s.predictor_corrector_dev(out.data_ptr(), feq.data_ptr(), x.data_ptr(), dt / lam, stream)
    return {"f": out, "rhs": rhs, "x": x, "feq": feq}


def work(case):
    """Bytes and operations of one pass. A step reads and writes the 9 populations
    and, with the consistent mass, reads the two increments its solve starts from
    and writes the new one. Operations: the 1-D element products of the
    right-hand side (3 for an axis population, 8 for a diagonal one), one tensor
    mass apply and one tensor mass solve per system, and 150 per node for the
    nodal maps."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    p = case["p"]
    n = (p * case["nx"] + (case["flow"] == "cavity")) * (p * case["ny"] + (case["flow"] != "tgv"))
    product = 2.0 * (p + 1) ** 2 / p
    flops = n * (44 * product + 150.0)
    if case["mass"] == "cg":
        flops += n * 8 * 4 * product
    elif case["mass"] == "richardson":
        flops += n * 8 * 2 * 2 * product
    if case["kind"] == "operators":
        # f read; feq, r, x and the new f written
        return {"bytes": 8.0 * n * (9 + 9 + 8 + 8 + 9), "flops": flops}
    size = 4.0 if case["precision"] == "mixed" else 8.0
    per_step = n * size * (18 + (24 if case["mass"] == "cg" else 0))
    return {"bytes": 2 * 8.0 * 9 * n + case["steps"] * per_step, "flops": case["steps"] * flops}


# ---------------------------------------------------------------------- exact
class _Axis:
    """The 1-D matrices of an axis on its distinct nodes, dense, in 64 bits: mass M,
    derivative C = int l_a l_b', stiffness K, the lumped mass, and the rows of the
    normal derivative at the two ends."""

    def __init__(self, v, p, periodic, dev):
        xi = _points(p)
        q, w = np.polynomial.legendre.leggauss(p + 1)
        q, w = (q + 1) / 2, w / 2
        val, der = np.empty((p + 1, p + 1)), np.empty((p + 1, p + 1))
        ends = np.empty((2, p + 1))
        for a in range(p + 1):
            poly = np.poly1d([1.0])
            for b in range(p + 1):
                if b != a:
                    poly = poly * np.poly1d([1.0, -xi[b]]) / (xi[a] - xi[b])
            val[a], der[a] = poly(q), poly.deriv()(q)
            ends[:, a] = poly.deriv()(0.0), poly.deriv()(1.0)
        m, c, k = (val * w) @ val.T, (val * w) @ der.T, (der * w) @ der.T
        nc = len(v) - 1
        n = p * nc + (0 if periodic else 1)
        h = np.diff(v)
        idx = (p * np.arange(nc)[:, None] + np.arange(p + 1)[None, :]) % n
        rows, cols = np.repeat(idx, p + 1, axis=1).ravel(), np.tile(idx, (1, p + 1)).ravel()

        def dense(el, scale):
            out = torch.zeros((n, n), dtype=torch.float64, device=dev)
            vals = torch.from_numpy((scale[:, None] * el.ravel()[None, :]).ravel()).to(dev)
            return out.index_put_((torch.from_numpy(rows).to(dev), torch.from_numpy(cols).to(dev)), vals, accumulate=True)

        self.n, self.periodic = n, periodic
        self.M, self.C, self.K = dense(m, h), dense(c, np.ones(nc)), dense(k, 1.0 / h)
        self.lump = self.M.sum(dim=1)
        self.d0, self.d1 = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
        if not periodic:
            self.d0[: p + 1] = torch.from_numpy(ends[0] / h[0]).to(dev)
            self.d1[n - p - 1:] = torch.from_numpy(ends[1] / h[-1]).to(dev)


class _Exact:
    """One case's operators in 64 bits, as dense 1-D products on the distinct nodes.
    The nodal maps run on all stored nodes: a periodic image updates its own value
    and gets no increment."""

    def __init__(self, case):
        dev = _device()
        self.case, p = case, case["p"]
        vx, vy = _vertices(case)
        self.X = _Axis(vx, p, case["flow"] != "cavity", dev)
        self.Y = _Axis(vy, p, case["flow"] == "tgv", dev)
        self.shape = (p * case["ny"] + 1, p * case["nx"] + 1)
        self.dt, self.lam = _times(case)
        self.wall = torch.zeros(self.shape, dtype=torch.bool, device=dev)
        self.uw = torch.zeros(self.shape, dtype=torch.float64, device=dev)
        if case["flow"] == "couette":
            self.wall[0], self.wall[-1] = True, True
            self.uw[-1] = case["u0"]
        elif case["flow"] == "cavity":
            self.wall[0], self.wall[-1], self.wall[:, 0], self.wall[:, -1] = True, True, True, True
            self.uw[-1, 1:-1] = case["u0"]
        if case["mass"] == "cg":
            self.Mxi, self.Myi = torch.linalg.inv(self.X.M), torch.linalg.inv(self.Y.M)

    def inner(self, f):
        return f[: self.Y.n, : self.X.n]

    def moments(self, f, impose):
        rho = f.sum(dim=0)
        mx = f[1] + f[2] + f[8] - f[4] - f[5] - f[6]
        my = f[2] + f[3] + f[4] - f[6] - f[7] - f[8]
        ux, uy = mx / rho, my / rho
        if impose:
            ux, uy = torch.where(self.wall, self.uw, ux), torch.where(self.wall, torch.zeros_like(uy), uy)
        return rho, ux, uy

    def feq(self, f, impose):
        return _equilibrium(*self.moments(f, impose))

    def rhs(self, f, feq, a, b, e, remove):
        """The right-hand sides of the 8 moving populations (distinct nodes)."""
        X, Y, c = self.X, self.Y, -0.5 * self.dt ** 2
        out, face = [], []
        for k in range(1, 9):
            ex, ey = e[k]
            u = self.inner(f[k])
            h = a * u if feq is None else a * u + b * self.inner(feq[k])
            r = torch.zeros_like(u)
            if ex:
                r += Y.M @ (ex * (h @ X.C.T) + c * ex * ex * (u @ X.K.T))
            if ey:
                r += (ey * (Y.C @ h) + c * ey * ey * (Y.K @ u)) @ X.M.T
            if ex and ey:
                r += c * ex * ey * ((Y.C @ u) @ X.C + (Y.C.T @ u) @ X.C.T)
            out.append(r)
            s = torch.zeros_like(u)
            half = 0.5 * self.dt ** 2
            if not Y.periodic and ey:
                for line, d, n in ((0, Y.d0, -1.0), (-1, Y.d1, 1.0)):
                    s[line] += half * n * ey * (ex * (X.C @ u[line]) + ey * (X.M @ (d @ u)))
            if not X.periodic and ex:
                for line, d, n in ((0, X.d0, -1.0), (-1, X.d1, 1.0)):
                    s[:, line] += half * n * ex * (ey * (Y.C @ u[:, line]) + ex * (Y.M @ (u @ d)))
            face.append(s)
        if not (X.periodic and Y.periodic):
            flux = sum(face)
            for k in range(8):
                out[k] = out[k] + face[k] - (W[k + 1] / (1.0 - W[0]) * flux if remove else 0.0)
        return out

    def solve(self, r):
        if self.case["mass"] == "cg":
            return self.Myi @ r @ self.Mxi.T
        inv = 1.0 / (self.Y.lump[:, None] * self.X.lump[None, :])
        x = inv * r
        if self.case["mass"] == "richardson":
            for _ in range(2):
                x = x + inv * (r - self.Y.M @ x @ self.X.M.T)
        return x

    def sweep(self, g, s):
        """One sweep of split TG3 on the collided populations g."""
        c = self.dt ** 2 / 6.0
        e = [(ex if s == 0 else 0, ey if s == 1 else 0) for ex, ey in E]
        r = self.rhs(g, None, -self.dt, 0.0, e, True)
        ax, ay = self.X.M, self.Y.M
        if s == 0:
            ax = ax + c * self.X.K
        else:
            ay = ay + c * self.Y.K
        ixt, iy = torch.linalg.inv(ax).T, torch.linalg.inv(ay)
        for k in range(1, 9):
            if e[k] != (0, 0):
                self.inner(g[k]).add_(iy @ r[k - 1] @ ixt)

    def step(self, f):
        if self.case["scheme"] == "leelin":
            fe = self.feq(f, True)
            b = -0.5 * self.dt ** 2 / self.lam
            return self.correct(f, fe, [self.solve(r) for r in self.rhs(f, fe, -self.dt - b, b, E, False)])
        omega = self.dt / (self.lam + 0.5 * self.dt)
        g = self.feq(f, True) + (1.0 - omega) * (f - self.feq(f, False))
        if self.case["streaming"] == "tg3-split":
            self.sweep(g, 0)
            self.sweep(g, 1)
            return g
        for k, r in enumerate(self.rhs(g, None, -self.dt, 0.0, E, True)):
            self.inner(g[k + 1]).add_(self.solve(r))
        return g

    def correct(self, f, fe, x):
        th = self.dt / self.lam
        fh = f + th * fe
        for k in range(8):
            self.inner(fh[k + 1]).add_(x[k])
        fh = fh / (1.0 + th)
        return fh + th * (self.feq(fh, True) - fe)


def exact(case, seed):
    if case["kind"] == "batch":
        return [exact(c, seed + 7 * k) for k, c in enumerate(_batch_cases(case))]
    if case["streaming"] == "tg3":
        return None  # its matrix has no tensor-product inverse
    ex = _Exact(case)
    f = _populations(case, seed).reshape((9,) + ex.shape)
    if case["kind"] == "step":
        for _ in range(case["steps"]):
            f = ex.step(f)
        return f.reshape(9, -1)
    fe = ex.feq(f, True)
    b = -0.5 * ex.dt ** 2 / ex.lam
    r = ex.rhs(f, fe, -ex.dt - b, b, E, False)
    x = [ex.solve(a) for a in r]
    out = ex.correct(f, fe, x)

    def stored(blocks):
        full = torch.zeros((8,) + ex.shape, dtype=torch.float64, device=f.device)
        for k, a in enumerate(blocks):
            full[k, : ex.Y.n, : ex.X.n] = a
        return full.reshape(8, -1)

    return {"f": out.reshape(9, -1), "rhs": stored(r), "x": stored(x), "feq": fe.reshape(9, -1)}
