"""The largest meshes whose FP64 mass solve runs in one launch (k_cg_fused, a cluster of 8 CTAs
per system), and the first beyond them: the nodes that a thread holds, the shared memory of
a wide mesh, the cell rows. A solve in one launch adds the same kernels to a step whatever its
iterations, the loop of kernels does not: the launch counts tell which form ran.

Both solvers stop at |r| <= tol |b|: solutions differ by at most 2 tol cond(M) |x|, with
cond(M) the product of the axes' condition numbers, below 40 per axis at p = 1, 2 and 150
at p = 3, 4 on these (nearly uniform) meshes."""
import ctypes as C

import numpy as np
import pytest

from helpers import rel_l2
from lbfem_gpu import cases, make_params

pytestmark = pytest.mark.gpu

TOL = 1e-13
SIZES = [("tgv", 195, 195, 1, True), ("couette", 196, 196, 1, False), ("couette", 96, 96, 2, True),
         ("tgv", 97, 97, 2, False), ("cavity", 67, 67, 3, True), ("tgv", 68, 68, 3, False), ("tgv", 40, 40, 4, True),
         ("couette", 41, 41, 4, False), ("tgv", 1826, 8, 1, True), ("tgv", 1827, 8, 1, False),
         ("cavity", 20, 8, 2, True), ("cavity", 20, 7, 2, False)]


def _case(flow, nx, ny, p):
    tc = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow}.get(flow)
    tc = tc(0.1) if tc else cases.LidDrivenCavity(0.1, 0.5)
    tc.set_reynolds(200.0)
    return tc, cases.build_mesh(tc, nx, p, ny)


def _launches(h):
    its, n = C.c_double(), C.c_int64()
    h._call("last_step_stats", h.h, C.byref(its), C.byref(n))
    return n.value


@pytest.mark.parametrize("flow,nx,ny,p,fits", SIZES)
def test_limits_of_the_one_launch_solve(gpu_lib, oracle_mod, flow, nx, ny, p, fits):
    import lbfem_gpu

    tc, m = _case(flow, nx, ny, p)
    dt, lam = m.time_step(0.2), tc.relaxation_time()
    x, y = m.nodes()
    f0 = tc.initial_populations(x, y, lam)
    counts = []
    for tol in (1e-2, TOL):
        h = lbfem_gpu.Solver(m, make_params("bardow", "cg", cg_tolerance=tol, cg_max_iterations=2000))
        h.set_time_step(dt, lam)
        h.set_initial_populations(f0)
        h.step(1)
        counts.append(_launches(h))
        h.close()
    assert (counts[0] == counts[1]) == fits, counts

    prm = make_params("bardow", "cg", cg_tolerance=TOL, cg_max_iterations=2000)
    rng = np.random.default_rng(nx + ny)
    r, x0 = rng.standard_normal(m.n_dofs), rng.standard_normal(m.n_dofs)
    out = []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        out.append(h.mass_solve(r, x=x0))
        h.close()
    cond = (40.0 if p <= 2 else 150.0) ** 2
    assert rel_l2(*out) <= 2 * TOL * cond
