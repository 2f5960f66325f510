"""The column kernels of the FP64 CG at degrees 3 and 4, which take meshes of 10^6 nodes or more,
for the mass matrix those whose rows fill the tiles of 128 columns to three quarters
(column_solve), against the oracle: exactly 10^6 nodes and just below, widths on both sides of the three quarters,
last tiles of one row, walls and periodic axes, the mass matrix and both
axis-parallel TG3 matrices. A step's launches per CG iteration tell which form ran: 2 of the
column kernels, 6 of the element kernels at these sizes.

Both solvers stop at |r| <= tol |b|: solutions differ by at most 2 tol cond(A) |x|; M's condition
number is at most 150 per axis on these (nearly uniform) meshes, and the TG3 term, 0.002 h^2 K
with K <= 600 / h^2 M, raises it by at most 2.2. A step's increment is at most 1e-3 of the
populations."""
import ctypes as C

import numpy as np
import pytest

from helpers import rel_l2
from lbfem_gpu import cases, make_params

pytestmark = pytest.mark.gpu

TOL = 1e-13
# (flow, nx, ny, p, column kernels for the mass matrix); tiles of 18 rows at p = 3, of 16 at p = 4
SIZES = [("tgv", 333, 333, 3, True), ("cavity", 333, 332, 3, False), ("cavity", 346, 336, 3, True),
         ("couette", 42, 2700, 3, True), ("couette", 64, 1730, 3, True), ("couette", 63, 1760, 3, False),
         ("tgv", 250, 250, 4, True), ("couette", 48, 1300, 4, True), ("cavity", 47, 1330, 4, False),
         ("cavity", 254, 252, 4, True)]


def _case(flow, nx, ny, p):
    tc = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow}.get(flow)
    tc = tc(0.1) if tc else cases.LidDrivenCavity(0.1, 0.5)
    tc.set_reynolds(200.0)
    return tc, cases.build_mesh(tc, nx, p, ny)


@pytest.mark.parametrize("e", [None, (1.0, 0.0), (0.0, -1.0)], ids=["mass", "tg3-x", "tg3-y"])
@pytest.mark.parametrize("flow,nx,ny,p,col", SIZES)
def test_solve_matches_the_oracle(gpu_lib, oracle_mod, flow, nx, ny, p, col, e):
    import lbfem_gpu

    _, m = _case(flow, nx, ny, p)
    prm = make_params("bardow", "cg", cg_tolerance=TOL, cg_max_iterations=2000)
    rng = np.random.default_rng(nx + ny)
    r, x0 = rng.standard_normal(m.n_dofs), rng.standard_normal(m.n_dofs)
    kw = {} if e is None else {"e": e, "tg3_coefficient": 0.002 * m.h_min**2}
    out, its = [], []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        out.append(h.mass_solve(r, x=x0, **kw))
        its.append(h.cg_iterations())
        h.close()
    assert rel_l2(*out) <= 2 * TOL * 2.2 * 150.0**2
    assert abs(its[0] - its[1]) <= 0.05 * its[1] + 2


@pytest.mark.parametrize("scheme,streaming", [("leelin", "tg2"), ("bardow", "tg3-split")])
@pytest.mark.parametrize("flow,nx,ny,p,col", SIZES)
def test_steps_match_the_oracle(gpu_lib, oracle_mod, flow, nx, ny, p, col, scheme, streaming):
    import lbfem_gpu

    tc, m = _case(flow, nx, ny, p)
    prm = make_params(scheme, "cg", cg_tolerance=TOL, cg_max_iterations=2000, streaming=streaming)
    dt, lam = m.time_step(0.2), tc.relaxation_time()
    x, y = m.nodes()
    f0 = tc.initial_populations(x, y, lam)
    out = []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        h.set_time_step(dt, lam)
        h.set_initial_populations(f0)
        h.step(1)
        out.append(h.get_populations())
        if len(out) == 1 and streaming == "tg2":
            its, n = C.c_double(), C.c_int64()
            h._call("last_step_stats", h.h, C.byref(its), C.byref(n))
            if its.value >= 16:  # a quarter of the systems may start at their solution
                assert (n.value < 4 * its.value) == col, (n.value, its.value)
        h.close()
    assert rel_l2(*out) <= 2 * 2 * TOL * 2.2 * 150.0**2 * 1e-3 + 1e-13
