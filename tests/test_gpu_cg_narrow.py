"""The FP64 mass solve on tall meshes around the width and the length at which degrees 1 and 2 change
from the column to the element kernels (column_solve: 64 nodes wide, 950 column CTAs of
16 rows over all systems), against the oracle, graph-launched and host-driven (bitwise the same).

Solver and oracle stop at |r| <= tol |b|: solutions differ by at most 2 tol cond(M) |x|, with
cond(M) at most 40 per axis on these uniform meshes; a step's increment is at most 1e-2 of the
populations (dt e.grad f in lattice units, one cell of a wall layer)."""
import numpy as np
import pytest

from helpers import rel_l2
from lbfem_gpu import cases, make_params

pytestmark = pytest.mark.gpu

TOL = 1e-13
# 8 x 118 and 8 x 119 CTAs; 64 and 65 nodes wide; one system: 950 and 951
STEPS = [("couette", 32, 1886, 1), ("couette", 32, 1890, 1), ("tgv", 30, 943, 2), ("tgv", 30, 945, 2),
         ("couette", 63, 2000, 1), ("tgv", 64, 2000, 1), ("cavity", 4, 3000, 1), ("cavity", 1, 1500, 2)]
SOLVES = [("couette", 3, 15190, 1), ("couette", 3, 15210, 1), ("tgv", 2, 7595, 2), ("tgv", 2, 7605, 2)]


def _case(flow, nx, ny, p):
    tc = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow}.get(flow)
    tc = tc(0.1) if tc else cases.LidDrivenCavity(0.1, 0.0)
    tc.set_reynolds(200.0)
    return tc, cases.build_mesh(tc, nx, p, ny)


@pytest.mark.parametrize("scheme,streaming", [("leelin", "tg2"), ("bardow", "tg3-split")])
@pytest.mark.parametrize("flow,nx,ny,p", STEPS)
def test_steps_on_narrow_meshes(gpu_lib, oracle_mod, flow, nx, ny, p, scheme, streaming, monkeypatch):
    import lbfem_gpu

    tc, m = _case(flow, nx, ny, p)
    prm = make_params(scheme, "cg", cg_tolerance=TOL, cg_max_iterations=2000, streaming=streaming)
    dt, lam = m.time_step(0.2), tc.relaxation_time()
    x, y = m.nodes()
    f0 = tc.initial_populations(x, y, lam)
    out = []
    for k in range(3):
        if k == 1:
            monkeypatch.setenv("LBFEM_TRACE", "1")
        h = oracle_mod.Oracle(m, prm) if k == 2 else lbfem_gpu.Solver(m, prm)
        h.set_time_step(dt, lam)
        h.set_initial_populations(f0)
        h.step(2)
        out.append(h.get_populations())
        h.close()
    assert np.array_equal(out[0], out[1])
    assert rel_l2(out[0], out[2]) <= 2 * 2 * 2 * TOL * 40.0**2 * 1e-2 + 1e-13  # two steps of up to two sweeps


@pytest.mark.parametrize("flow,nx,ny,p", SOLVES)
def test_single_solves_on_narrow_meshes(gpu_lib, oracle_mod, flow, nx, ny, p):
    import lbfem_gpu

    _, m = _case(flow, nx, ny, p)
    prm = make_params("bardow", "cg", cg_tolerance=TOL, cg_max_iterations=2000)
    r = np.random.default_rng(ny).standard_normal(m.n_dofs)
    out = []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        out.append(h.mass_solve(r))
        h.close()
    assert rel_l2(*out) <= 2 * TOL * 40.0**2
