"""The CG kernels of the FP64 path beyond one cluster (column tiles, cg_column.cuh, and element
tiles, both with their sums in the last CTA) against the oracle: one column tile and
several, tile remainders in both directions, one system and eight, the image column
and row, and meshes of either side of the dispatch.

Both solvers stop at |r| <= tol |b|: solutions differ by at most 2 tol cond(M) |x|, with
cond(M) the product of the axes' condition numbers, below 40 per axis at p = 1, 2 and 150
at p = 3, 4 on these (nearly uniform) meshes."""
import numpy as np
import pytest

from helpers import rel_l2
from lbfem_gpu import cases, make_params

pytestmark = pytest.mark.gpu

TOL = 1e-13
# few cell rows: no cluster takes them. 1, 2 and 5 column tiles; rows of one tile, exact, one over
SIZES = [("tgv", 40, 7, 1), ("couette", 300, 6, 1), ("cavity", 63, 7, 2), ("tgv", 256, 4, 2), ("couette", 130, 5, 2),
         ("cavity", 50, 6, 3), ("tgv", 33, 5, 4)]


def _case(flow, nx, ny, p):
    tc = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow}.get(flow)
    tc = tc(0.1) if tc else cases.LidDrivenCavity(0.1, 0.5)
    tc.set_reynolds(200.0)
    return tc, cases.build_mesh(tc, nx, p, ny)


@pytest.mark.parametrize("e", [None, (1.0, 0.0), (0.0, 1.0)], ids=["mass", "tg3-x", "tg3-y"])
@pytest.mark.parametrize("flow,nx,ny,p", SIZES)
def test_solve_matches_the_oracle(gpu_lib, oracle_mod, flow, nx, ny, p, e):
    import lbfem_gpu

    tc, m = _case(flow, nx, ny, p)
    prm = make_params("bardow", "cg", cg_tolerance=TOL, cg_max_iterations=2000)
    rng = np.random.default_rng(nx + ny)
    r, x0 = rng.standard_normal(m.n_dofs), rng.standard_normal(m.n_dofs)
    kw = {} if e is None else {"e": e, "tg3_coefficient": 0.02 * m.h_min**2}
    out, its = [], []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        out.append(h.mass_solve(r, x=x0, **kw))
        its.append(h.cg_iterations())
        assert not h.mass_solve(np.zeros_like(r), x=x0, **kw).any()
        h.close()
    cond = (40.0 if p <= 2 else 150.0) ** 2
    assert rel_l2(*out) <= 2 * TOL * cond
    assert abs(its[0] - its[1]) <= 0.05 * its[1] + 2


@pytest.mark.parametrize("scheme,streaming", [("leelin", "tg2"), ("bardow", "tg2"), ("bardow", "tg3-split")])
@pytest.mark.parametrize("flow,nx,ny,p", [("tgv", 256, 4, 2), ("couette", 300, 6, 1), ("cavity", 50, 6, 3)])
def test_steps_match_the_oracle(gpu_lib, oracle_mod, flow, nx, ny, p, scheme, streaming, monkeypatch):
    """Whole steps, graph-launched and host-driven (bitwise the same), against the oracle."""
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
        h.step(3)
        out.append(h.get_populations())
        h.close()
    assert np.array_equal(out[0], out[1])
    assert rel_l2(out[0], out[2]) <= 1e-12
