"""The element kernels of the FP64 CG on both sides of the CTA counts at which they end with the
sums and scalar work of a phase instead of leaving them to further launches (tail_solve),
against the oracle: the general TG3 matrix at every degree with eight systems and one, the
mass matrix at degrees 3 and 4, and steps graph-launched and host-driven (bitwise the same).

Solver and oracle stop at |r| <= tol |b|: solutions differ by at most 2 tol cond(A) |x|; the
TG3 coefficients are small enough that cond(A) <= 2 cond(M), and M's is at most 40^2 at
p = 1, 2 and 150^2 at p = 3, 4 on these uniform meshes. A step's increment is at most
1e-3 of the populations here (dt e.grad f with u = 0.06 and wave number 25)."""
import numpy as np
import pytest

from helpers import rel_l2
from lbfem_gpu import cases, make_params

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _tiles(nx, ny, p):
    """Tiles of 64 x 24 nodes (63 and 60 wide at p = 3, 4)."""
    w = {1: 64, 2: 64, 3: 63, 4: 60}[p]
    return -(-(p * nx + 1) // w) * -(-(p * ny + 1) // 24)


# 8 x 150 and 8 x 152 CTAs at p = 1 .. 3; at p = 4 the mass changes at 2200 (275 and 280 tiles)
STEPS = [("tg2", 3, 199, 119, 150, True), ("tg2", 3, 160, 150, 152, False), ("tg2", 4, 164, 149, 275, True),
         ("tg2", 4, 149, 167, 280, False), ("tg3", 1, 639, 359, 150, True), ("tg3", 1, 511, 455, 152, False),
         ("tg3", 2, 159, 359, 150, True), ("tg3", 2, 255, 227, 152, False), ("tg3", 3, 199, 119, 150, True),
         ("tg3", 4, 119, 110, 152, False)]


@pytest.mark.parametrize("streaming,p,nx,ny,tiles,tail", STEPS)
def test_steps_around_the_change(gpu_lib, oracle_mod, streaming, p, nx, ny, tiles, tail, monkeypatch):
    import lbfem_gpu

    assert _tiles(nx, ny, p) == tiles
    tc = cases.TaylorGreenVortex(0.1)
    tc.set_reynolds(200.0)
    m = cases.build_mesh(tc, nx, p, ny)
    prm = make_params("bardow", "cg", cg_tolerance=TOL, cg_max_iterations=2000, streaming=streaming)
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
    cond = (40.0 if p <= 2 else 150.0) ** 2 * (1 if streaming == "tg2" else 2)
    assert rel_l2(out[0], out[2]) <= 2 * 2 * TOL * cond * 1e-3 + 1e-13  # two steps, and rounding


# one system: 2400 and 2480 tiles
@pytest.mark.parametrize("p,nx,ny,tiles", [(1, 2559, 1439, 2400), (1, 2559, 1487, 2480),
                                           (2, 1279, 719, 2400), (2, 1279, 743, 2480)])
def test_single_solves_around_the_change(gpu_lib, oracle_mod, p, nx, ny, tiles):
    import lbfem_gpu

    assert _tiles(nx, ny, p) == tiles
    tc = cases.CouetteFlow(0.1)
    tc.set_reynolds(200.0)
    m = cases.build_mesh(tc, nx, p, ny)
    tol = 1e-10  # keeps the oracle's solve short
    prm = make_params("bardow", "cg", cg_tolerance=tol, cg_max_iterations=2000)
    rng = np.random.default_rng(nx + ny)
    r = rng.standard_normal(m.n_dofs)
    out = []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        out.append(h.mass_solve(r, e=(1.0, -1.0), tg3_coefficient=0.002 * m.h_min**2))
        h.close()
    assert rel_l2(*out) <= 2 * tol * 2 * 40.0**2
