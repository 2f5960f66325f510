"""The streaming right-hand side on meshes of few tiles, where several CTAs share a tile's
populations (split_of), against the oracle: one tile, tiles with remainders, and tile
counts on both sides of each change of the split; every mode of the FP64 kernel and,
by a step, the FP32 pair kernel against the FP64 one.

A right-hand side is a sum of at most 4 (2p + 1)^2 products of O(1) factors, so two
correctly rounded evaluations differ by less than 1e-12 relative (1e5 roundings); the
mixed step keeps the velocity to 1e-5, its stated bound."""
import numpy as np
import pytest

from helpers import random_populations, rel_l2
from lbfem_gpu import cases, d2q9, make_params

pytestmark = pytest.mark.gpu

# (flow, nx, ny, p): 1, 2 x 2, 18 / 19, 36 / 40, 72 / 78, 144 / 152 tiles of the FP64 kernel
SIZES = [("cavity", 3, 5, 1), ("tgv", 65, 25, 1), ("couette", 190, 140, 1), ("cavity", 66, 70, 2), ("tgv", 62, 70, 3),
         ("cavity", 130, 110, 2), ("couette", 95, 75, 4), ("tgv", 260, 284, 2)]


def _case(flow, nx, ny, p):
    tc = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow, "cavity": cases.LidDrivenCavity}[flow](0.1)
    tc.set_reynolds(400.0)
    return tc, cases.build_mesh(tc, nx, p, ny)


@pytest.mark.parametrize("kind", ["taylor_galerkin", "leelin"])
@pytest.mark.parametrize("flow,nx,ny,p", SIZES)
def test_advection_of_few_tiles(gpu_lib, oracle_mod, flow, nx, ny, p, kind):
    import lbfem_gpu

    tc, m = _case(flow, nx, ny, p)
    f = random_populations(m, seed=nx)
    dt, lam = m.time_step(0.25), tc.relaxation_time()
    out = []
    for h in (lbfem_gpu.Solver(m, make_params("bardow", "lumped")), oracle_mod.Oracle(m, make_params("bardow", "lumped"))):
        feq = h.compute_equilibrium(f) if kind == "leelin" else None
        out.append(h.advection(f, d2q9.E, dt, lam, kind=kind, feq=feq))
        h.close()
    assert rel_l2(*out) <= 1e-12


@pytest.mark.parametrize("scheme", ["leelin", "bardow"])
@pytest.mark.parametrize("flow,nx,ny,p", SIZES)
def test_steps_of_few_tiles(gpu_lib, oracle_mod, flow, nx, ny, p, scheme):
    import lbfem_gpu

    tc, m = _case(flow, nx, ny, p)
    dt, lam = m.time_step(0.25), tc.relaxation_time()
    x, y = m.nodes()
    f0 = tc.initial_populations(x, y, lam)
    out = []
    for make, precision in ((lbfem_gpu.Solver, "fp64"), (oracle_mod.Oracle, "fp64"), (lbfem_gpu.Solver, "mixed")):
        h = make(m, make_params(scheme, "lumped", precision=precision))
        h.set_time_step(dt, lam)
        h.set_initial_populations(f0)
        h.step(2)
        out.append(h.get_populations())
        h.close()
    assert rel_l2(out[0], out[1]) <= 1e-12
    u = [np.stack(d2q9.moments(f)[1:]) for f in out]
    assert rel_l2(u[2], u[1]) <= 1e-5
