"""The streaming right-hand side where the CTAs per tile change (split_of: 8 to 37 tiles, 4 to 74,
2 to 148, else 1), at every degree against the oracle; and batches, whose instances share
the GPU and split less: every instance ends bitwise where its own steps take it.

A right-hand side is a sum of at most 4 (2p + 1)^2 products of O(1) factors, so two
correctly rounded evaluations differ by less than 1e-12 relative (1e5 roundings)."""
import numpy as np
import pytest

from helpers import random_populations, rel_l2, setup_case
from lbfem_gpu import cases, d2q9, make_params

pytestmark = pytest.mark.gpu

WIDTH = {1: 64, 2: 64, 3: 63, 4: 60}  # nodes of a tile; 24 rows
# tiles along x and y; the cells of a mesh with that many, whatever the degree
TILES = [(1, 37), (2, 19), (2, 37), (3, 25), (4, 37), (10, 15)]


def _cells(n_tiles, width, p):
    """The fewest cells whose p n + 1 nodes need n_tiles tiles, and one more if that fits."""
    n = (width * (n_tiles - 1)) // p
    while p * n + 1 <= width * (n_tiles - 1):
        n += 1
    return n + 1 if p * (n + 1) + 1 <= width * n_tiles else n


@pytest.mark.parametrize("kind", ["taylor_galerkin", "leelin"])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("tx,ty", TILES)
def test_advection_at_the_changes(gpu_lib, oracle_mod, tx, ty, p, kind):
    import lbfem_gpu

    nx, ny = max(2, _cells(tx, WIDTH[p], p)), _cells(ty, 24, p)
    assert -(-(p * nx + 1) // WIDTH[p]) == tx and -(-(p * ny + 1) // 24) == ty
    tc = cases.CouetteFlow(0.1)
    tc.set_reynolds(400.0)
    m = cases.build_mesh(tc, nx, p, ny)
    f = random_populations(m, seed=nx + ny)
    dt, lam = m.time_step(0.25), tc.relaxation_time()
    prm = make_params("bardow", "lumped")
    out = []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        feq = h.compute_equilibrium(f) if kind == "leelin" else None
        out.append(h.advection(f, d2q9.E, dt, lam, kind=kind, feq=feq))
        h.close()
    assert rel_l2(*out) <= 1e-12


# the FP64 kernel has one tile shape, the FP32 one three
@pytest.mark.parametrize("scheme", ["leelin", "bardow"])
@pytest.mark.parametrize("mass,precision,shape", [("lumped", "fp64", "0"), ("richardson", "fp64", "0"), ("cg", "fp64", "0")]
                         + [(m, "mixed", s) for m in ("lumped", "richardson") for s in ("0", "alt", "small")])
def test_batches_split_less(gpu_lib, monkeypatch, mass, precision, scheme, shape):
    """2 and 11 instances of all degrees, whose tiles alone are split 8, 4 and 2 times."""
    import lbfem_gpu

    monkeypatch.setenv("LBFEM_TUNE", shape)
    table = [("tgv", 60, 1), ("cavity", 130, 2), ("tgv", 20, 4), ("cavity", 70, 3), ("couette", 380, 1), ("tgv", 35, 2),
             ("cavity", 45, 4), ("couette", 25, 3), ("cavity", 8, 1), ("tgv", 100, 2), ("couette", 60, 4)]
    flows = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow, "cavity": cases.LidDrivenCavity}
    for n in (2, 11):
        batched, single = [], []
        for flow, nx, p in table[:n]:
            tc = flows[flow](0.1)
            tc.set_reynolds(300.0)
            m = cases.build_mesh(tc, nx, p)
            prm = make_params(scheme, mass, precision=precision, cg_tolerance=1e-6)
            for hs in (batched, single):
                hs.append(setup_case(lbfem_gpu.Solver, tc, m, prm, m.time_step(0.3), tc.relaxation_time()))
        b = lbfem_gpu.Batch(batched)
        b.step(3)
        b.close()
        for hb, hs in zip(batched, single):
            hs.step(3)
            assert np.array_equal(hb.get_populations(), hs.get_populations())
            hb.step(1)  # alone again
            hs.step(1)
            assert np.array_equal(hb.get_populations(), hs.get_populations())
            hb.close()
            hs.close()
