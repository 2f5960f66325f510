"""The status of a step in which some systems of the FP64 mass solve meet the iteration cap
and others turn non-finite in the same iteration: non-finite, whichever form of
the solve runs (one launch per solve, or the loop of kernels) and whichever
system ends first."""
import numpy as np
import pytest

from helpers import tgv
from lbfem_gpu import LbfemError, NoConvergence, _abi, cases, d2q9, make_params

pytestmark = pytest.mark.gpu


def _populations(oracle_mod, tc, m, dt, lam):
    """Fluid at rest whose density varies much along y and little along x, scaled so that
    r.D^-1 r of the populations along +-y alone overflows FP64: their first alpha is inf / inf,
    while the others take an ordinary first iteration (the right-hand side is linear in the scale)."""
    x, y = m.nodes()
    rho = 1.0 + 0.1 * np.cos(2 * np.pi * y) + 0.001 * np.cos(2 * np.pi * x)
    f = d2q9.equilibrium(rho, 0 * rho, 0 * rho)
    h = oracle_mod.Oracle(m, make_params("bardow", "cg"))
    r, diag = h.advection(f, d2q9.E, dt, lam), h.jacobi_diagonal()
    h.close()
    free = m.independent()
    rz = (r[:, free] ** 2 / diag[free]).sum(axis=1)
    along_y = np.array([d2q9.E[a][0] == 0 for a in range(1, 9)])
    low, high = rz[~along_y].max(), rz[along_y].min()
    assert along_y.sum() == 2 and high > 8 * low
    return f * (np.sqrt(np.finfo(float).max) / (low * high) ** 0.25)


# 32^2 and 48^2: one launch per solve; 260^2 (column tiles) and 80 x 7 Q3 (element tiles): the loop
@pytest.mark.parametrize("host_driven", [False, True])
@pytest.mark.parametrize("nx,ny,p", [(32, 32, 1), (48, 48, 1), (260, 260, 1), (80, 7, 3)])
def test_non_finite_wins_over_the_iteration_cap(gpu_lib, oracle_mod, monkeypatch, nx, ny, p, host_driven):
    import lbfem_gpu

    tc, _ = tgv(8)
    m = cases.build_mesh(tc, nx, p, ny)
    dt, lam = m.time_step(0.3), tc.relaxation_time()
    f = _populations(oracle_mod, tc, m, dt, lam)
    if host_driven:
        monkeypatch.setenv("LBFEM_TRACE", "1")
    h = lbfem_gpu.Solver(m, make_params("bardow", "cg", cg_tolerance=1e-14, cg_max_iterations=1))
    h.set_time_step(dt, lam)
    for _ in range(20):
        h.set_populations(f)
        with pytest.raises(LbfemError) as e:
            h.step(1)
        assert e.value.status == _abi.LBFEM_ERR_NONFINITE and not isinstance(e.value, NoConvergence)
        assert np.array_equal(h.get_populations(), f)  # left as before the failing step
    h.close()
