"""The mass solve in one launch (k_cg_fused): a system's bands of cell rows over the CTAs of
a cluster, at the mesh sizes where the banding can go wrong, against the oracle.

Both solvers stop at |r| <= tol |b|, so their solutions differ by at most
2 tol cond(A) |x| (A = M, or the product of the 1-D matrices of an axis-parallel
TG3 matrix): the tolerance of the comparison."""
import numpy as np
import pytest

from lbfem_gpu import cases, make_params

pytestmark = pytest.mark.gpu

TOL = 1e-12
# the last cell row alone in its band; as many cell rows as CTAs; fewer than 16 (clusters of 8);
# too few for any cluster (the loop of kernels); wide and tall; the last that fits 16 CTAs' registers
SIZES = [("tgv", 9, 17, 1), ("cavity", 20, 16, 1), ("couette", 5, 8, 2), ("cavity", 7, 7, 3), ("couette", 160, 16, 1),
         ("couette", 6, 96, 2), ("tgv", 21, 33, 3), ("cavity", 11, 19, 4), ("tgv", 128, 128, 1), ("cavity", 60, 64, 2),
         ("cavity", 60, 65, 3), ("tgv", 48, 48, 4)]


def _flow(name):
    tc = {"tgv": cases.TaylorGreenVortex, "couette": cases.CouetteFlow, "cavity": cases.LidDrivenCavity}[name](0.1)
    tc.set_reynolds(100.0)
    return tc


def _cond(v, p, periodic, c):
    """The condition number of M + c K on one axis."""
    xi = cases.gauss_lobatto(p)
    q, w = np.polynomial.legendre.leggauss(p + 1)
    q, w = (q + 1) / 2, w / 2
    val, der = np.empty((p + 1, p + 1)), np.empty((p + 1, p + 1))
    for a in range(p + 1):
        poly = np.poly1d([1.0])
        for b in range(p + 1):
            if b != a:
                poly = poly * np.poly1d([1.0, -xi[b]]) / (xi[a] - xi[b])
        val[a], der[a] = poly(q), poly.deriv()(q)
    nc = len(v) - 1
    n = p * nc + (0 if periodic else 1)
    A = np.zeros((n, n))
    for k, h in enumerate(np.diff(v)):
        i = (p * k + np.arange(p + 1)) % n
        A[np.ix_(i, i)] += h * (val * w) @ val.T + c / h * (der * w) @ der.T
    return np.linalg.cond(A)


@pytest.mark.parametrize("e", [None, (1.0, 0.0), (0.0, -1.0)], ids=["mass", "tg3-x", "tg3-y"])
@pytest.mark.parametrize("flow,nx,ny,p", SIZES)
def test_one_launch_solve_matches_the_oracle(gpu_lib, oracle_mod, flow, nx, ny, p, e):
    import lbfem_gpu

    tc = _flow(flow)
    m = cases.build_mesh(tc, nx, p, ny)
    prm = make_params("bardow", "cg", cg_tolerance=TOL, cg_max_iterations=2000)
    rng = np.random.default_rng(nx * 1000 + ny)
    r, x0 = rng.standard_normal(m.n_dofs), rng.standard_normal(m.n_dofs)
    c = 0.0 if e is None else 0.05 * m.h_min**2
    kw = {} if e is None else {"e": e, "tg3_coefficient": c}
    ex, ey = (0.0, 0.0) if e is None else e
    cond = _cond(m.vertex_x, p, m.periodic_x, c * ex * ex) * _cond(m.vertex_y, p, m.periodic_y, c * ey * ey)
    out = []
    for h in (lbfem_gpu.Solver(m, prm), oracle_mod.Oracle(m, prm)):
        out.append(h.mass_solve(r, x=x0, **kw))
        zero = h.mass_solve(np.zeros_like(r), x=x0, **kw)
        assert not zero.any()  # an exactly zero right-hand side: x = 0
        h.close()
    err = np.linalg.norm(out[0] - out[1]) / np.linalg.norm(out[1])
    assert err <= 2 * TOL * cond, (err, cond)
