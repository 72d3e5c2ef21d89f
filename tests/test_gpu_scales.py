"""Mixed solves of small right-hand sides: the inner residual is not scaled, so
its squares reach the lower end of FP32's range.  A power of two in the
right-hand side changes no rounding until then, so the solve must go on as the
one-kernel-per-operation form's does -- in one cluster (32x32x32) and by plane
marches (40x64x64)."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu


def _solve(shape, pc, deg, fused, scale):
    m = G.Mesh(*shape, 1 / 32, 1 / 32, 1 / 32)
    b = np.random.default_rng(7).standard_normal(shape)
    b[-1] = 0.0
    b = b.reshape(-1) * scale
    with G.Context(m) as c:
        c.set_option(G.OPT_FUSED, fused)
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        lmax = c.lambda_max(20) * 1.05
        c.upload("b", b)
        c.upload("p", np.zeros(m.n))
        st, r = c.pcg(G.pcg_opts(precond=pc, max_iter=4000, tol=1e-9 * np.linalg.norm(b), lambda_min=lmax / 400,
                                 lambda_max=lmax, degree=max(deg, 1), precision=G.MIXED, inner_rtol=1e-4))
        return st, r.iters, c.download("p") / scale


# 2^-36: p.q falls below 2^-128 before the solve has converged
@pytest.mark.parametrize("e", [0, -20, -36])
@pytest.mark.parametrize("pc,deg", [(G.PC_CHEBYSHEV, 4), (G.PC_JACOBI, 0)], ids=["cheb4", "jacobi"])
@pytest.mark.parametrize("shape", [(32, 32, 32), (40, 64, 64)], ids=["cluster", "plane"])
def test_small_right_hand_sides_converge(shape, pc, deg, e):
    a, u = _solve(shape, pc, deg, 1, 2.0 ** e), _solve(shape, pc, deg, 0, 2.0 ** e)
    assert a[0] == u[0] == G.OK, (a[:2], u[:2])
    assert abs(a[1] - u[1]) <= 0.02 * u[1] + 2
    # both to a residual of 1e-9 ||b||; the smallest eigenvalue is about pi^2 / L^2, L <= 2
    nb = np.linalg.norm(np.random.default_rng(7).standard_normal(shape)[:-1])
    assert np.linalg.norm(a[2] - u[2]) <= 2e-9 * nb * (2 / np.pi) ** 2 * 4
