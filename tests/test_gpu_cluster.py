"""The inner solve in one thread-block cluster (small grids): the iterate after
a few inner iterations against the one-kernel-per-operation form, and the same
solve to its tolerance by the plane marches (which run while kernels are
timed)."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu

# one to several planes per block, evenly and not; row lengths of every
# remainder modulo four; one and several thread groups per plane range; a plane
# of as many vectors as a block has threads
SHAPES = [(16, 14, 14), (17, 15, 29), (31, 16, 18), (33, 33, 32), (40, 21, 67), (64, 32, 32), (70, 16, 16), (95, 17, 20),
          (18, 64, 40), (130, 14, 15)]
PCS = [(G.PC_JACOBI, 0)] + [(G.PC_CHEBYSHEV, d) for d in (2, 3, 4, 5, 6, 7)]
IDS = ["jacobi", "cheb2", "cheb3", "cheb4", "cheb5", "cheb6", "cheb7"]
H = (0.03, 0.025, 0.04)


def _solve(m, b, pc, deg, fused, cap, tol, passes=False):
    with G.Context(m) as c:
        c.set_option(G.OPT_FUSED, fused)
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", np.zeros(m.n))
        if passes:
            c.profile(1)
        st, r = c.pcg(G.pcg_opts(precond=pc, max_iter=cap, tol=tol * np.linalg.norm(b), lambda_min=3 * np.pi ** 2,
                                 lambda_max=4 * sum(1 / d ** 2 for d in H), degree=max(deg, 1), precision=G.MIXED,
                                 inner_rtol=1e-4))
        return st, r, c.download("p")


def _rhs(shape):
    b = np.random.default_rng(sum(shape)).standard_normal(shape)
    b[-1] = 0.0
    return b.reshape(-1)


@pytest.mark.parametrize("pc,deg", PCS, ids=IDS)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_cluster_follows_unfused(shape, pc, deg):
    m, b = G.Mesh(*shape, *H), _rhs(shape)
    f = _solve(m, b, pc, deg, 1, 8, 1e-12)
    u = _solve(m, b, pc, deg, 0, 8, 1e-12)
    assert (f[0], f[1].iters) == (u[0], u[1].iters) == (G.NOT_CONVERGED, 8)
    # eight FP32 iterations, each within some FP32 roundings of the other form
    assert np.max(np.abs(f[2] - u[2])) < 1e-4 * np.max(np.abs(u[2]))


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_cluster_solves_as_plane_marches(shape):
    """To a residual of 1e-9 ||b||: both stop there, so the solutions are within
    the sum of two such residuals over the smallest eigenvalue, about pi^2 / L^2
    with L the domain's longest side."""
    m, b = G.Mesh(*shape, *H), _rhs(shape)
    f = _solve(m, b, G.PC_CHEBYSHEV, 4, 1, 5000, 1e-9)
    p = _solve(m, b, G.PC_CHEBYSHEV, 4, 1, 5000, 1e-9, passes=True)
    assert f[0] == p[0] == G.OK
    assert f[1].outer == p[1].outer and abs(f[1].iters - p[1].iters) <= max(3, 0.1 * p[1].iters)
    side = max(n * d for n, d in zip(shape, H))
    assert np.linalg.norm(f[2] - p[2]) <= 2e-9 * np.linalg.norm(b) * (side / np.pi) ** 2 * 4
