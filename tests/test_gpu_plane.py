"""The plane marches of the mixed-precision inner iteration on grids whose rows,
tiles and chunks end unevenly: the iterate after a few inner iterations against
the one-kernel-per-operation form."""
import numpy as np
import pytest

import les_cases
import les_gb300 as G

pytestmark = pytest.mark.gpu

# rows of every length modulo four, one and several tiles along j and k, odd
# row counts (a mirrored row in the last pair), the smallest grids the passes take
SHAPES = [(16, 14, 14), (17, 15, 29), (20, 33, 31), (19, 40, 130), (24, 19, 129), (18, 14, 257), (33, 70, 36),
          (16, 97, 64), (16, 50, 300), (70, 16, 16)]


def _iterate(m, b, lmax, pc, deg, fused, cap):
    with G.Context(m) as c:
        c.set_option(G.OPT_FUSED, fused)
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", np.zeros(m.n))
        st, r = c.pcg(G.pcg_opts(precond=pc, max_iter=cap, tol=1e-12 * np.linalg.norm(b), lambda_min=3 * np.pi ** 2,
                                 lambda_max=lmax, degree=max(deg, 1), precision=G.MIXED, inner_rtol=1e-4))
        return st, r.iters, c.download("p")


@pytest.mark.parametrize("pc,deg", [(G.PC_JACOBI, 0)] + [(G.PC_CHEBYSHEV, d) for d in (2, 3, 4, 5, 6, 7)],
                         ids=["jacobi", "cheb2", "cheb3", "cheb4", "cheb5", "cheb6", "cheb7"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_plane_march_follows_unfused(shape, pc, deg):
    h = (0.03, 0.025, 0.04)
    m = G.Mesh(*shape, *h)
    b = np.random.default_rng(sum(shape)).standard_normal(m.n).reshape(shape)
    b[-1] = 0.0
    lmax = 4 * sum(1 / d ** 2 for d in h)
    f = _iterate(m, b.reshape(-1), lmax, pc, deg, 1, 8)
    u = _iterate(m, b.reshape(-1), lmax, pc, deg, 0, 8)
    assert f[:2] == u[:2] == (G.NOT_CONVERGED, 8)
    # eight FP32 iterations, each within some FP32 roundings of the other form
    assert np.max(np.abs(f[2] - u[2])) < 1e-4 * np.max(np.abs(u[2]))


def test_batched_ensemble_of_odd_rows_follows_cases_stepped_alone():
    """A batched ensemble (unpadded rows) of cases whose row lengths are no
    multiple of four takes as many corrections and about as many iterations as
    the cases stepped alone (padded rows)."""
    shapes, h = [(40, 24, 37), (33, 31, 34), (48, 20, 35)], 1.0 / 32

    def setup(c, shape, seed):
        solid = les_cases.box_mask(shape, (8, 14, 6, 12, 9, 15))
        f = les_cases.init_fields(shape, 0.02, seed)
        les_cases.velocity_bcs_np(shape, f, solid)
        c.upload_mask(np.zeros(c.n, np.uint8))
        c.build_stencil()
        lmax = c.lambda_max(20)
        c.upload_mask(solid)
        c.upload_fields(f)
        return G.step_params(nu=1e-5, rho=1.2, cs=0.17, cfl_conv=0.3, rel_tol=1e-8,
                             pcg=G.pcg_opts(precond=G.PC_CHEBYSHEV, max_iter=5000, lambda_min=3 * np.pi ** 2,
                                            lambda_max=lmax, degree=4, precision=G.MIXED, inner_rtol=1e-4))

    with G.Ensemble([G.Mesh(*s, h, h, h) for s in shapes]) as ens:
        together = ens.step([setup(c, s, i) for i, (c, s) in enumerate(zip(ens.cases, shapes))])
    for i, s in enumerate(shapes):
        with G.Context(G.Mesh(*s, h, h, h)) as c:
            alone = c.step(setup(c, s, i))
        assert together[i].status == alone.status == G.OK
        assert together[i].outer == alone.outer, (i, together[i].outer, alone.outer)
        assert abs(together[i].iters - alone.iters) <= max(3, 0.15 * alone.iters), (i, together[i].iters, alone.iters)
