"""The plane marches on grids that one cluster would serve (they run while
kernels are timed): rows, tiles and chunks that end unevenly, against the
one-kernel-per-operation form after a few inner iterations."""
import numpy as np
import pytest

import les_gb300 as G

pytestmark = pytest.mark.gpu

SHAPES = [(16, 14, 14), (17, 15, 29), (20, 33, 31), (24, 19, 129), (70, 16, 16), (18, 14, 18)]
H = (0.03, 0.025, 0.04)


def _iterate(shape, pc, deg, fused):
    m = G.Mesh(*shape, *H)
    b = np.random.default_rng(sum(shape)).standard_normal(shape)
    b[-1] = 0.0
    b = b.reshape(-1)
    with G.Context(m) as c:
        c.set_option(G.OPT_FUSED, fused)
        c.upload_mask(np.zeros(m.n, np.uint8))
        c.build_stencil()
        c.upload("b", b)
        c.upload("p", np.zeros(m.n))
        c.profile(1)
        st, r = c.pcg(G.pcg_opts(precond=pc, max_iter=8, tol=1e-12 * np.linalg.norm(b), lambda_min=3 * np.pi ** 2,
                                 lambda_max=4 * sum(1 / d ** 2 for d in H), degree=max(deg, 1), precision=G.MIXED,
                                 inner_rtol=1e-4))
        launches = {k: n for k, (n, _) in c.profile_all().items()}
        return st, r.iters, c.download("p"), launches


@pytest.mark.parametrize("pc,deg", [(G.PC_JACOBI, 0)] + [(G.PC_CHEBYSHEV, d) for d in (2, 3, 4, 5, 6, 7)],
                         ids=["jacobi", "cheb2", "cheb3", "cheb4", "cheb5", "cheb6", "cheb7"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_plane_march_of_small_grids_follows_unfused(shape, pc, deg):
    f, u = _iterate(shape, pc, deg, 1), _iterate(shape, pc, deg, 0)
    assert f[3]["inner_spmv_f32"] >= 8 and f[3]["inner_precond_f32"] >= 8   # the passes ran, not the cluster
    assert f[:2] == u[:2] == (G.NOT_CONVERGED, 8)
    # eight FP32 iterations, each within some FP32 roundings of the other form
    assert np.max(np.abs(f[2] - u[2])) < 1e-4 * np.max(np.abs(u[2]))
